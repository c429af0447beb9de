"""The tuner times a TF32 plan with the re-run of the queries that it lists, also on host buffers, where that
follows the batch (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex, kernel_launch_count

pytestmark = pytest.mark.gpu


def test_tuning_a_host_batch_runs_what_the_candidate_scan_lists():
    # a quarter of the rows are copies of one row: queries beside it find more equals than a list holds
    rng = np.random.default_rng(7)
    m = rng.normal(size=(60_000, 64)).astype(np.float32)
    m[::4] = m[0]
    clean = rng.normal(size=(12, 64)).astype(np.float32)
    clean -= (clean @ m[:1].T) / np.dot(m[0], m[0]) * m[0]  # none of them beside it
    near = (m[0] + 1e-3 * rng.normal(size=(12, 64))).astype(np.float32)
    tuning = {}
    for name, q in (("clean", clean), ("near", near)):
        index = NNdex(m)
        before = kernel_launch_count()
        index.search(q, k=10)
        st = index.last_search_stats()
        assert st["tuned"] == 1 and st["tune_candidates"] == 2, st
        tuning[name] = kernel_launch_count() - before - st["kernel_launches"]
    # two runs of the candidate scan, each with the FP32 scan and the merge of the listed queries
    assert tuning["near"] == tuning["clean"] + 4, tuning
