"""The batched autotuner and the library agree on which group sizes there are: a
plan's items show the size that runs, and every candidate that the search times
is a plan of its own."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def items(n, count, group):
    import ctypes
    from bola_gb300.batch import Batch, Tuning
    batch = Batch([n] * count, [1] * count, [0] * count, tuning=Tuning(group_size=[group] * 8))
    k = ctypes.c_int32()
    assert batch.L.bola_batch_plan_info(batch.plan, ctypes.byref(k), None, None) == 0
    return k.value


def test_groups_that_run_as_given():
    from bola_gb300.batch import BUCKET_N, GROUP_CHOICES, group_choices
    count = 64
    for b, top in enumerate(BUCKET_N):
        as_given = tuple(g for g in GROUP_CHOICES if items(top, count, g) == count * g // 256)
        assert group_choices(b) == as_given and as_given[0] >= min(top, 256), (b, top)


def test_autotuned_sizes_are_the_ones_that_run(tmp_path):
    from bola_gb300.batch import Batch, autotune, bucket_of, group_choices
    rng = np.random.default_rng(5)
    ns = np.array([5, 16, 30, 40, 64, 90, 128, 200], dtype=np.int32)
    batch = Batch(ns, np.ones(8, np.int32), np.zeros(8, np.int32))
    for i, n in enumerate(ns):
        batch.a_view(i).copy_(torch.from_numpy(rng.uniform(-1.0, 1.0, (n, n)) + n * np.eye(n)))
        batch.b_view(i).copy_(torch.from_numpy(rng.uniform(-1.0, 1.0, (n, 1))))
    best, trials = autotune(batch, reps=1, path=tmp_path / "table.json")
    for n in ns:
        b = bucket_of(int(n))
        tried = {int(key.split("/")[0]) for key in trials[b]}
        assert tried == set(group_choices(b))
        assert best.group_size[b] in tried
