"""GPU: tile choices that an earlier version of the kernels cached are not taken; the
ones of this version are."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_choices_of_another_version_are_timed_again(cuda, native, tmp_path):
    import torch

    from rtxrmq_gb300.batch import autotune, bucket_of
    lengths = np.array([5000, 6000, 7000])
    starts = np.cumsum(lengths) - lengths
    qcounts = np.full(3, 500)
    qstarts = np.cumsum(qcounts) - qcounts
    A = torch.rand(int(lengths.sum()), device=cuda)
    Q = torch.tensor([[10, 4000]], dtype=torch.int32, device=cuda).repeat(1500, 1)
    cache = tmp_path / "tiles.json"
    dev, b = torch.cuda.get_device_name(), int(bucket_of(5000))
    old = {f"b{b}_qna_tiles": [64, 7, 9], f"b{b}_qna": 96}
    cache.write_text(json.dumps({dev: old}))
    args = (starts, lengths, qstarts, qcounts, A, Q)
    got = autotune(*args, reps=1, cache=cache, tiles=True)[b]
    assert got != (64, 7, 9) and autotune(*args, reps=1, cache=cache)[b] != 96
    table = json.loads(cache.read_text())[dev]
    assert {k: table[k] for k in old} == old and len(table) == 4
    assert autotune(*args, reps=1, cache=cache, tiles=True)[b] == got
    key, = [k for k in table if k not in old and k.endswith("_tiles")]
    table[key] = [64, 7, 9]
    cache.write_text(json.dumps({dev: table}))
    assert autotune(*args, reps=1, cache=cache, tiles=True)[b] == (64, 7, 9)


@pytest.mark.parametrize("light", [False, True])
def test_candidates(cuda, native, light):
    """One list of block sizes with and without the light flag, which changes no
    structure, and none of them twice (above 2^15 the blocks are the default's)."""
    import torch

    from rtxrmq_gb300.batch import autotune
    lengths = np.array([300, 5000, 90_000, 400_000, 700_000])
    starts = np.cumsum(lengths) - lengths
    qcounts = np.full(5, 300)
    qstarts = np.cumsum(qcounts) - qcounts
    A = torch.rand(int(lengths.sum()), device=cuda)
    Q = torch.tensor([[10, 250]], dtype=torch.int32, device=cuda).repeat(1500, 1)
    cfg = autotune(starts, lengths, qstarts, qcounts, A, Q, reps=1, cache=None, tiles=True, light=light)
    assert {t[0] for t in cfg} <= {0, 64, 256, 1024, 4096, 16384}
