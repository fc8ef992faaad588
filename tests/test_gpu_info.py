"""GPU: the sizes that rmq_info reports of an index add up to the memory it holds: block
tables (both of a large array), micro-block minima and masks, rounded up part by
part, and the counter."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 999, 100_003, (1 << 20) + 9, (1 << 22) + 77, 50_000_000])
def test_parts_of_an_index(cuda, native, n):
    import torch

    import rtxrmq_gb300 as R
    A = torch.zeros(n, device=cuda)
    for bs, light in ((0, False), (128, False), (4096, True))[:2 if n < 64 else 3]:  # no light index below 64
        with R.RMQIndex(A, bs, light=light) as ix:
            info = ix.info()
            parts = info["table_bytes"] + info["micro_table_bytes"]
            assert parts < info["struct_bytes"] <= parts + 8 * 256, info
    with R.RMQIndex(A, 128, micro=False) as ix:
        info = ix.info()
        parts = info["table_bytes"] + 16 * n
        assert parts < info["struct_bytes"] <= parts + 8 * 256, info
