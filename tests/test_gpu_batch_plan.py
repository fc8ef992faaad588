"""GPU: what a batch plan reports of its tiles is what it was cut into."""
import pytest

pytestmark = pytest.mark.gpu


def test_query_items_stay_below_the_numbering(cuda, native):
    """The queries of an item are numbered in 30 bits, beside two flags: larger
    items than 2^29 are cut whatever is asked for. The plan alone; nothing runs."""
    from rtxrmq_gb300.batch import RMQBatch
    for chunk, items in (((1 << 31) - 1, 4), (1 << 30, 4), (1 << 29, 4), ((1 << 29) - 1, 5), (1 << 28, 8)):
        q = 4 << 29
        with RMQBatch([0], [1000], [0], [q], [(64, chunk, 4096)] * 32) as b:
            assert b.info()["query_items"] == items, chunk
            assert b.tiles()[9][1] == min(chunk, 1 << 29)


@pytest.mark.parametrize("q", [1000, 1_000_000, 50_000_000])
def test_default_tiles_are_the_plans(cuda, native, q):
    """Without a chunk asked for, the reported one is the one that the items have:
    4096 queries, fewer in a plan that has not that many for every CTA."""
    import torch

    from rtxrmq_gb300.batch import RMQBatch
    ctas = torch.cuda.get_device_properties(cuda).multi_processor_count * 4
    chunk = min(max(q // ctas, 512), 4096)
    for tiles in (None, [(64, 0, 0)] * 32, [64] * 32):
        with RMQBatch([0], [1000], [0], [q], tiles) as b:
            assert {t[1] for t in b.tiles()} == {chunk}
            assert b.info()["query_items"] == (q + chunk - 1) // chunk
