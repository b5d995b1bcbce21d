"""The MXFP8 grouped GEMM kernel at the edges of its tiles: row counts around the MMA's multiples of 16, the token boxes, the
192-row sub-tiles, the 128-row scale atoms and the 384-row items; one to thirteen K steps (the first and last two go sub-tile
by sub-tile); odd numbers of weight tiles; both divisions of shared memory (mean rows per expert below and above 112)."""
import pytest
import torch

from oracle import grouped_gemm_oracle as G
from tests import _cases as C

pytestmark = pytest.mark.gpu
# fp32 sums on both sides, in another order, and one rounding to the output's type on each: half a unit in the last place
# each, 2^-9 (bf16) or 2^-12 (fp16) of a value at most, so their 2-norms differ by less than twice that
REL = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}

EDGES = [1, 15, 16, 17, 31, 33, 64, 65, 112, 113, 127, 128, 129, 191, 192, 193]
LARGE = [255, 256, 257, 272, 320, 383, 384, 385, 400, 512, 513, 640, 769, 0, 7, 130]


def _compare(inp, d, dt):
    ref = G.mxfp8_grouped_mm(torch.from_numpy(inp["a_codes"]), torch.from_numpy(inp["w_codes"]),
                             torch.from_numpy(inp["sfa"]), torch.from_numpy(inp["sfb"]), inp["ps"], inp["eo"], inp["bo"],
                             out_dtype=dt)
    for e in range(len(inp["ps"])):
        m, off = int(inp["ps"][e][0]), int(inp["eo"][e])
        if m == 0:
            continue
        x, y = d[off:off + m].double(), ref[off:off + m].double()
        # every row by itself: a misplaced row or sub-tile must not vanish in the norm of the others
        rel = ((x - y).norm(dim=1) / y.norm(dim=1)).max()
        assert rel <= REL[dt], f"expert {e}, {m} rows: {rel:.2e}"
    rc, raw = C.device_status()
    assert rc == 0, f"device status {raw:#x}"


@pytest.mark.parametrize("counts,n,k,dt", [
    (EDGES, 256, 128, torch.bfloat16),
    (EDGES, 384, 256, torch.float16),
    (EDGES, 128, 384, torch.bfloat16),
    (EDGES, 640, 1664, torch.bfloat16),
    (LARGE, 256, 128, torch.float16),
    (LARGE, 384, 256, torch.bfloat16),
    (LARGE, 256, 384, torch.bfloat16),
    (LARGE, 128, 512, torch.float16),
    (LARGE, 384, 640, torch.bfloat16),
    (LARGE + EDGES + [3] * 40, 384, 512, torch.bfloat16),     # few rows on average, heavy and light items mixed
])
def test_edges_of_the_tiles(counts, n, k, dt):
    inp = C.mxfp8_gemm_inputs(counts, n, k, seed=n + k)
    _compare(inp, C.run_mxfp8_mm_op(inp, dt), dt)


def test_one_pair_of_ctas_works_through_everything():
    """All items, of changing sizes, through the rings and the queue of one CTA pair; and dealt without counters."""
    from expert_specialization_moe_b200 import _cabi
    inp = C.mxfp8_gemm_inputs(LARGE + EDGES, 384, 640, seed=5)
    want = C.run_mxfp8_mm_op(inp)
    _compare(inp, want, torch.bfloat16)
    try:
        for name, value in (("mm_pair_max_clusters", 1), ("mm_dynamic", 0), ("mm_item_k_steps", 40)):
            _cabi.set_tunable(name, value)
            assert torch.equal(C.run_mxfp8_mm_op(inp), want), name
    finally:
        _cabi.set_tunable("mm_pair_max_clusters", 0)
        _cabi.set_tunable("mm_dynamic", 1)
        _cabi.set_tunable("mm_item_k_steps", 16)
    rc, raw = C.device_status()
    assert rc == 0, f"device status {raw:#x}"
