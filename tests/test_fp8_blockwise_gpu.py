"""GPU parity of the FP8-blockwise grouped GEMM (fp32 scales: 1x128 on A, 128x128 on B) against the restated torch
dequant-matmul path of the reference's test (test/test_es_grouped_gemm.py:36-86).  Floating point: relative error
<= 1e-2, cosine >= 0.9999 versus the dequantised fp32 matmul, and the reference test's own acceptance
calc_diff < 1e-3 versus the UNQUANTISED matmul (test_es_grouped_gemm.py:140,195-199)."""
import pytest
import torch

from oracle import grouped_gemm_oracle as G
from tests import _cases as C

pytestmark = pytest.mark.gpu


def _check(inp, d, out_dtype):
    ref = G.fp8_blockwise_grouped_mm(inp["a_q"].view(torch.uint8), inp["w_q"].view(torch.uint8), inp["sa"], inp["sb"],
                                     inp["ps"], inp["eo"], out_dtype=out_dtype)
    for e in range(len(inp["ps"])):
        m, off = int(inp["ps"][e][0]), int(inp["eo"][e])
        if m == 0:
            continue
        rel, cos = G.rel_err_and_cosine(d[off:off + m].float(), ref[off:off + m].float())
        assert rel <= 1e-2 and cos >= 0.9999, f"expert {e} (m={m}): rel={rel:.3e} cos={cos:.6f}"
        unq = inp["a"][off:off + m].float() @ inp["w"][e].float().t()
        assert G.calc_diff(d[off:off + m], unq) < 1e-3
    rc, raw = C.device_status()
    assert rc == 0, f"device status {raw:#x}"


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,N,K", [
    ([0, 1, 3, 7, 16, 64, 128, 293], 1024, 512),     # the CPU-runnable configuration of the build target
    ([1], 128, 128),
    ([130, 0, 77], 256, 384),
    ([200, 31], 128, 7168),
])
def test_blockwise_matches_oracle(counts, N, K, out_dtype):
    inp = C.fp8_blockwise_inputs(counts, N, K, seed=0, dtype=out_dtype)
    d = C.run_fp8_blockwise_op(inp, out_dtype)
    _check(inp, d, out_dtype)


@pytest.mark.parametrize("lo,hi,E,N,K", [
    (1, 32, 96, 1024, 1280),      # <= 32 rows: 768 tiles of 10 K blocks (two scale chunks per tile)
    (33, 64, 96, 1024, 512),      # 33..64 rows: tiles of 4 K blocks = one pass over the TMEM partials
    (65, 200, 40, 1024, 1152),    # >= 65 rows, some experts with two token tiles
    (1, 150, 120, 896, 384),      # all three buckets in one call
    (1, 40, 150, 640, 256),       # two K blocks: work items of four weight tiles, 5 tiles per expert (4 + 1)
    (1, 100, 100, 1408, 512),     # four K blocks: items of two weight tiles, 11 tiles per expert (5 x 2 + 1)
    (1, 32, 200, 7168, 256),      # the short-K point of the reference's benchmark at test size
])
def test_blockwise_many_tiles_per_cta(lo, hi, E, N, K):
    """More tiles than SMs, so that every CTA walks several tiles: covers the hand-over between the two epilogue
    groups, the rings wrapping across tile boundaries, and the chained per-bucket launches."""
    import random
    rnd = random.Random(11)
    counts = [rnd.randint(lo, hi) for _ in range(E)]
    inp = C.fp8_blockwise_inputs(counts, N, K, seed=5)
    d = C.run_fp8_blockwise_op(inp)
    _check(inp, d, torch.bfloat16)


def test_blockwise_more_experts_than_the_shared_memory_tables_hold():
    """400 experts: the per-expert tables behind the item prefix hold the first 312; the rest come from global memory."""
    counts = [(5 * e) % 37 for e in range(400)]
    counts[2], counts[350], counts[399] = 140, 90, 50
    inp = C.fp8_blockwise_inputs(counts, 256, 256, seed=8)
    d = C.run_fp8_blockwise_op(inp)
    _check(inp, d, torch.bfloat16)


def test_blockwise_reference_test_shapes():
    """The reference's own test draws n, k in 128*[1,64], m in [1,256], E in {8..128}; one seeded draw of that family."""
    import random
    rnd = random.Random(3)
    E = 16
    N, K = rnd.randint(1, 16) * 128, rnd.randint(1, 16) * 128
    counts = [rnd.randint(1, 256) for _ in range(E)]
    inp = C.fp8_blockwise_inputs(counts, N, K, seed=1)
    d = C.run_fp8_blockwise_op(inp)
    _check(inp, d, torch.bfloat16)


def test_blockwise_rejects_bad_arguments():
    inp = C.fp8_blockwise_inputs([4], 128, 128, seed=2)
    from expert_specialization_moe_b200 import es_fp8_blockwise_scaled_grouped_mm as op
    dev = "cuda"
    a = inp["a_q"].to(dev); b = inp["w_q"].to(dev).transpose(1, 2)
    sa = inp["sa"].to(dev); sb = inp["sb"].to(dev).transpose(1, 2)
    ps = torch.from_numpy(inp["ps"]).to(dev); eo = torch.from_numpy(inp["eo"]).to(dev)
    st = torch.full((1,), 128, dtype=torch.int64, device=dev)
    ws = torch.empty(16, dtype=torch.uint8, device=dev)
    with pytest.raises(RuntimeError, match="output must be bfloat16 or half"):
        op(torch.zeros((4, 128), dtype=torch.float32, device=dev), a, b, sa, sb, st, st, st, ps, eo, ws)
    with pytest.raises(RuntimeError, match="problem_sizes must be int32"):
        op(torch.zeros((4, 128), dtype=torch.bfloat16, device=dev), a, b, sa, sb, st, st, st, ps.long(), eo, ws)


@pytest.mark.parametrize("counts,N,K", [
    ([33], 128, 128),                                    # one K block, one tile
    ([32, 33, 64, 65, 128, 129, 256, 257], 384, 640),    # edges of the split, of the token boxes and of the 128-row tiles
    ([96] * 40, 1024, 1280),                             # ten K blocks: scales read four at a time with a rest of two
    ([40] * 160, 640, 256),                              # short tiles: five or six per CTA
])
def test_blockwise_many_rows_edges(counts, N, K):
    """Experts of more than 32 rows; an output that is only 16-byte aligned (and token scales that start elsewhere) gives the
    same bits."""
    from expert_specialization_moe_b200 import es_fp8_blockwise_scaled_grouped_mm as op
    inp = C.fp8_blockwise_inputs(counts, N, K, seed=17)
    d = C.run_fp8_blockwise_op(inp)
    _check(inp, d, torch.bfloat16)
    T, dev = sum(counts), "cuda"
    out = torch.zeros(T * N + 8, dtype=torch.bfloat16, device=dev)[8:].view(T, N)
    sa = torch.zeros(T * (K // 128) + 1, device=dev)[1:].view(T, K // 128)
    sa.copy_(inp["sa"])
    ld = torch.full((len(counts),), K, dtype=torch.int64, device=dev)
    op(out, inp["a_q"].to(dev), inp["w_q"].to(dev).transpose(1, 2), sa, inp["sb"].to(dev).transpose(1, 2), ld, ld, ld,
       torch.from_numpy(inp["ps"]).to(dev), torch.from_numpy(inp["eo"]).to(dev),
       torch.empty(16, dtype=torch.uint8, device=dev))
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), d)


@pytest.mark.parametrize("E,N", [(220, 3072), (148, 4096)])
def test_blockwise_many_rows_long_work_list(E, N):
    """Over 32 tiles per CTA — a second batch of the work list — and, with 148 SMs, exactly 32 (a batch without an end
    mark), at one K block per tile."""
    counts = [40] * E
    inp = C.fp8_blockwise_inputs(counts, N, 128, seed=23)
    d = C.run_fp8_blockwise_op(inp)
    _check(inp, d, torch.bfloat16)


@pytest.mark.parametrize("shift_a,shift_b", [(1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("K", [512, 1024])
def test_blockwise_scales_only_4_byte_aligned(K, shift_a, shift_b):
    """K blocks that the many-rows kernel reads four scales at a time where they start on 16 bytes: scales that do not
    give the same bits."""
    from expert_specialization_moe_b200 import es_fp8_blockwise_scaled_grouped_mm as op
    counts, N = [20, 40, 129, 33], 256
    inp = C.fp8_blockwise_inputs(counts, N, K, seed=29)
    d = C.run_fp8_blockwise_op(inp)
    _check(inp, d, torch.bfloat16)
    dev = "cuda"

    def shifted(t, by):
        out = torch.zeros(t.numel() + 4, device=dev)[by:by + t.numel()].view(t.shape)
        out.copy_(t)
        assert out.data_ptr() % 16 == 4 * by
        return out

    out = torch.zeros((sum(counts), N), dtype=torch.bfloat16, device=dev)
    ld = torch.full((len(counts),), K, dtype=torch.int64, device=dev)
    op(out, inp["a_q"].to(dev), inp["w_q"].to(dev).transpose(1, 2), shifted(inp["sa"], shift_a),
       shifted(inp["sb"], shift_b).transpose(1, 2), ld, ld, torch.full_like(ld, N), torch.from_numpy(inp["ps"]).to(dev),
       torch.from_numpy(inp["eo"]).to(dev), torch.empty(16, dtype=torch.uint8, device=dev))
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), d)
