"""The gate_up GEMM with silu(gate) * up and the requantisation in its epilogue, at the edges of its tiles: row counts around
64-row tile steps (tiles that start in the middle of a scale atom), one to five K steps, an odd number of weight tiles."""
import numpy as np
import pytest
import torch

from tests import _cases as C

pytestmark = pytest.mark.gpu


def _unswizzle(sf, kb):
    """flat 512-byte atoms -> [rows, kb] scale bytes"""
    r = sf.size // kb
    return sf.reshape(r // 128, kb // 4, 32, 4, 4).transpose(0, 3, 2, 1, 4).reshape(r, kb)


def _dequant(codes, sf):
    v = torch.from_numpy(codes).view(torch.float8_e4m3fn).double()
    s = torch.exp2(torch.from_numpy(sf.astype(np.float64)) - 127.0)
    return (v.view(v.shape[0], -1, 32) * s.unsqueeze(-1)).reshape(v.shape)


@pytest.mark.parametrize("counts,inter,k", [
    ([1, 15, 17, 63, 64, 65, 127, 129, 191, 192, 193], 128, 128),
    ([0, 200, 255, 257, 320, 384, 385, 400, 3], 256, 256),
    ([1000, 0, 577, 33], 384, 384),
    ([5] * 60 + [640], 128, 640),
])
def test_codes_and_scales(counts, inter, k):
    from expert_specialization_moe_b200 import _cabi
    lib = _cabi.load()
    inp = C.mxfp8_gemm_inputs(counts, 2 * inter, k, seed=inter + k, w_std=0.3)
    rows, e = int(sum(counts)), len(counts)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    a, w, sfa, sfb, ps, eo, bo = (dev(inp[n]) for n in ("a_codes", "w_codes", "sfa", "sfb", "ps", "eo", "bo"))
    sf_rows = inp["sfa"].size // (k // 32)
    codes = torch.full((rows + 3, inter), 0x55, dtype=torch.uint8, device="cuda")
    sf = torch.full((sf_rows * (inter // 32),), 0xCD, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    scratch = _cabi.grouped_mm_scratch(codes.device, stream)
    _cabi.check(lib.es_b200_mxfp8_grouped_mm_silu_mul_quant(
        a.data_ptr(), w.data_ptr(), sfa.data_ptr(), sfb.data_ptr(), codes.data_ptr(), sf.data_ptr(), ps.data_ptr(),
        eo.data_ptr(), bo.data_ptr(), e, rows, inter, k, sf_rows, scratch.data_ptr(), scratch.numel(), stream))
    rc, raw = C.device_status()
    assert rc == 0, f"device status {raw:#x}"
    assert int(scratch.view(torch.int32).abs().sum()) == 0
    assert bool((codes[rows:] == 0x55).all()), "rows past the last expert were written"
    codes, sfo = codes[:rows].cpu().numpy(), _unswizzle(sf.cpu().numpy(), inter // 32)
    sfi = _unswizzle(inp["sfa"], k // 32)
    wsf = _unswizzle(inp["sfb"], k // 32).reshape(e, 2 * inter, k // 32)
    for x in range(e):
        m, r, b = counts[x], int(inp["eo"][x]), int(inp["bo"][x])
        if m == 0:
            continue
        h = _dequant(inp["a_codes"][r:r + m], sfi[b:b + m]) @ _dequant(inp["w_codes"][x], wsf[x]).t()
        act = h[:, :inter] / (1 + torch.exp(-h[:, :inter])) * h[:, inter:]
        blk = act.view(m, inter // 32, 32)
        amax = blk.abs().amax(-1)
        scale = torch.exp2(torch.from_numpy(sfo[b:b + m].astype(np.float64)) - 127.0)
        # the smallest power of two that brings the block's largest magnitude to 448; one that is a hair's breadth from a
        # power of two may fall on either side (fp32 sums and exponential: 2^-18 of it is generous)
        assert bool((amax <= 448 * scale * (1 + 2.0 ** -18)).all() and (amax >= 224 * scale * (1 - 2.0 ** -18)).all())
        got = _dequant(codes[r:r + m], sfo[b:b + m]).view(m, inter // 32, 32)
        # half a step of e4m3: 2^-4 of the value, or of the smallest normal number (2^-6) of the block's scale
        bound = torch.maximum(blk.abs(), (scale * 2.0 ** -6).unsqueeze(-1)) * 2.0 ** -4 * (1 + 2.0 ** -8)
        assert bool(((got - blk).abs() <= bound + amax.unsqueeze(-1) * 2.0 ** -18).all()), f"expert {x}, {m} rows"
    with pytest.raises(_cabi.EsB200Error):
        _cabi.check(lib.es_b200_mxfp8_grouped_mm_silu_mul_quant(
            a.data_ptr(), w.data_ptr(), sfa.data_ptr(), sfb.data_ptr(), 16, 16, ps.data_ptr(), eo.data_ptr(),
            bo.data_ptr(), e, rows, 64, k, sf_rows, scratch.data_ptr(), scratch.numel(), stream))
