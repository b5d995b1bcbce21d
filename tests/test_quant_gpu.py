"""GPU parity of the MXFP8 grouped quantisation (through ops.py -> C ABI) against the CPU oracle and against the
golden fixtures produced by the reference's own kernel.  Bit-exact: codes everywhere, scale bytes on valid rows,
zeros on the padding rows."""
import hashlib
import json
from pathlib import Path

import numpy as np
import pytest

from oracle import mxfp8_quant_oracle as Q
from tests import _cases as C

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


def _compare(x_bits, is_bf16, counts):
    codes, sf, ps, eo, bo = C.run_quant_op(x_bits, is_bf16, counts)
    ocodes, osf = C.oracle_quant(x_bits, is_bf16, counts)
    assert np.array_equal(codes, ocodes), f"codes differ at {np.argwhere(codes != ocodes)[:5]}"
    assert np.array_equal(sf, osf), f"scale bytes differ at {np.argwhere(sf != osf)[:5]}"


@pytest.mark.parametrize("is_bf16", [True, False])
@pytest.mark.parametrize("counts,K", [
    ([1], 128), ([0, 0, 5], 128), ([127, 128, 129], 256), ([8, 0, 300, 17, 1, 1, 64], 384),
    ([513], 1152), ([3] * 40, 7168), ([0], 128),
])
def test_quant_matches_oracle(counts, K, is_bf16):
    x = C.activations_bits(sum(counts), K, seed=sum(counts) + K, is_bf16=is_bf16)
    if sum(counts) == 0:
        x = np.full((1, K), 0x3F80, dtype=np.uint16)   # an all-empty problem list must leave the outputs untouched
        codes, sf, *_ = C.run_quant_op(x, is_bf16, [0])
        assert not codes.any()
        return
    _compare(x, is_bf16, counts)


def test_quant_edge_values():
    x = Q.edge_case_rows_bf16(512, seed=0)
    _compare(x, True, [x.shape[0]])
    _compare(x, True, [7, 0, x.shape[0] - 7])


def test_quant_many_experts():
    counts = list(Q.zipf_counts(4096, 1024, 1.2, 3))
    _compare(C.activations_bits(4096, 256, 5), True, counts)


def test_quant_rows_outside_experts_untouched():
    """expert ranges need not cover the buffer: rows that belong to no expert keep their previous contents."""
    import torch
    from expert_specialization_moe_b200 import es_sm100_mxfp8_blockscaled_grouped_quant as quant
    K = 256
    x_bits = C.activations_bits(64, K, 11)
    x = C.bits_to_tensor(x_bits, True, "cuda")
    ps = torch.tensor([[10, 0, K], [5, 0, K]], dtype=torch.int32, device="cuda")
    eo = torch.tensor([4, 40], dtype=torch.int32, device="cuda")
    bo = torch.tensor([0, 128], dtype=torch.int32, device="cuda")
    codes = torch.full((64, K), 0x55, dtype=torch.uint8, device="cuda")
    sf = torch.full((256, K // 32), 0xCD, dtype=torch.uint8, device="cuda")
    quant(x, ps, eo, bo, codes, sf)
    torch.cuda.synchronize()
    c = codes.cpu().numpy()
    oc, osf = Q.quantize_rows(x_bits, True)
    touched = np.zeros(64, dtype=bool); touched[4:14] = True; touched[40:45] = True
    assert np.array_equal(c[touched], oc[touched])
    assert (c[~touched] == 0x55).all()
    s = sf.cpu().numpy().reshape(-1)
    assert np.array_equal(Q.unswizzle_sf(s[: 128 * (K // 32)], 10, K), osf[4:14])
    assert np.array_equal(Q.unswizzle_sf(s[128 * (K // 32):], 5, K), osf[40:45])


@pytest.mark.parametrize("name", ["edge_bf16", "ragged_bf16", "ragged_fp16"])
def test_quant_matches_reference_fixture(name):
    f = GOLDEN / f"ref_quant_{name}.npz"
    if not f.exists():
        pytest.skip("fixture not generated yet")
    z = np.load(f)
    counts = z["ps"][:, 0]
    codes, sf, ps, eo, bo = C.run_quant_op(z["x_bits"], bool(z["is_bf16"]), counts)
    assert np.array_equal(codes, z["codes"])
    idx = C.valid_sf_index(counts, bo, z["x_bits"].shape[1])
    assert np.array_equal(sf[idx], z["sf"][idx])


def test_quant_full_size_digest_matches_reference():
    """The benchmark shape (T=32768, K=7168, E=256, Zipf counts): SHA-256 of all codes and of the valid scale bytes
    equals the digest of the reference kernel's output on the same seeded input."""
    f = GOLDEN / "ref_quant_digests.json"
    if not f.exists():
        pytest.skip("fixture not generated yet")
    for d in json.loads(f.read_text()):
        T, K, E, seed = d["T"], d["K"], d["E"], d["seed"]
        x_bits = C.activations_bits(T, K, seed)
        assert hashlib.sha256(x_bits.tobytes()).hexdigest() == d["input_sha256"]
        counts = Q.zipf_counts(T, E, 1.2, seed)
        codes, sf, ps, eo, bo = C.run_quant_op(x_bits, True, counts)
        assert hashlib.sha256(codes.tobytes()).hexdigest() == d["codes_sha256"]
        idx = C.valid_sf_index(counts, bo, K)
        assert hashlib.sha256(sf[idx].tobytes()).hexdigest() == d["sf_valid_sha256"]


# ---- fused SiLU * mul + quant -----------------------------------------------------------------------------------
def _run_silu_mul_quant(gu_bits, is_bf16, counts):
    import torch
    from expert_specialization_moe_b200 import es_sm100_mxfp8_silu_mul_grouped_quant as fused
    T, K2 = gu_bits.shape
    K = K2 // 2
    ps, eo, bo, sf_rows = Q.offsets_from_counts(counts, 0, K)
    dev = "cuda"
    gu = C.bits_to_tensor(gu_bits, is_bf16, dev)
    codes = torch.zeros((T, K), dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn)
    sf = torch.full((max(sf_rows, 1), K // 32), 0xCD, dtype=torch.uint8, device=dev)
    fused(gu, torch.from_numpy(ps).to(dev), torch.from_numpy(eo).to(dev), torch.from_numpy(bo).to(dev), codes, sf)
    torch.cuda.synchronize()
    return codes.view(torch.uint8).cpu().numpy(), sf.cpu().numpy().reshape(-1)[: sf_rows * (K // 32)], gu


@pytest.mark.parametrize("is_bf16", [True, False])
@pytest.mark.parametrize("counts,K", [([5, 0, 130, 64], 128), ([300], 768), ([1] * 7 + [90], 2048)])
def test_fused_silu_mul_quant_equals_unfused_sequence(counts, K, is_bf16):
    """Bit-exact against the unfused GPU sequence (torch silu*mul in fp32 -> input type -> grouped quant op)."""
    import torch
    gu_bits = C.activations_bits(sum(counts), 2 * K, seed=K + len(counts), is_bf16=is_bf16, outliers=False)
    codes, sf, gu = _run_silu_mul_quant(gu_bits, is_bf16, counts)
    act = (torch.nn.functional.silu(gu[:, :K].float()) * gu[:, K:].float()).to(gu.dtype)
    act_bits = act.view(torch.int16).cpu().numpy().view(np.uint16)
    ucodes, usf, *_ = C.run_quant_op(act_bits, is_bf16, counts)
    assert np.array_equal(codes, ucodes)
    assert np.array_equal(sf, usf)


def test_fused_silu_mul_quant_matches_cpu_oracle():
    """Against the numpy oracle; its float32 exp may differ from the GPU's in the last bit, so a small fraction of
    16-bit activations (and with them codes) may differ: allowance 1e-3 of the codes, scales 1e-3 of the bytes."""
    counts, K = [40, 3, 200], 512
    gu_bits = C.activations_bits(sum(counts), 2 * K, seed=5, outliers=False)
    codes, sf, _ = _run_silu_mul_quant(gu_bits, True, counts)
    act_bits = Q.silu_mul_bits(gu_bits, True)
    ocodes, osf = C.oracle_quant(act_bits, True, counts)
    assert (codes != ocodes).mean() < 1e-3
    assert (sf != osf).mean() < 1e-3


@pytest.mark.parametrize("is_bf16", [True, False])
def test_fused_silu_mul_quant_every_gate_value(is_bf16):
    """Every finite 16-bit gate value (subnormals, zeros, the largest) times up values over the whole exponent range,
    bit-exact against the unfused GPU sequence: the fast form of the activation and its hand-over to the exact one."""
    import torch
    bits = np.arange(65536, dtype=np.uint16)
    exp_mask = 0x7F80 if is_bf16 else 0x7C00
    bits[(bits & exp_mask) == exp_mask] = 0x3C00
    rng = np.random.default_rng(3)
    T, K = 640, 512                                    # five passes over the 65536 gate values
    gate = np.stack([rng.permutation(bits) for _ in range(5)]).reshape(T, K)
    up = rng.integers(0, 65536, size=(T, K)).astype(np.uint16)
    up[(up & exp_mask) == exp_mask] = 0x0001
    half = rng.random((T, K)) < 0.5                    # half of them ordinary values: |up| in [0.25, 8)
    plain = C.activations_bits(T, K, seed=9, is_bf16=is_bf16, outliers=False)
    gu_bits = np.concatenate([gate, np.where(half, plain, up)], axis=1)
    counts = [600, 1, 39]
    codes, sf, gu = _run_silu_mul_quant(gu_bits, is_bf16, counts)
    act = (torch.nn.functional.silu(gu[:, :K].float()) * gu[:, K:].float()).to(gu.dtype)
    ucodes, usf, *_ = C.run_quant_op(act.view(torch.int16).cpu().numpy().view(np.uint16), is_bf16, counts)
    assert np.array_equal(codes, ucodes)
    assert np.array_equal(sf, usf)


@pytest.mark.parametrize("counts,K", [([1], 128), ([3, 0, 2], 128), ([37, 129, 1], 640), ([33] * 9, 768),
                                      ([700, 1, 260], 2176)])
def test_quant_unit_edges_and_alignment(counts, K):
    """Ragged last steps (K tiles per row that do not divide a step of 32), at most one step per CTA; an input that starts
    16 bytes past a 32-byte boundary, and scale offsets whose padding words are only 4-byte aligned."""
    import torch
    from expert_specialization_moe_b200 import es_sm100_mxfp8_blockscaled_grouped_quant as quant
    T = sum(counts)
    x_bits = C.activations_bits(T, K, seed=T + K)
    ocodes, osf = C.oracle_quant(x_bits, True, counts)
    ps, eo, bo, sf_rows = Q.offsets_from_counts(counts, 0, K)
    flat = torch.empty(T * K + 8, dtype=torch.bfloat16, device="cuda")
    x = flat[8:].view(T, K)
    assert x.data_ptr() % 32 == 16
    x.copy_(C.bits_to_tensor(x_bits, True, "cuda"))
    codes = torch.zeros((T, K), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    sf = torch.full((sf_rows + 8, K // 32), 0xCD, dtype=torch.uint8, device="cuda")
    dev = [torch.from_numpy(a).to("cuda") for a in (ps, eo, bo + 1)]
    quant(x, *dev, codes, sf)
    torch.cuda.synchronize()
    assert np.array_equal(codes.view(torch.uint8).cpu().numpy(), ocodes)
    got = sf.cpu().numpy().reshape(-1)
    lead = K // 32
    assert np.array_equal(got[lead:lead + osf.size], osf)
    assert (got[:lead] == 0xCD).all() and (got[lead + osf.size:] == 0xCD).all()


def _silu_special_rows(is_bf16):
    """Blocks of 32 products in which one gate / up pair is special — zeros, infinities, NaN, gates around -64 (end of the
    fast form's range) and -88.7 (where exp overflows), the extremes of the type — next to ordinary values, zeros, or
    values whose products are next to the fp32 subnormals."""
    import torch
    dt = torch.bfloat16 if is_bf16 else torch.float16
    top = torch.finfo(dt).max
    gates = [0.0, -0.0, float("inf"), -float("inf"), float("nan"), -63.75, -64.0, -64.5, -70.0, -87.0, -88.5, -89.0, -90.5,
             -200.0, -top, 65.0, 200.0, top, 1.0, torch.finfo(dt).smallest_normal, -2.0 ** -24]
    ups = [0.0, -0.0, float("inf"), -float("inf"), float("nan"), 1.0, -3.0, top, -torch.finfo(dt).smallest_normal, 2.0 ** -24]
    gen = torch.Generator().manual_seed(21)
    n = len(gates) * len(ups)
    g = torch.randn((4, n, 32), generator=gen)
    u = torch.randn((4, n, 32), generator=gen)
    g[1], u[1] = 0.0, torch.where(u[1] < 0, -0.0, 0.0)
    if is_bf16:                                # products of 2^-84 .. 2^-133; the largest of a block near the limit
        g[2] *= 2.0 ** -60
        u[2] *= 2.0 ** torch.randint(-75, -20, (n, 1), generator=gen).float()
        g[3, :, 1:16] = 0.0                    # a lane of zeros next to one of gates that leave the fast form
    g[3] *= 40.0
    at = torch.randint(0, 32, (4, n), generator=gen)
    g.scatter_(2, at.unsqueeze(2), torch.tensor(gates).repeat_interleave(len(ups)).expand(4, n).unsqueeze(2).contiguous())
    u.scatter_(2, at.unsqueeze(2), torch.tensor(ups).repeat(len(gates)).expand(4, n).unsqueeze(2).contiguous())
    K = 128
    as_bits = lambda t: t.reshape(-1, K).to(dt).view(torch.int16).numpy().view(np.uint16)
    return np.concatenate([as_bits(g), as_bits(u)], axis=1), K


@pytest.mark.parametrize("is_bf16", [True, False])
def test_fused_silu_mul_quant_special_values(is_bf16):
    """Infinities, NaN, zeros and the ends of the fast form's range, bit-exact against the unfused GPU sequence."""
    import torch
    gu_bits, K = _silu_special_rows(is_bf16)
    counts = [gu_bits.shape[0] - 7, 0, 7]
    codes, sf, gu = _run_silu_mul_quant(gu_bits, is_bf16, counts)
    act = (torch.nn.functional.silu(gu[:, :K].float()) * gu[:, K:].float()).to(gu.dtype)
    ucodes, usf, *_ = C.run_quant_op(act.view(torch.int16).cpu().numpy().view(np.uint16), is_bf16, counts)
    assert np.array_equal(codes, ucodes), np.argwhere(codes != ucodes)[:8]
    assert np.array_equal(sf, usf)


@pytest.mark.parametrize("is_bf16", [True, False])
def test_fused_silu_mul_quant_time_does_not_depend_on_the_values(is_bf16):
    """Zeros (single ones and whole rows) and outlier gates cost next to nothing: a form of the activation that hands
    such values to the exact sequence lane by lane takes two to three times as long."""
    import torch
    from expert_specialization_moe_b200 import es_sm100_mxfp8_silu_mul_grouped_quant as fused
    T, K, E = 65536, 768, 64
    ps, eo, bo, sf_rows = Q.offsets_from_counts([T // E] * E, 0, K)
    lists = [torch.from_numpy(a).cuda() for a in (ps, eo, bo)]
    gen = torch.Generator(device="cuda").manual_seed(4)
    plain = torch.randn((T, 2 * K), generator=gen, device="cuda")
    plain = torch.where(plain.abs() < 2.0 ** -20, 1.0, plain)          # the generator itself gives zeros now and then
    chance = torch.rand((T, 2 * K), generator=gen, device="cuda")
    codes = torch.empty((T, K), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    sf = torch.empty((sf_rows, K // 32), dtype=torch.uint8, device="cuda")
    inputs = {"plain": plain, "zeros": torch.where(chance < 0.01, 0.0, plain),
              "zero rows": torch.where(chance[:, :1] < 0.1, 0.0, plain),
              "outliers": torch.where(chance < 0.01, 50.0 * plain, plain)}
    took = {}
    for name, x in inputs.items():
        x = x.to(torch.bfloat16 if is_bf16 else torch.float16)
        times = []
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                fused(x, *lists, codes, sf)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        took[name] = sorted(times)[4]
    # measured: up to 1.03 (outliers); 1.4 leaves room for a busy GPU
    assert max(took.values()) < 1.4 * took["plain"], took


# Rows that give every CTA several steps of 32 K tiles: a grid is at most 4 CTAs (3 with silu) on each of up to 160 SMs.
def _rows_for_steps(steps, K, ctas_per_sm):
    return steps * ctas_per_sm * 160 * 32 * 128 // K + 3


def _silu_bits_on_gpu(gu, K):
    import torch
    return (torch.nn.functional.silu(gu[:, :K].float()) * gu[:, K:].float()).to(gu.dtype)


def _quantise_on_gpu(x, counts, lists, sf_rows, op, K):
    import torch
    codes = torch.zeros((x.shape[0], K), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    sf = torch.full((sf_rows, K // 32), 0xCD, dtype=torch.uint8, device="cuda")
    op(x, *lists, codes, sf)
    torch.cuda.synchronize()
    return codes.view(torch.uint8), sf


@pytest.mark.parametrize("K,is_bf16", [(128, True), (640, True), (640, False), (2176, False)])
def test_quant_several_steps_per_cta(K, is_bf16):
    """Five to six steps per CTA (the loads two steps ahead, the carry of row and tile from step to step, every place of
    the register rotation), an expert's end and another's start inside a CTA's stretch: against the CPU oracle; and from
    an input that starts 16 bytes past a 32-byte boundary."""
    import torch
    from expert_specialization_moe_b200 import es_sm100_mxfp8_blockscaled_grouped_quant as quant
    T = _rows_for_steps(6, K, 4)
    counts = [T // 3, 0, T - T // 3 - 1, 1]
    x_bits = C.activations_bits(T, K, seed=K, is_bf16=is_bf16)
    _compare(x_bits, is_bf16, counts)
    ps, eo, bo, sf_rows = Q.offsets_from_counts(counts, 0, K)
    lists = [torch.from_numpy(a).to("cuda") for a in (ps, eo, bo)]
    x = C.bits_to_tensor(x_bits, is_bf16, "cuda")
    shifted = torch.empty(T * K + 8, dtype=x.dtype, device="cuda")[8:].view(T, K)
    shifted.copy_(x)
    assert x.data_ptr() % 32 == 0 and shifted.data_ptr() % 32 == 16
    for a, b in zip(_quantise_on_gpu(x, counts, lists, sf_rows, quant, K),
                    _quantise_on_gpu(shifted, counts, lists, sf_rows, quant, K)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("steps,K", [(30, 640), (52, 7168)])
def test_quant_long_share(steps, K):
    """More than 27 steps per CTA, dealt eight at a time, over several experts: the bits of one call per expert, whose
    CTAs have fewer; and the same from an input that starts 16 bytes past a 32-byte boundary."""
    import torch
    from expert_specialization_moe_b200 import es_sm100_mxfp8_blockscaled_grouped_quant as quant
    T = _rows_for_steps(steps, K, 4)
    counts = [T // 5, T // 4, 1, T - T // 5 - T // 4 - 1]
    ps, eo, bo, sf_rows = Q.offsets_from_counts(counts, 0, K)
    lists = [torch.from_numpy(a).to("cuda") for a in (ps, eo, bo)]
    x = torch.randn((T, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).to(torch.bfloat16)
    whole = _quantise_on_gpu(x, counts, lists, sf_rows, quant, K)
    parts = [torch.zeros((T, K), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn),
             torch.full((sf_rows, K // 32), 0xCD, dtype=torch.uint8, device="cuda")]
    for e in range(len(counts)):
        for first in range(0, counts[e], T // 8 // 128 * 128):       # whole scale atoms
            rows = min(counts[e] - first, T // 8 // 128 * 128)
            one = [torch.tensor(v, dtype=torch.int32, device="cuda")
                   for v in ([[rows, 0, K]], [int(eo[e]) + first], [int(bo[e]) + first])]
            quant(x, *one, *parts)
    torch.cuda.synchronize()
    shifted = torch.empty(T * K + 8, dtype=x.dtype, device="cuda")[8:].view(T, K)
    shifted.copy_(x)
    again = _quantise_on_gpu(shifted, counts, lists, sf_rows, quant, K)
    for a, b, c in zip(whole, parts, again):
        assert torch.equal(a, b.view(torch.uint8)) and torch.equal(a, c)


@pytest.mark.parametrize("shift", [0, 8])
@pytest.mark.parametrize("is_bf16", [True, False])
@pytest.mark.parametrize("K", [128, 640, 2176])
def test_fused_silu_mul_quant_several_steps_per_cta(K, is_bf16, shift):
    """As above for the fused form, against the unfused GPU sequence (whose quantisation the tests above pin)."""
    import torch
    from expert_specialization_moe_b200 import es_sm100_mxfp8_blockscaled_grouped_quant as quant
    from expert_specialization_moe_b200 import es_sm100_mxfp8_silu_mul_grouped_quant as fused
    T = _rows_for_steps(6, K, 3)
    counts = [T // 3, 0, T - T // 3 - 1, 1]
    ps, eo, bo, sf_rows = Q.offsets_from_counts(counts, 0, K)
    lists = [torch.from_numpy(a).to("cuda") for a in (ps, eo, bo)]
    gen = torch.Generator(device="cuda").manual_seed(K)
    gu = torch.empty(T * 2 * K + 8, dtype=torch.bfloat16 if is_bf16 else torch.float16, device="cuda")[shift:shift + T * 2 * K]
    gu = gu.view(T, 2 * K)
    gu.copy_(torch.randn((T, 2 * K), device="cuda", generator=gen))
    for a, b in zip(_quantise_on_gpu(gu, counts, lists, sf_rows, fused, K),
                    _quantise_on_gpu(_silu_bits_on_gpu(gu, K), counts, lists, sf_rows, quant, K)):
        assert torch.equal(a, b)
