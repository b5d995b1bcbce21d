"""Rules that the CUDA sources keep and that no run on a GPU would show broken."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "expert_specialization_moe_b200" / "csrc"

# kernels that read their operands as (or among) the first launch of a call: with programmatic stream serialisation they
# start while the producer of these operands may still run.  (fp8_blockwise_many_rows.cu is always the second launch: it
# starts after the first has waited for the stream's earlier work.)
FIRST_OF_CALL = ["mxfp8_group_quant.cu", "mxfp8_grouped_mm.cu", "mxfp8_grouped_mm_pair.cu", "fp8_blockwise_grouped_mm.cu"]


def _code(name):
    return re.sub(r"//.*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("name", FIRST_OF_CALL)
def test_no_read_only_loads_of_memory_that_is_still_being_written(name):
    """ld.global.nc (also as __ldg, or as the compiler's choice for a const __restrict__ parameter) wants memory that
    nothing writes during the kernel's whole life, which griddepcontrol.wait inside the kernel does not give."""
    code = _code(name)
    assert "cudaLaunchAttributeProgrammaticStreamSerialization" in code
    assert "ld.global.nc" not in code and "__ldg(" not in code and "ld_stream_16B(" not in code
    assert not re.findall(r"const\s+\w+\s*\*\s*__restrict__", code)


def test_predicated_streaming_loads_are_ordinary_loads():
    code = _code("mxfp8_quant_math.cuh")
    for fn in ("ld_stream_32B_if", "ld_stream_16B_if"):
        body = code[code.index("void " + fn):]
        body = body[:body.index("\n}\n")]
        assert "ld.global." in body and ".nc" not in body, fn


def test_kernels_with_read_only_loads_are_launched_without_programmatic_serialisation():
    for path in CSRC.glob("*.cu"):
        code = _code(path.name)
        if "ld_stream_16B(" in code:
            assert "cudaLaunchAttributeProgrammaticStreamSerialization" not in code, path.name


@pytest.mark.parametrize("name", [p.name for p in sorted(CSRC.glob("*.cu")) if "mbar_wait(" in p.read_text()])
def test_a_kernel_that_gave_up_lets_its_copies_land(name):
    """Between the end of the roles and the release of TMEM: a CTA whose roles gave up may have loads into its shared
    memory and MMAs in flight.  (A wait cannot be made to run out in a test without withholding an arrival from a running
    pipeline, so the sources are checked.)"""
    code = re.sub(r"\s+", " ", _code(name))
    last_free = max(m.start() for m in re.finditer(r"ptx::tmem_dealloc(_pair)?\(tmem_base", code))
    tail = code[:last_free]
    settle = tail.rfind("ptx::settle_if_aborted(abort_flag);")
    assert settle > 0, "no settling before the release of TMEM"
    assert tail[:settle].rstrip().endswith("__syncthreads();"), "all roles must have ended"
    assert "mbar_wait" not in tail[settle:] and "tma_load" not in tail[settle:]
