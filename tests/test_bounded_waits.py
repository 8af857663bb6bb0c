"""A CTA one of whose bounded waits gives up lets its own copies in flight land
(bounded again) before it returns, and issues none after it: a copy must not
outlive the shared memory that it writes. Every kernel of the sources that waits
on an mbarrier is checked for it here, and one such failure runs on the GPU."""
import ctypes
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "spm-iqc_b200", "csrc")


def _kernels(name):
    with open(os.path.join(CSRC, name)) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    for m in re.finditer(r"__global__ void[^{;]*?(\w+_kernel)\([^{;]*\{", code):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(code[i], 0)
            i += 1
        yield m.group(1), code[m.end():i]


def test_every_waiting_kernel_drains_its_copies():
    waiting = {}
    for name in ("fft_kernels.cuh", "tile_kernels.cuh", "blockops.cuh", "spm_cuda.cu"):
        for k, body in _kernels(name):
            if re.search(r"\bmbar_wait(_n)?\(", body):
                waiting[name, k] = "drain_copies(" in body or re.search(r"if \(s_err\) \{[^}]*mbar_try_wait", body)
    # plane_fwd, pencil, plane_inv; gram and combine; the self-test (the tile passes wait in Stage)
    assert len(waiting) == 6 and all(waiting.values()), waiting


def test_the_tile_passes_stage_drains_and_stops_issuing():
    with open(os.path.join(CSRC, "tile_kernels.cuh")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    assert code.count("mbar_wait(") == 2  # wait() and next()
    assert "tid == 0 && mbar_wait(empty + g, round & 1, err)" in code
    end = code[code.index("void run(const TileParams"):code.index("bool last(")]
    assert re.search(r"\*st\.err && threadIdx\.x == 0\) st\.drain\(\);", end)
    assert "drain_copies(full + g, issued[g])" in code


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("N", [32, 256])
def test_copies_in_flight_land_before_a_timed_out_cta_returns(cuda, N, prec):
    """One poll (the copy is in flight, if ever), and the same with the copy long there."""
    import spmiqc
    f = spmiqc.lib().spm_selftest_bounded_wait
    f.argtypes = [ctypes.c_void_p, ctypes.c_int]
    f.restype = ctypes.c_int
    c = spmiqc.SpmContext(N, precision=prec)
    for polls in [1] * 50 + [2000]:
        assert f(c.h, polls) == spmiqc.SPM_ERR_CUDA
        assert b"bounded wait" in spmiqc.lib().spm_last_error()
    c.sync()
    c.close()
