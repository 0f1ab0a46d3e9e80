"""Register spills of the kernels that the library holds, by name: each kernel
on a main path is compiled (its host symbol is in the library, so a renamed or
removed kernel shows here) and does not spill, and the kernels that do spill
are these and no others, within today's bytes."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "tsqr_gb300", "_build")

# kernel -> (spill store bytes, spill load bytes) at most
SPILLS = {
    # FP64 column split, 3 CTAs per SM: the FP64 rate bounds it
    "tsqr::factor_split_tiles<double, 32, 4, 8, 3, false>": (616, 984),
    # FP64 norm, beta and tau in FP32 tiles: an option, off by default
    "tsqr::factor_split_tiles<float, 16, 4, 16, 4, true>": (108, 228),
    "tsqr::factor_split_tiles<float, 32, 4, 16, 2, true>": (112, 248),
    "tsqr::factor_split_tiles<float, 64, 8, 16, 1, true>": (132, 132),
    "tsqr::factor_split_tiles<float, 64, 8, 8, 1, true>": (68, 68),
    # two registers of loop state at the 64-register limit of 4 CTAs per SM
    "tsqr::factor_split_tiles_tma<float, 16, 4, 16, 4>": (8, 8),
    "tsqr::gram_partial_kernel<float>": (4, 4),
    "tsqr::gram_partial_kernel<double>": (4, 4),
}

MAIN = ["tsqr::factor_panel_tiles_tma<16, 16, 4>", "tsqr::factor_panel_tiles<16, 16, 4>",
        "tsqr::factor_panel_tiles<32, 16, 1>", "tsqr::factor_panel_tiles<32, 16, 2>",
        "tsqr::factor_split_tiles<float, 32, 4, 16, 2, false>", "tsqr::factor_split_tiles<float, 16, 4, 16, 4, false>",
        "tsqr::factor_tiles<8, 256, 4, 3>", "tsqr::apply_tiles_f32<8, 1024, 4>", "tsqr::apply_tiles_f32<16, 512, 4>",
        "tsqr::apply_tiles_f32<32, 512, 2>", "tsqr::apply_tiles_f32<32, 512, 3>", "tsqr::apply_tiles_f32<64, 512, 1>",
        "tsqr::apply_tiles_f32<64, 512, 2>", "tsqr::tc_apply_tiles<32, 512, true>", "tsqr::tc_apply_tiles<64, 512, true>",
        "tsqr::factor_stack_tiles<8, 4, 16>", "tsqr::factor_stack_tiles<16, 4, 16>", "tsqr::factor_stack_tiles<32, 8, 16>",
        "tsqr::apply_f64_tiles<32, 256, 1, 2, false>", "tsqr::apply_f64_tiles<32, 256, 4, 2, true>",
        "tsqr::batched_factor_panels<16, 16, 4>", "tsqr::batched_factor_panels<32, 16, 2>",
        "tsqr::batched_factor_split<32, 4, 16, 2>", "tsqr::batched_apply_f32<32, 512>", "tsqr::batched_apply_f32<64, 512>",
        "tsqr::gemm_tn_tma", "tsqr::gemm_nn_fused<true>", "tsqr::tc_nn_kernel<128>", "tsqr::tc_nn_kernel<64>",
        "tsqr::tc_tn_tma_kernel<256>", "tsqr::hr_reconstruct<float>", "tsqr::rows_times_upper<float, true>",
        "tsqr::apply_qt_column<float, 32>"]

WARN = re.compile(r"Registers are spilled to local memory in function '([^']+)', (\d+) bytes spill stores, "
                  r"(\d+) bytes spill loads")


def _kernel(name):
    name = name.replace("(anonymous namespace)::", "")
    return (name[5:] if name.startswith("void ") else name).split("(")[0]


@pytest.fixture(scope="module")
def compiled(tg):
    if shutil.which("nm") is None or shutil.which("c++filt") is None:
        pytest.skip("binutils not available")
    out = subprocess.run(["nm", "-C", tg.library_path()], capture_output=True, text=True, check=True).stdout
    return {_kernel(line.split(" ", 2)[2]) for line in out.splitlines() if line[:1] not in (" ", "") and "tsqr::" in line}


@pytest.fixture(scope="module")
def spills(compiled):
    from tsqr_gb300 import build as tb
    logs = [os.path.join(BUILD, s.replace(".cu", ".ptxas.log")) for s in tb.SOURCES]
    found = []
    for p in logs:
        with open(p) as f:
            found += WARN.findall(f.read())
    names = subprocess.run(["c++filt"], input="\n".join(f[0] for f in found), capture_output=True, text=True,
                           check=True).stdout.splitlines()
    # the CUDA math library's own slow paths (FP64 reciprocal, square root) are not the library's
    return {_kernel(n): (int(f[1]), int(f[2])) for n, f in zip(names, found) if not n.startswith("__cuda_")}


@pytest.mark.parametrize("kernel", MAIN)
def test_main_kernels_are_there_and_do_not_spill(compiled, spills, kernel):
    assert kernel in compiled
    assert kernel not in spills


def test_spilling_kernels_are_the_known_ones(compiled, spills):
    assert set(SPILLS) <= compiled
    assert set(spills) == set(SPILLS)
    assert all(st <= SPILLS[k][0] and ld <= SPILLS[k][1] for k, (st, ld) in spills.items()), spills
