"""Launch bounds of passes that wait on their neighbours: a few instances of the stage kernels compiled on their own, their
registers and spills as the assembler reports them."""
import re
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "hypercloudcore.jl_gb300" / "csrc"


def _compile(tmp_path, body):
    """{instance: (registers, spilled bytes)} of the explicit instantiations in `body`, FP32 flags."""
    (tmp_path / "t.cu").write_text('#include "hcc_stage_impl.cuh"\nnamespace hcc {\n' + body + "}\n")
    try:
        r = subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                            "-ftz=true", f"-I{CSRC}", "-Xptxas", "-v", "-c", "t.cu", "-o", "t.o"], cwd=tmp_path, text=True,
                           capture_output=True)
    except FileNotFoundError:
        pytest.skip("no nvcc")
    assert r.returncode == 0, r.stderr[-2000:]
    out = {}
    for part in r.stderr.split("Compiling entry function")[1:]:
        name = re.search(r"_ZN3hcc\d+([a-z_]+)I(\w+?)E+v", part)
        out[name.group(1) + "<" + ",".join(re.findall(r"L[ib](\d+)E", name.group(2) + "E")) + ">"] = (
            int(re.search(r"Used (\d+) registers", part).group(1)), int(re.search(r"(\d+) bytes spill stores", part).group(1)))
    return out


def _instances(kernel, *args):
    return "".join(f"template __global__ void {kernel}<float, {a}>(const StageArgs<float>);\n" for a in args)


def test_3d_scalar_passes_do_not_spill(tmp_path):
    got = _compile(tmp_path, _instances("k_gather", "3, 1, HCC_PDE_ADVECTION, 2, false", "3, 1, HCC_PDE_ADVECTION, 2, true",
                                        "3, 1, HCC_PDE_ADVECTION, 1, false", "3, 1, HCC_PDE_ADVECTION, 1, true") +
                   _instances("k_flux", "3, 1, HCC_PDE_ADVECTION, 2, false, false", "3, 1, HCC_PDE_ADVECTION, 2, true, false"))
    assert len(got) == 6
    for name, (registers, spilled) in got.items():
        assert spilled == 0 and registers <= (64 if "gather" in name else 72), (name, registers, spilled)


def test_2d_two_variable_reconstruction_keeps_its_warps(tmp_path):
    """Ten blocks of four warps an SM: 48 registers."""
    got = _compile(tmp_path, _instances("k_gather", "2, 2, HCC_PDE_ADVECTION, 1, false", "2, 2, HCC_PDE_ADVECTION, 1, true"))
    assert len(got) == 2
    for name, (registers, spilled) in got.items():
        assert registers <= 51 and spilled <= 80, (name, registers, spilled)


def test_central_passes_take_the_list_in_fp64_only(tmp_path):
    """The FP32 pass reads its slot streams in step with the warps."""
    _compile(tmp_path, "static_assert(central_lists<double>() && !central_lists<float>(), \"lists of the central pass\");\n")


def test_third_order_worklists_of_3d_systems_do_not_spill(tmp_path):
    got = _compile(tmp_path, _instances("k_flux_tiles", "3, 5, HCC_PDE_EULER, 2, false, false", "3, 5, HCC_PDE_EULER, 2, true, false"))
    assert len(got) == 2
    for name, (registers, spilled) in got.items():
        assert spilled == 0, (name, registers, spilled)


def test_limited_reconstruction_of_3d_tiles_does_not_spill(tmp_path):
    got = _compile(tmp_path, "template __global__ void k_gather_tile<3, 5, HCC_PDE_EULER, true>(const StageArgs<float>);\n")
    assert len(got) == 1
    for name, (registers, spilled) in got.items():
        assert spilled == 0, (name, registers, spilled)
