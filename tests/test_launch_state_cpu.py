"""Launch state that belongs to a device: kernel attributes are set where a context's tables are built, and no function
keeps a flag for the whole process that says they were (a second device would miss them)."""
import re

from conftest import ROOT

CSRC = ROOT / "hypercloudcore.jl_gb300" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def test_no_process_wide_flags():
    found = [(p.name, m.group(0).strip()) for p in sorted(CSRC.iterdir())
             for m in re.finditer(r"\bstatic\s+(?:bool|char|int|unsigned|size_t|u?int\d+_t)\s+\w+\s*(?:=[^;]*)?;", _code(p))]
    assert found == []


def test_tile_kernels_are_set_up_with_the_tables():
    code = _code(CSRC / "hcc_stage_impl.cuh")
    body = code[code.index("static cudaError_t tile_setup()"):]
    body = body[:body.index("static const StageOps *ops()")]
    assert code.count("cudaFuncSetAttribute") == body.count("cudaFuncSetAttribute") == 1
    for kernel in ("k_flux_wide", "k_flux_tile", "k_gather_tile", "k_cfl_tile"):
        assert f"allow({kernel}<" in body
    api = _code(CSRC / "hcc_api.cu")
    assert api.count("tile_setup()") == 1 and api.index("tile_setup()") > api.index("hcc_status build_tiles(hcc_ctx *c) {")
