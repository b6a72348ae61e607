"""The roofline entries of the bench line name the kernels that run and rate them with their own records (no GPU)."""
import sys

import pytest

from conftest import ROOT

sys.path.insert(0, str(ROOT))
import bench  # noqa: E402

KT = {"flux_ms": 3.0, "flux_launches": 3, "gather_ms": 1.0, "gather_launches": 3, "recompute_ms": 0.1, "recompute_launches": 1,
      "predict_ms": 0.0, "steps": 1}


@pytest.mark.parametrize("D,tiled,flux,gather,key", [
    (2, False, "k_flux<float,2,4,EULER,1>", "k_gather<float,2,4,EULER,1>", "flux_f32_w"),
    (2, True, "k_flux_tile<2,4,EULER>", "k_gather<float,2,4,EULER,1>", "flux_tile_f32_w"),
    (3, True, "k_flux_tile<3,5,EULER>", "k_gather_tile<3,5,EULER>", "flux_f32_w")])
def test_flux_record_is_of_the_pass_that_ran(monkeypatch, D, tiled, flux, gather, key):
    records = {"flux_f32_w": 500.0, "flux_tile_f32_w": 400.0, "gather_f32_w": 300.0}
    monkeypatch.setattr(bench, "recorded_traffic", lambda: {f"{k}_bytes_per_point_stage": v for k, v in records.items()})
    r = bench.roofline_of("w", D, D + 2, 20.0, 1000, KT, 6800.0, "measured", tiled=tiled)
    assert r["kernel"] == flux and r["gather"]["kernel"] == gather
    assert r["traffic"] == records[key] * 1000
    assert ("3d" in r["limiter"]) == (D == 3 and tiled)
    monkeypatch.setattr(bench, "recorded_traffic", lambda: {"flux_f32_w_bytes_per_point_stage": 500.0})
    assert (bench.roofline_of("w", D, D + 2, 20.0, 1000, KT, 6800.0, "measured", tiled=tiled)["traffic"] is None) == (D == 2 and tiled)


@pytest.mark.parametrize("D,n,kernel", [(3, 8000000, "k_flux_split<3,5,EULER,1>"), (2, 1000000, "k_flux<double,2,4,EULER,1>"),
                                        (2, 20000, "k_flux_split<2,4,EULER,1>")])
def test_fp64_flux_kernel(D, n, kernel):
    assert bench.fp64_roofline(D, D + 2, 20.0, n, KT, {"tflops": 1.2, "source": "x"})["kernel"] == kernel
