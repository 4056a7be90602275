"""bench.py's roofline of the forward convolutions names the launch that was timed."""

import pytest

import bench


@pytest.mark.parametrize("layers,chain,kernel,n,byts,unit", [(16, True, "chain", 16, 16 * 64 - 32, "TFLOP/s"),
                                                             (5, True, "chain", 4, 4 * 64 - 32, "TFLOP/s"),
                                                             (16, False, "stack", 15, 15 * 128, "GB/s")])
def test_roofline_of_the_timed_launch(layers, chain, kernel, n, byts, unit):
    r = bench.roofline_conv([0.2, 0.4], 800, {"hbm_gbs": 6000.0, "bf16_tflops": 1600.0}, layers=layers, chain=chain)
    assert r["kernel"].startswith(f"conv3x3_{kernel}_kernel") and f"{n} layers" in r["kernel"] and r["unit"] == unit
    assert r["algorithmic_bytes"] == byts * 800 * 800 and r["avg_layer_us"] == round(300.0 / n, 2) and r["launches"] == 2
    want = 2 * 9 * 32 * (5 + 32 * (n - 1)) * 800 * 800 / 3e-4 / 1e12 if chain else byts * 800 * 800 / 3e-4 / 1e9
    assert abs(r["achieved"] - want) < 0.06 and abs(r["frac"] - want / r["peak"]) < 1e-4
