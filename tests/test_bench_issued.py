"""The digit products that the benchmark's roofline counts per multiply-add
follow the split plans' rule on the longest reduction (or the tuned count), not
the model space's size: 15 of five digits above 339, 21 of six up to it."""
import pytest

import bench
import imsrg_gb300 as ig


@pytest.mark.parametrize("emax,ref,ladder", [(4, "O16", 21), (6, "O16", 21), (7, "O16", 15), (7, "He4", 15), (8, "O16", 15)])
def test_issued_products(emax, ref, ladder, monkeypatch):
    monkeypatch.setenv("IMSRG_GB300_TUNING", "off")
    ms = ig.ModelSpace(emax, ref, ref)
    assert bench.issued_products(ms, "ladder") == ladder
    assert bench.issued_products(ms, "zbar") == 21
    ms.set_tuning("ladder.digits", 7)
    assert bench.issued_products(ms, "ladder") == 28
    phases = {"split_gemm_ladder": (1.0, 1)}
    ms.set_tuning("ladder.digits", 0)
    roof = bench.roofline(phases, {"ladder_flops": 1e9}, ms)
    assert roof["issued_bf16_tflops"] == pytest.approx(ladder * roof["achieved"])
