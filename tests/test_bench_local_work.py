"""The pair-domain figures of the benchmark are those of the form that ran: its own flops and kernel."""
import pytest

import bench


@pytest.mark.parametrize("form,precision,flops,kernel", [("cholesky", "fp64", 20e12, "gemm_mma_f64"),
                                                         ("cholesky", "tf32x3", 20e12, "tma_gemm"),
                                                         ("dense", "tf32x3", 9e12, "allext_tf32x3_kernel"),
                                                         ("integral", "fp64", 4e12, "local_integral")])
def test_flops_and_kernel_of_the_form(form, precision, flops, kernel):
    st = {"form": form, "flops": 20e12, "dense_flops": 9e12, "integral_flops": 4e12}
    r = bench.local_work(precision, st, 0.125, 1600.0)
    assert r["flops_per_apply"] == flops and r["roofline"]["achieved"] == pytest.approx(flops / 0.125 / 1e12)
    assert r["roofline"]["kernel"].startswith(kernel)
    assert (r["useful_tflops"] is None) == (form != "cholesky")
