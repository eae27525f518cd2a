"""bench.py's line on the finest-level products names the kernel that ran and
the bound it has: matrix-free by its compulsory bytes, whatever shape the outer
product was tuned to, else the stored operator's."""
import pytest

import bench

N_EL, N = 200 * 40 * 40, 201 * 41 * 41
BOX = [8 * N_EL + 32 * N + 24 * N, 8 * N_EL + 16 * N + 24 * N, 8 * N_EL + 68 * N + 12 * N]


@pytest.mark.parametrize("kernel,shape,box,name", [
    (0, 0, True, "k_box_product"), (0, 0, False, "k_mg_spmv_dot_staged<2,3>"), (0, 1, False, "k_mg_spmv_dot_pair"),
    (1, 0, True, "k_box_resid"), (1, 3, True, "k_box_resid"), (1, 0, False, "k_vc_resid_staged"),
    (2, 5, True, "k_box_post"), (2, 0, False, "k_vc_post_staged")])
def test_name_and_bound(kernel, shape, box, name):
    nbytes = BOX[kernel] if box else 3.6e8
    e = bench.finest_product(kernel, shape, 0.05, nbytes, N_EL, N, 6801.3, "measured")
    assert e["kernel"].startswith(name + " ")
    assert e["achieved"] == pytest.approx(nbytes / 5e-5 / 1e9)
    if box:
        assert e["bound"] == ("issue" if kernel == 0 else "latency") and e["frac"] is None and e["peak"] is None and e["traffic"] is None
    else:
        assert e["bound"] == "hbm" and e["frac"] == pytest.approx(e["achieved"] / 6801.3)
        assert e["traffic"] == bench.ncu_traffic(kernel)
