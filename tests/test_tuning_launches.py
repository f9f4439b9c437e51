"""What the autotuner times: the pipelined launch, whose stride it sets, also on a domain
small enough for the launch with every line kept by a warp, which has no stride."""
import pytest

from kernel_names import launched

pytestmark = pytest.mark.gpu


# the 40x20x14 domain fits the resident launch, rows of 530 (270 FP64) cells do not
@pytest.mark.parametrize("prec,nx,ny,nz,kernel", [(1, 40, 20, 14, "float"), (2, 40, 20, 14, "float"),
                                                  (0, 40, 20, 14, "double"), (1, 530, 12, 7, "float"),
                                                  (0, 270, 12, 7, "double")])
def test_every_stride_times_the_pipelined_launch(prec, nx, ny, nz, kernel, tmp_path):
    import amcfd
    import amcfd_decks as D
    d = amcfd.Deck(D.small("tune", nx=nx, ny=ny, nz=nz, steps=2).write(str(tmp_path)))
    made = []
    n = launched(lambda: made.append(amcfd.Solver(d, order=amcfd.ORDER_REDBLACK, precision=prec, autotune=1)))
    assert n[f"sweep_rb_pipe_kernel<{kernel}>"] == 12, n  # three strides, four rounds
    assert not any(k.startswith("sweep_resident_kernel") for k in n), n
    assert made[0].tuning()["pipe_stride"] in (8, 16, 32)
    # and the solve itself is the one the domain calls for
    n = launched(made[0].step)
    resident = nx == 40
    assert any(k.startswith("sweep_resident_kernel") for k in n) == resident, n
    assert (n[f"sweep_rb_pipe_kernel<{kernel}>"] > 0) != resident, n
    made[0].close()
