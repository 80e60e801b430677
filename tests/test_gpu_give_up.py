"""The CTAs of a symmetric solve wait for one another for a bounded time. With no time at all they give up together: the solve
ends with the device error set, the host hears of it, and the next solve is whole."""
import pytest
import torch

from test_gpu_two_sided import _clouds, _dense, cta_limit  # noqa: F401

pytestmark = pytest.mark.gpu


# the kernels of the symmetric steps (operands resident, streamed, tiles of 256 x 256 and 128 x 128); 300 steps: the launch of
# the second table of step records finds what the first one has left
@pytest.mark.parametrize("n,m,d,kernel", [(1900, 1430, 64, 1), (2100, 1950, 200, 2), (2200, 2050, 512, 3), (300, 515, 200, 4)])
def test_solve_that_gives_up(cta_limit, n, m, d, kernel):  # noqa: F811
    from flash_sinkhorn_b200 import _lib
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric
    lib = _lib.load()
    cta_limit(0)
    assert lib.fs_two_sided_kernel(n, m, d, _lib.PREC_FP32) == kernel
    ref = _clouds(n, m, d, seed=40)
    args = [torch.as_tensor(v, dtype=torch.float32).cuda() for v in ref]
    kw = dict(use_epsilon_scaling=False, eps=0.05 * d, allow_tf32=False)
    usual = lib.fs_set_meeting_limit(0)
    try:
        sinkhorn_flashstyle_symmetric(*args, n_iters=300, **kw)
        assert lib.fs_device_error() == 1
        with pytest.raises(_lib.FlashSinkhornError):
            sinkhorn_flashstyle_symmetric(*args, n_iters=300, return_n_iters=True, **kw)
    finally:
        lib.fs_set_meeting_limit(usual)
        torch.cuda.synchronize()
        assert lib.fs_clear_device_error() == 0
    got = sinkhorn_flashstyle_symmetric(*args, n_iters=10, return_prelast=True, **kw)
    want = _dense(*ref, 0.05 * d, 10)
    size = float((ref[0] ** 2).sum(1).max())
    for u, v in zip(got, want):  # potentials of size |x|^2 carry 2^-24 of it per step (100 ulp)
        assert float((u.double() - v).abs().max()) < 1e-5 * size
    assert lib.fs_device_error() == 0
