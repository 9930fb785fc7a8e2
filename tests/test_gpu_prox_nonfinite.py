"""The proximal step of the compressed-sensing OS-EM where a voxel or one of its six neighbours is NaN, infinite
or so large that their sum overflows: the reference's exchange loop decides the order among such values, and
the selected value is its bit for bit.  The first step's operator (one subset, one iteration: the step alone)
and, with the plain OS-EM kernels, whose sums are the oracle's, the later steps' as well."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _image(seed, shape):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.1, 1.0, shape).astype(np.float32)
    for value, share in ((np.nan, 0.03), (np.inf, 0.02), (-np.inf, 0.02), (3.0e38, 0.03), (-3.0e38, 0.03)):
        x[rng.random(shape) < share] = value
    return x


@pytest.mark.parametrize("shape", [(1, 9, 11), (3, 40, 37), (5, 33, 64)])
def test_first_step_on_non_finite_images(gpu_ctx, oracle_lib, shape):
    import xct
    O = oracle_lib
    dN, ny, nx = shape
    lam = 1.0e-2
    x = _image(nx, shape)
    ang = (np.arange(8) * 22.5).astype(np.float32)
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, nx, ang, 1, 1, max_batch=dN)
    d = torch.from_numpy(x).cuda()
    plan.cs_run_device(torch.ones((dN, 8, nx), device="cuda"), d, cs_lambda=lam)
    want = O.ista3d(x, O.cs_lambda(lam))
    assert np.array_equal(d.cpu().numpy(), want, equal_nan=True)
    plan.close()


def test_later_steps_on_non_finite_images(gpu_ctx, oracle_lib):
    import xct
    O = oracle_lib
    dN, n, ss, it, lam = 3, 24, 2, 2, 1.0e-2
    ang = (np.arange(8) * 22.5).astype(np.float32)
    rng = np.random.default_rng(4)
    x = rng.uniform(0.1, 1.0, (dN, n, n)).astype(np.float32)
    meas = rng.uniform(0.5, 2.0, (dN, 8, n)).astype(np.float32)
    meas[:, :, 10] = np.inf  # dead bins: infinite ratios, an infinite band in the OS-EM update
    so = O.subset_order(ss)
    first = O.ista3d(x, O.cs_lambda(lam))
    v = O.osem2(first[0], O.osem1(first[0], meas[0], ang, ss, int(so[1]), order=O.ORDER_GPU), ang, ss, int(so[1]), order=O.ORDER_GPU)
    assert not np.isfinite(v).all() and np.isfinite(v).any()
    plan = xct.OSEMPlan(gpu_ctx, n, n, n, ang, ss, it, max_batch=dN, kernels=xct.KERNELS_PLAIN)
    d = torch.from_numpy(x).cuda()
    plan.cs_run_device(torch.from_numpy(meas).cuda(), d, cs_lambda=lam)
    want = O.cs_osem_run(x, meas, ang, ss, it, lam, order=O.ORDER_GPU)
    assert np.array_equal(d.cpu().numpy(), want, equal_nan=True)
    plan.close()
