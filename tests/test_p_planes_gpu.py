"""The stage-time p planes, p = M(t)^-1 grad(phi), to the last bit that their arithmetic has."""
import numpy as np
import pytest

from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("N", [64, 512])
def test_from_derivative_planes(torch_cuda, N):
    """float64 arithmetic and one rounding to float32, with the reference's det + 1e-12, also where M is singular or
    nearly so: phi_xx = -1 + 2^-j and -1 itself, at quarter times, where numpy's float64 formula is exact up to the
    1e-12 and the quotient.  Tolerance: half a float32 unit (2^-24), and 2^-44 for both sides' float64 roundings."""
    torch = torch_cuda
    from cmblensing_b200 import engine
    n = 2
    plan = engine.get_plan(N, 1, R.pix_width_of(2.0))
    rng = np.random.default_rng(5)
    d = np.zeros((5, N, N), dtype=np.float32)
    d[0], d[1] = rng.uniform(0.5, 2.0, (2, N, N))
    j = rng.integers(0, 25, (N, N))
    d[2] = np.where(j == 24, -1.0, -1.0 + 2.0 ** -np.minimum(j, 23)).astype(np.float32)
    d[2, 0] = -1.0
    f = torch.zeros((1, 1, N, N), dtype=torch.float32, device="cuda")
    base = plan.workspace_bytes(1, False)
    ws = torch.empty(plan.workspace_bytes(1, False, n), dtype=torch.uint8, device="cuda")
    plan.lense_flow(f, torch.as_tensor(d[None], device="cuda"), n=n, workspace=ws)
    pp = ws[base:].view(torch.float32).view(2 * n + 1, 2, N, N).cpu().numpy()
    px, py, pxx = (d[k].astype(np.float64) for k in range(3))
    for k in range(2 * n + 1):
        m = 1.0 + k / (2.0 * n) * pxx
        for got, want in ((pp[k, 0], px / (m + 1e-12)), (pp[k, 1], py * m / (m + 1e-12))):
            err = np.abs(got - want)
            assert np.all(err <= (2.0 ** -24 + 2.0 ** -44) * np.abs(want) + 2.0 ** -50), (k, np.max(err / np.abs(want)))


@pytest.mark.parametrize("N", [64, 256, 1024])
def test_from_phi(torch_cuda, N):
    """The precompute's float32 loop from float64 coefficients, with correctly rounded reciprocals: numpy's float32
    values from the float64 plan's derivatives.  The two float64 derivatives differ in their last bits, which moves a
    float32 rounding in about 2^-25 of the values per coefficient: 1e-4 of them is the bound."""
    torch = torch_cuda
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import gaussian_phi
    n, theta = 3, 2.0
    pw = R.pix_width_of(theta)
    phi = torch.as_tensor(gaussian_phi(N, theta, seed=7)[None], device="cuda")
    p32, p64 = engine.get_plan(N, 1, pw), engine.get_plan(N, 1, pw, "f64")
    planes = torch.empty((1, 5, N, N), dtype=torch.float32, device="cuda")
    pp = p32.phi_pp(phi, n, planes_out=planes)[0].cpu().numpy()
    d = p64.phi_planes(phi)[0].cpu().numpy()
    f32, f64 = np.float32, np.float64
    gx, gy, A, B, C = d
    co = [f32(v) for v in (gx, gy, C * gx - B * gy, A * gy - B * gx, A + C, A * C - B * B)]
    gx, gy, bx, by, lt, qt = (v.astype(f64) for v in co)
    for k in range(2 * n + 1):
        t = f64(f32(k * (1.0 / (2 * n))))
        D = f32(t * f32(t * qt + lt).astype(f64) + 1.0)
        r = f32(1.0 / D.astype(f64)).astype(f64)
        for c, (g, b) in enumerate(((gx, bx), (gy, by))):
            want = f32(f32(t * b + g).astype(f64) * r)
            assert np.mean(pp[k, c] != want) < 1e-4, (k, c, np.mean(pp[k, c] != want))


def test_singular_pixel_is_infinite(torch_cuda):
    """A phi whose determinant is exactly zero at a pixel and time: p is infinite there, with phi_x's sign, not NaN."""
    torch = torch_cuda
    from cmblensing_b200 import engine
    N, n = 64, 2
    pw = R.pix_width_of(3.0)
    k = 2.0 * np.pi / (N * pw)
    x = np.arange(N) * (2.0 * np.pi / N)
    phi = np.repeat((np.sqrt(2.0) / k ** 2 * np.cos(x))[:, None], N, axis=1)  # phi_xx = -sqrt(2) cos x: -1 at x = pi/4
    plan = engine.get_plan(N, 1, pw)
    planes = torch.empty((1, 5, N, N), dtype=torch.float32, device="cuda")
    pp = plan.phi_pp(torch.as_tensor(phi[None], device="cuda"), n, check_det=False, planes_out=planes)[0].cpu().numpy()
    d = planes[0].cpu().numpy()
    for i in (N // 8, N - N // 8):
        hit = d[2, i] == -1.0
        assert hit.any()
        assert np.array_equal(pp[2 * n, 0, i][hit], np.copysign(np.float32(np.inf), d[0, i][hit]))
