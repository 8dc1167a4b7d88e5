"""Performance cases of the LenseFlow engine: what its users run, over the sizes the package supports.

A case names one public entry point and its sizes.  Kinds:

  field   ``lense_flow(field, phi)``, the reference-shaped call on one device-resident field
          (components float32, phi a float64 MAP or a FOURIER matrix); the phi is kept between calls.
  kept    ``engine.lense_flow_batch`` on a batch whose phi maps are kept: what CG iterations, posterior
          evaluations and repeated (de)lensing by one potential do.
  fresh   ``Plan.phi_pp`` and ``Plan.lense_flow_pp``: a new potential for every call, as in simulation
          pipelines and the benchmark's step.
  grad    ``engine.lense_flow_ad``, forward and backward: lensed field and the gradients with respect to the
          field and the potential, with the reference's reverse scheme or the exact checkpointed one.
  wiener  ``DeviceWienerFilter.apply_A`` with the float64 operator (true residuals, reference solutions),
          through a pixel mask.
  host    ``engine.HostPipeline``: fields and potentials in pinned host memory, the result back in it.

Fields and potentials are Gaussian random fields with the package's spectra (T 100 uK rms, E 5 uK rms and
B = 0, 2.5 arcmin rms deflection); pixels are 3 arcmin up to 256^2 and 2 arcmin above.
"""
import math

import torch

import cmblensing_b200 as cl
from cmblensing_b200 import engine
from cmblensing_b200 import matrix_operators as mo
from cmblensing_b200.lense_flow import lense_flow
from cmblensing_b200.wf_engine import DeviceWienerFilter

ARCMIN = math.pi / (180.0 * 60.0)


# ------------------------------------------------------------------- cases
def _case(kind, N, C, B, n, direction=1, adjoint=False, precision="f32", basis="map", scheme="reference"):
    return dict(kind=kind, N=N, C=C, B=B, n=n, direction=direction, adjoint=adjoint, precision=precision,
                basis=basis, scheme=scheme)


def listed():
    named = [
        # one small patch lensed at a time: launch latency is all there is
        ("field_t64", _case("field", 64, 1, 1, 7)),
        # the smallest configuration of the benchmark's serving mix, one request, a new potential each time
        ("fresh_t128_b1", _case("fresh", 128, 1, 1, 7)),
        # the reference call with its default ten steps on a temperature + polarisation field, phi in Fourier space
        ("field_tqu256", _case("field", 256, 3, 1, 10, basis="fourier")),
        # a server's batch of small delensing requests
        ("kept_inverse_qu128_b13", _case("kept", 128, 2, 13, 7, direction=-1)),
        # simulating a set of medium maps
        ("fresh_qu256_b48", _case("fresh", 256, 2, 48, 7)),
        # the benchmark's step: 64 independent (QU, phi) pairs at 512^2
        ("fresh_qu512_b64", _case("fresh", 512, 2, 64, 7)),
        # the adjoint half of a Wiener-filter iteration for a batch of eight problems
        ("kept_adjoint_qu512_b8", _case("kept", 512, 2, 8, 7, adjoint=True)),
        # large maps, all three components, an odd batch
        ("fresh_tqu1024_b3", _case("fresh", 1024, 3, 3, 7, basis="fourier")),
        # the differentiation workload: 256^2 IQU forward and reverse
        ("grad_tqu256_b16", _case("grad", 256, 3, 16, 7)),
        # the exact gradient for a sampler's batch of chains
        ("grad_exact_qu128_b6", _case("grad", 128, 2, 6, 10, scheme="exact")),
        # the float64 operator of true-residual refinement, two masked problems
        ("wiener_qu256_b2_f64", _case("wiener", 256, 2, 2, 7, precision="f64")),
        # maps streamed from and to pinned host memory
        ("host_qu512_b12", _case("host", 512, 2, 12, 7)),
    ]
    return [dict(c, name=name) for name, c in named]


# work of the largest listed case in component pixels x RK4 steps, and about how much dearer one is per kind
_MOST = 64 * 2 * 512 ** 2 * 7
_DEARER = {"field": 1, "kept": 1, "fresh": 1.2, "grad": 8, "wiener": 24, "host": 2}


def draw(rng):
    kind = rng.choice(["field", "kept", "kept", "fresh", "fresh", "grad", "wiener", "host"])
    N = rng.choice([64, 128, 128, 256, 256, 512, 512, 1024])
    C = rng.choice([1, 2, 2, 3])
    n = rng.randint(5, 12)
    if kind == "wiener":
        N, C = min(N, 512), min(C, 2)
    if kind == "host":
        N = min(N, 512)
    most = max(1, min(64, int(_MOST / (_DEARER[kind] * C * N * N * n))))
    if kind == "field":
        most = 1
    if kind == "wiener":
        most = min(most, 4)
    if kind == "host":
        most = min(most, 24)
    B = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    adjoint = kind in ("field", "kept", "fresh") and rng.random() < 0.35
    return _case(kind, N, C, max(1, min(B, most)), n,
                 direction=rng.choice([1, 1, -1]) if kind != "wiener" else 1, adjoint=adjoint,
                 precision="f64" if kind == "wiener" or (kind in ("field", "kept") and B * C * N <= 1024
                                                         and rng.random() < 0.3) else "f32",
                 basis="fourier" if kind in ("field", "kept", "fresh") and rng.random() < 0.4 else "map",
                 scheme="exact" if kind == "grad" and rng.random() < 0.5 else "reference")


# ------------------------------------------------------------------ inputs
def _theta(N):
    return 3.0 if N <= 256 else 2.0


def _grid(N, pw, dev):
    kx = 2 * math.pi * torch.fft.fftfreq(N, pw, dtype=torch.float64, device=dev)[:, None]
    ky = 2 * math.pi * torch.fft.rfftfreq(N, pw, dtype=torch.float64, device=dev)
    return kx, ky[None, :]


def _grf(gen, shape, N, pw, spectrum, rms):
    """Gaussian random maps with the isotropic spectrum C(l), scaled to ``rms`` each."""
    dev = gen.device
    kx, ky = _grid(N, pw, dev)
    ell = torch.sqrt(kx ** 2 + ky ** 2)
    safe = torch.where(ell > 0, ell, torch.ones_like(ell))
    amp = torch.where(ell > 0, torch.sqrt(spectrum(safe)), torch.zeros_like(ell))
    white = torch.randn(shape + (N, N), generator=gen, dtype=torch.float64, device=dev)
    m = torch.fft.irfft2(torch.fft.rfft2(white) * amp, s=(N, N))
    return m * (rms / m.square().mean(dim=(-2, -1), keepdim=True).sqrt())


def _angles(N, theta, dev):
    """cos, sin of twice the EB rotation angle on the rfft2 grid (half-axis Nyquist column flipped)."""
    d = math.radians(theta / 60.0)
    lx = 2 * math.pi * torch.fft.rfftfreq(N, d, dtype=torch.float64, device=dev)[None, :].repeat(N, 1)
    ly = 2 * math.pi * torch.fft.fftfreq(N, d, dtype=torch.float64, device=dev)[:, None].repeat(1, N // 2 + 1)
    lx[: N // 2 + 1, -1] *= -1
    a = torch.atan2(lx, ly)
    return torch.cos(2 * a), torch.sin(2 * a)


def _inputs(case, seed):
    """float64 fields (B, C, N, N), potentials (B, N, N) and a white cotangent, on the GPU, from the seed."""
    N, C, B = case["N"], case["C"], case["B"]
    theta = _theta(N)
    pw = theta * ARCMIN
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    phi = _grf(gen, (B,), N, pw, lambda l: 1.0 / (l ** 2 * (l + 1) ** 2 * (1 + (l / 60.0) ** 2)), 1.0)
    kx, ky = _grid(N, pw, phi.device)
    F = torch.fft.rfft2(phi)
    grad2 = (torch.fft.irfft2(1j * kx * F, s=(N, N)) ** 2 + torch.fft.irfft2(1j * ky * F, s=(N, N)) ** 2)
    phi = phi * (2.5 * ARCMIN / grad2.mean(dim=(-2, -1), keepdim=True).sqrt())
    comps = []
    if C in (1, 3):
        comps.append(_grf(gen, (B,), N, pw, lambda l: l ** -2 * torch.exp(-(l / 2500.0) ** 2), 100.0))
    if C in (2, 3):
        E = torch.fft.rfft2(_grf(gen, (B,), N, pw, lambda l: l ** -2 * torch.exp(-(l / 2000.0) ** 2), 5.0))
        c2, s2 = _angles(N, theta, phi.device)
        comps += [torch.fft.irfft2(-E * c2, s=(N, N)), torch.fft.irfft2(-E * s2, s=(N, N))]
    f = torch.stack(comps, dim=1).contiguous()
    cot = torch.randn(f.shape, generator=gen, dtype=torch.float64, device=f.device)
    return f, phi.contiguous(), cot, pw


def _basis(case, phi):
    return torch.fft.rfft2(phi).contiguous() if case["basis"] == "fourier" else phi


def _wiener_parts(case, f):
    """Spectra of the problem's operators (float64, (N, N/2+1)) and its pixel mask."""
    N, theta = case["N"], _theta(case["N"])
    pw = theta * ARCMIN
    kx, ky = _grid(N, pw, f.device)
    ell = torch.sqrt(kx ** 2 + ky ** 2)
    safe = torch.where(ell > 0, ell, torch.ones_like(ell))
    scale, width = (100.0, 2500.0) if case["C"] == 1 else (5.0, 2000.0)
    cov = torch.where(ell > 0, safe ** -2 * torch.exp(-(safe / width) ** 2), torch.zeros_like(ell))
    w = torch.full((N // 2 + 1,), 2.0, dtype=torch.float64, device=f.device)
    w[0] = w[-1] = 1.0
    cov = cov * (scale ** 2 * N * N / float((cov * w).sum()))  # per-pixel variance of the map's rms
    sig = 1.0 * ARCMIN / math.sqrt(8 * math.log(2))
    beam = torch.exp(-(ell ** 2) * sig ** 2 / 2)
    beam[0, 0] = 0.0
    noise = torch.full_like(ell, ((10.0 if case["C"] == 1 else 2.0) / theta) ** 2)
    # one apodised square hole per quadrant
    x = torch.arange(N, dtype=torch.float64, device=f.device)
    d = (torch.remainder(x, N / 2) - N / 4).abs()
    edge = torch.clamp((torch.maximum(d[:, None], d[None, :]) - N / 32) / (N / 32), 0.0, 1.0)
    return cov, beam, noise, 0.5 * (1 - torch.cos(math.pi * edge))


# ------------------------------------------------------------- prepare, run
def prepare(case, seed):
    N, C, B, n = case["N"], case["C"], case["B"], case["n"]
    f, phi, cot, pw = _inputs(case, seed)
    kind, prec = case["kind"], case["precision"]
    dt = torch.float64 if prec == "f64" else torch.float32
    s = dict(case=case, pw=pw, n=n)
    if kind == "field":
        kw = dict(nside=N, theta_pix=_theta(N), pix_width=pw)
        m = [f[0, c].to(dt).contiguous() for c in range(C)]
        cls, names = [(cl.FlatS0, ["scalar_matrix"]), (cl.FlatS2, ["polar_matrix_1", "polar_matrix_2"]),
                      (cl.FlatS02, ["scalar_matrix", "polar_matrix_1", "polar_matrix_2"])][C - 1]
        s["field"] = cls(basis=cl.Basis.MAP, **dict(zip(names, m)), **kw)
        s["names"] = names
        s["phi"] = cl.FlatS0(scalar_matrix=_basis(case, phi)[0].contiguous(),
                             basis=cl.Basis.FOURIER if case["basis"] == "fourier" else cl.Basis.MAP, **kw)
    elif kind in ("kept", "fresh"):
        s["f"] = f.to(dt).contiguous()
        s["phi"] = _basis(case, phi)
        if kind == "fresh":
            plan = s["plan"] = engine.get_plan(N, C, pw, prec)
            dev = f.device
            s["pp"] = torch.empty((B, 2 * n + 1, 2, N, N), dtype=torch.float32, device=dev)
            s["out"] = torch.empty_like(s["f"])
            s["ws"] = torch.empty(plan.workspace_bytes(B, case["adjoint"]), dtype=torch.uint8, device=dev)
            s["phi_ws"] = torch.empty(plan.phi_workspace_bytes(B), dtype=torch.uint8, device=dev)
    elif kind == "grad":
        s["f"] = f.to(dt).requires_grad_(True)
        s["phi"] = phi.to(dt).requires_grad_(True)
        s["cot"] = cot.to(dt)
    elif kind == "wiener":
        cov, beam, noise, mask = _wiener_parts(case, f)
        kw = dict(nside=N, theta_pix=_theta(N), pix_width=pw)
        F = torch.fft.rfft2(f)
        if C == 1:
            field = lambda a: cl.FlatS0(scalar_matrix=a[0], **kw)
            op = lambda a, b: mo.DiagonalScalar(scalar_matrix=a, **kw)
        else:
            field = lambda a: cl.FlatS2(polar_matrix_1=a[0], polar_matrix_2=a[1], **kw)
            op = lambda a, b: mo.DiagonalEB(matrix_EE=a, matrix_BB=b, **kw)
        m = mo.PixelMask(mask_map=mask, **kw)
        problems = [dict(phi=cl.FlatS0(scalar_matrix=torch.fft.rfft2(phi[b]), **kw), data=field(F[b]),
                         Cf=op(cov, 0.01 * cov), Cn=op(noise, noise), M=m, B=op(beam, beam)) for b in range(B)]
        s["wf"] = DeviceWienerFilter(problems=problems, n=n, precision=prec)
        s["x"] = F.contiguous()
    else:
        plan = engine.get_plan(N, C, pw, prec)
        s["pipe"] = engine.HostPipeline(plan, B, io_dtype=dt)
        s["f"] = f.to(dt).cpu().pin_memory()
        s["phi"] = phi.cpu().pin_memory()
        s["out"] = torch.empty_like(s["f"]).pin_memory()
    return s


def run(s):
    case = s["case"]
    kind, n, d, adj = case["kind"], s["n"], case["direction"], case["adjoint"]
    if kind == "field":
        out = lense_flow(s["field"], s["phi"], n=n, direction=d, adjoint=adj, precision=case["precision"])
        return [getattr(out, k) for k in s["names"]]
    if kind == "kept":
        return engine.lense_flow_batch(s["f"], s["phi"], s["pw"], n=n, direction=d, adjoint=adj,
                                       precision=case["precision"])
    if kind == "fresh":
        s["plan"].phi_pp(s["phi"], n, check_det=False, out=s["pp"], workspace=s["phi_ws"])
        return s["plan"].lense_flow_pp(s["f"], s["pp"], n, direction=d, adjoint=adj, out=s["out"], workspace=s["ws"])
    if kind == "grad":
        out = engine.lense_flow_ad(s["f"], s["phi"], s["pw"], n=n, direction=d, precision=case["precision"],
                                   scheme=case["scheme"])
        df, dphi = torch.autograd.grad(out, (s["f"], s["phi"]), grad_outputs=s["cot"])
        return {"lensed": out.detach(), "df": df, "dphi": dphi}
    if kind == "wiener":
        return s["wf"].apply_A(s["x"])
    return s["pipe"](s["f"], s["phi"], s["out"], n=n, direction=d)


def work(case):
    """Inputs once, outputs once; the transforms of every RK4 stage (one forward and two inverse real 2-D
    transforms per component, 2.5 log2(N^2) flops a pixel each) and of the potential's derivatives."""
    N, C, B, n, kind = case["N"], case["C"], case["B"], case["n"], case["kind"]
    P = N * N
    el = 8 if case["precision"] == "f64" else 4
    fft = 2.5 * 2 * math.log2(N) * P
    lens = 4 * n * C * 3 * fft
    phi_flops = 6 * fft
    io = 2 * C * el * P
    if kind in ("field", "kept"):  # phi or what was kept of it: five derivatives
        return {"bytes": B * (io + 5 * el * P), "flops": B * lens}
    if kind in ("fresh", "host"):
        return {"bytes": B * (io + 8 * P), "flops": B * (lens + phi_flops)}
    if kind == "grad":  # f, phi, cotangent; lensed, df, dphi; forward lens, and both systems on the way back
        return {"bytes": B * (5 * C + 2) * el * P - B * C * el * P,
                "flops": B * (3 * lens + (5 + 1) * fft + phi_flops)}
    half = 16 * N * (N // 2 + 1)
    operators = 4 * C * 8 * N * (N // 2 + 1)
    return {"bytes": B * (2 * C * half + 5 * 8 * P + operators) + 8 * P, "flops": B * (2 * lens + 8 * C * fft)}


# ------------------------------------------------------------ 64-bit values
def _irf(X, N):
    """irfft2 that ignores the imaginary parts of the DC and Nyquist columns after the column transform."""
    X = torch.fft.ifft(X, dim=-2)
    X[..., 0] = X[..., 0].real.to(X.dtype)
    X[..., -1] = X[..., -1].real.to(X.dtype)
    return torch.fft.irfft(X, n=N, dim=-1)


class _Flow:
    """LenseFlow in 64 bits for a batch: (b, C, N, N) fields, phi (b, N, N) or its rfft2."""

    def __init__(self, phi, N, pw):
        self.N = N
        kx, ky = _grid(N, pw, phi.device)
        ky = ky.clone()
        ky[:, -1] *= -1
        self.kx, self.ky = kx, ky
        F = phi if phi.is_complex() else torch.fft.rfft2(phi)
        self.mult = [1j * kx, 1j * ky, -kx * kx + 0j, -kx * ky + 0j, -ky * ky + 0j]
        self.d = [_irf(m * F, N) for m in self.mult]

    def p(self, t):
        """p = M^-1 grad phi and the entries of M^-1, M = 1 + t grad grad phi."""
        px, py, xx, xy, yy = self.d
        a, b, c = 1 + t * xx, t * xy, 1 + t * yy
        inv = 1.0 / (a * c - b * b + 1e-12)
        ixx, ixy, iyy = c * inv, -b * inv, a * inv
        return px * ixx + py * ixy, px * ixy + py * iyy, ixx, ixy, iyy

    def grad(self, y):
        F = torch.fft.rfft2(y)
        return _irf(self.mult[0] * F, self.N), _irf(self.mult[1] * F, self.N)

    def rate(self, t, y, adjoint):
        px, py = [v[:, None] for v in self.p(t)[:2]]
        if not adjoint:
            gx, gy = self.grad(y)
            return px * gx + py * gy
        return _irf(self.mult[0] * torch.fft.rfft2(px * y) + self.mult[1] * torch.fft.rfft2(py * y), self.N)

    def stages(self, t, h, y, adjoint):
        """The four stage inputs and rates of one RK4 step, and its result."""
        u = [y]
        k = []
        for s, c in enumerate((0.0, 0.5, 0.5, 1.0)):
            k.append(self.rate(t + c * h, u[s], adjoint))
            if s < 3:
                u.append(y + (0.5, 0.5, 1.0)[s] * h * k[s])
        return u, y + h * (k[0] + 2 * k[1] + 2 * k[2] + k[3]) / 6

    def lens(self, f, n, direction, adjoint):
        t0 = 0.0 if (direction == 1) != adjoint else 1.0
        h = (1.0 - 2.0 * t0) / n
        for i in range(n):
            f = self.stages(t0 + i * h, h, f, adjoint)[1]
        return f

    def dphi_terms(self, t, u, v):
        """The five maps whose derivatives sum to the delta-phi rate of stage inputs u (field), v (cotangent)."""
        gx, gy = self.grad(u)
        fx, fy = (v * gx).sum(1), (v * gy).sum(1)
        px, py, ixx, ixy, iyy = self.p(t)
        ax, ay = ixx * fx + ixy * fy, ixy * fx + iyy * fy
        return torch.stack([ax, ay, t * px * ax, t * (px * ay + py * ax), t * py * ay])

    def backward(self, f, lensed, cot, n, direction, scheme):
        """(delta f, delta phi map) of the reference's reverse ODE or of the exact transpose of the RK4 steps."""
        t1 = 1.0 if direction == 1 else 0.0
        h = (1.0 - 2.0 * t1) / n  # from t1 back to 1 - t1
        w = (1.0, 2.0, 2.0, 1.0)
        c = (0.0, 0.5, 0.5, 1.0)
        acc = 0.0
        if scheme == "exact":
            ys = [f]
            for i in range(n):
                ys.append(self.stages((1.0 - t1) - i * h, -h, ys[-1], False)[1])
        y, v = lensed, cot
        for i in range(n):
            t = t1 + i * h
            vs, v = self.stages(t, h, v, True)
            if scheme == "exact":
                us = self.stages(t + h, -h, ys[n - 1 - i], False)[0][::-1]
            else:
                us, y = self.stages(t, h, y, False)
            for s in range(4):
                acc = acc + h / 6 * w[s] * self.dphi_terms(t + c[s] * h, us[s], vs[s])
        F = sum(m * torch.fft.rfft2(a) for m, a in zip(self.mult, acc))
        return v, _irf(F, self.N)


def exact(case, seed):
    N, C, B, n, kind = case["N"], case["C"], case["B"], case["n"], case["kind"]
    f, phi, cot, pw = _inputs(case, seed)
    if case["precision"] == "f32":  # the values that the call is given
        f, cot = f.float().double(), cot.float().double()
        if kind == "grad":
            phi = phi.float().double()
    phi = _basis(case, phi)
    if kind == "wiener":
        return _exact_wiener(case, f, phi, pw)
    outs = []
    step = max(1, (1 << 22) // (C * N * N))
    for b in range(0, B, step):
        flow = _Flow(phi[b:b + step], N, pw)
        fb = f[b:b + step]
        if kind == "grad":
            out = flow.lens(fb, n, case["direction"], False)
            df, dphi = flow.backward(fb, out, cot[b:b + step], n, case["direction"], case["scheme"])
            outs.append((out, df, dphi))
        else:
            outs.append((flow.lens(fb, n, case["direction"], case["adjoint"]),))
    outs = [torch.cat(v) for v in zip(*outs)]
    if kind == "grad":
        return dict(zip(("lensed", "df", "dphi"), outs))
    if kind == "field":
        return [outs[0][0, c] for c in range(C)]
    return outs[0].cpu() if kind == "host" else outs[0]


def _exact_wiener(case, f, phi, pw):
    """A x = -(R z + Cf^-1 x), z = rfft2(L^T irfft2(W rfft2(L irfft2(R^T x)))), W = R^T B M Cn^-1 M B R."""
    N, C, B, n = case["N"], case["C"], case["B"], case["n"]
    cov, beam, noise, mask = _wiener_parts(case, f)
    x = torch.fft.rfft2(f)
    c2, s2 = _angles(N, _theta(N), f.device)

    def to_eb(q):
        return q if C == 1 else torch.stack([-q[:, 0] * c2 - q[:, 1] * s2, q[:, 0] * s2 - q[:, 1] * c2], 1)

    def to_qu(e):
        return e if C == 1 else torch.stack([-e[:, 0] * c2 + e[:, 1] * s2, -e[:, 0] * s2 - e[:, 1] * c2], 1)

    def masked(q):
        return torch.fft.rfft2(_irf(q, N) * mask)

    covs = torch.stack([cov] if C == 1 else [cov, 0.01 * cov])
    inv = torch.where(covs != 0, 1.0 / torch.where(covs != 0, covs, torch.ones_like(covs)), torch.zeros_like(covs))
    flow = _Flow(torch.fft.irfft2(torch.fft.rfft2(phi), s=(N, N)), N, pw)
    y = torch.fft.rfft2(flow.lens(_irf(to_qu(x), N), n, 1, False))
    t = masked(to_qu(beam * to_eb(y)))
    t = masked(to_qu(to_eb(t) / noise))
    h = to_qu(beam * to_eb(t))
    z = torch.fft.rfft2(flow.lens(_irf(h, N), n, 1, True))
    return -(to_eb(z) + inv * x)
