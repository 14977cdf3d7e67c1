"""Every line length on each axis and layout of the right-hand side's passes: the x kernel's plans and its ragged last
block, the strided kernel's plans, and the pruned (compact) workspace rows against the full ones."""
import numpy as np
import pytest
import torch

from oracle import dnsbox_oracle as O

pytestmark = pytest.mark.gpu
SIZES = (8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 512, 1024)
# the bars of the other right-hand-side tests: FP64 round-off of a transform chain, FP32 likewise
TOL = {"fp64": 1e-12, "fp32": 2e-6}


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))


def rough(g, nx, ny, nz, seed):
    rng = np.random.default_rng(seed)
    return O.state_dealias(g, O.state_project(g, O.state_u2uhat(g, rng.standard_normal((3, nz, ny, nx)))))


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("axis", ["x", "y", "z"])
@pytest.mark.parametrize("n", SIZES)
def test_line_length(n, axis, prec):
    from dnsbox_b200.ops import Box
    nx, ny, nz = {"x": (n, 12, 8), "y": (12, n, 8), "z": (24, 8, n)}[axis]
    kw = dict(nu=2e-3, kCutOff=2.5, Pin=0.1, bandlim=True)
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, tstep_fix=True, **kw))
    uh = rough(g, nx, ny, nz, seed=n)
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec, tstep_fix=True, dt=1e-3, **kw)
    u = b.from_numpy(uh)
    got, _ = b.rhs_nonlinear(u)   # the full passes
    assert rel(got.cpu().numpy(), O.rhs_nonlinear(g, uh)) < TOL[prec]
    b.step(u, 1)                  # the pruned passes
    assert b.step_pruned()
    assert rel(u.cpu().numpy(), O.heun_step(g, uh, 1e-3)) < 2 * TOL[prec]   # two right-hand sides
    b.close()


@pytest.mark.parametrize("nx", [8, 12, 24, 32])
def test_maxima_of_boxes_sharing_a_warp(nx):
    """144 lines a box: a warp's lines (32 P-lane groups at most) cross box boundaries."""
    from dnsbox_b200.ops import Box
    ny = nz = 12
    kw = dict(nx=nx, ny=ny, nz=nz, nu=2e-3, bandlim=False, tstep_fix=True, dt=1e-3)
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, bandlim=False))
    fields = [rough(g, nx, ny, nz, seed=s) * (s + 1) for s in range(3)]
    batch = Box(nbatch=3, **kw)
    u = batch.zeros()
    for i, f in enumerate(fields):
        u[:, i] = torch.from_numpy(f).to(u.device)
    recs = batch.step(u, 1)[0]
    for i, f in enumerate(fields):
        one = Box(**kw)
        v = one.from_numpy(f)
        assert one.step(v, 1)[0]["umax"] == recs[i]["umax"]
        assert torch.equal(v, u[:, i])
        one.close()
    batch.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx", SIZES[:-1])
def test_transposed_term_line_length(nx, prec):
    """The transposed right-hand side at every x length (fused kernel and, at 512 in FP64, the physical fields)."""
    from dnsbox_b200.ops import Box
    ny, nz = 12, 8
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, bandlim=False))
    uh, gr = rough(g, nx, ny, nz, seed=nx), rough(g, nx, ny, nz, seed=nx + 1) * 1e-3
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec, bandlim=False)
    got = b.rhs_nonlinear_vjp(b.from_numpy(uh), b.from_numpy(gr))
    # a chain of transforms for u and one for g: twice the bar of a right-hand side
    assert rel(got.cpu().numpy(), O.rhs_nonlinear_vjp(g, uh, gr)) < 2 * TOL[prec]
    b.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,nbatch", [(96, 40), (192, 20)])
def test_x_kernel_of_many_lines(nx, nbatch, prec):
    """Boxes enough for the split x kernel (two waves of its blocks) against the same boxes one by one (the other one)."""
    from dnsbox_b200.ops import Box
    ny, nz = 12, 48
    kw = dict(nx=nx, ny=ny, nz=nz, precision=prec, nu=2e-3, bandlim=False, tstep_fix=True, dt=1e-3)
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, bandlim=False))
    fields = [rough(g, nx, ny, nz, seed=s) * (s + 1) for s in range(3)]
    batch = Box(nbatch=nbatch, **kw)
    u = batch.zeros()
    for i in range(nbatch):
        u[:, i] = torch.from_numpy(fields[i % 3]).to(u.device, u.dtype)
    recs = batch.step(u, 1)[0]
    for i in range(3):
        one = Box(**kw)
        v = one.from_numpy(fields[i])
        r = one.step(v, 1)[0]
        for j in range(i, nbatch, 3):
            assert rel(u[:, j].cpu().numpy(), v.cpu().numpy()) < 2 * TOL[prec]   # two right-hand sides
            assert np.allclose(recs[j]["umax"], r["umax"], rtol=TOL[prec], atol=0)
        one.close()
    batch.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx", SIZES[:-1])
def test_vanishing_component(nx, prec):
    """A mean flow with w(x, y): the z vorticity is exactly zero where w is not, and (transposed) a cotangent without z
    part; each shares a complex sequence of the x kernels with a nonzero field and must stay zero."""
    from dnsbox_b200.ops import Box
    ny, nz = 12, 8
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, bandlim=False))
    rng = np.random.default_rng(nx)
    w = np.broadcast_to(rng.standard_normal((1, ny, nx)), (nz, ny, nx))
    u = O.state_dealias(g, O.state_u2uhat(g, np.stack([np.zeros_like(w), np.zeros_like(w), w])))
    u[:2, 0, 0, 0] = nx * ny * nz * np.array([0.7, -1.3])   # the mean flow, kept by every mask but dealias's
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec, bandlim=False)
    ub = b.from_numpy(u)
    got, _ = b.rhs_nonlinear(ub)
    assert rel(got.cpu().numpy(), O.rhs_nonlinear(g, u)) < TOL[prec]
    z = b.zeros()
    assert not b.rhs_nonlinear_vjp(ub, z).abs().max().item()   # a zero cotangent: exactly zero
    c = u.copy()
    c[2] = 0
    c[0] = O.state_dealias(g, O.state_u2uhat(g, np.stack([np.roll(w, 3, 1)] * 3)))[0]
    assert rel(b.rhs_nonlinear_vjp(ub, b.from_numpy(c)).cpu().numpy(), O.rhs_nonlinear_vjp(g, u, c)) < 2 * TOL[prec]
    b.close()


@pytest.mark.parametrize("n", [8, 12, 24, 32])
def test_band_energy_in_pass_a(n):
    """The band energy of a box whose pass-A block has fewer threads than a warp (n = 8, 12, 24)."""
    from dnsbox_b200.ops import Box
    kw = dict(nu=2e-3, kCutOff=2.5, Pin=0.1, bandlim=True)
    g = O.Grid(O.Params(nx=24, ny=16, nz=n, **kw))
    uh = rough(g, 24, 16, n, seed=n)
    b = Box(nx=24, ny=16, nz=n, tstep_fix=True, dt=1e-3, **kw)
    u = b.from_numpy(uh)
    assert abs(b.rhs_nonlinear(u)[1] / O.rhs_eband(g, uh) - 1) < 1e-13
    assert abs(b.step(u, 1)[0]["eband"] / O.rhs_eband(g, uh) - 1) < 1e-13
    b.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx", [12, 96, 256, 512])
def test_cut_check_single_mode(nx, prec):
    """One mode at the edges of the kept set decides whether a step prunes: rows of several rounds of the check and
    of a part of one, every component, a value that is not a number."""
    from dnsbox_b200.ops import Box
    ny, nz = 12, 16
    ax, ay, az, nyq = -(-nx // 3), -(-ny // 3), -(-nz // 3), nx // 2   # kept: i < a, n/2, i > n - a
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec, bandlim=False, tstep_fix=True, dt=1e-3)
    kept = [(2, 0, 0, ax - 1), (0, 0, 0, nyq), (1, nz - az + 1, ny // 2, nyq), (2, az - 1, ay - 1, 0)]
    cut = [(0, 0, 0, ax), (2, 0, 0, nyq - 1), (1, az, 0, 0), (2, nz - az, ny // 2, nyq), (0, 0, ny - ay, 0)]
    for at in kept + cut:
        u = b.zeros()
        u[at] = 1e-30 if at in cut else 1.0
        b.step(u, 1, diag=False)
        assert b.step_pruned() == (at in kept), at
    u = b.zeros()
    u[2, 0, 0, nyq - 1] = float("nan")
    b.step(u, 1, diag=False)
    assert not b.step_pruned()
    b.close()


def single_parts(nx, ny, nz, delta):
    """(name, u, g, component): fields whose transposed term's `component` comes from the part of size delta alone,
    which shares a complex sequence of the x kernel with a part of size 1 (u and v, phi_x and phi_y, omega_x and omega_y;
    the products of each likewise)."""
    z, y, x = np.meshgrid(*(2 * np.pi * np.arange(n) / n for n in (nz, ny, nx)), indexing="ij")
    full = lambda *f: np.stack([a + 0 * x for a in f])
    s = np.cos(y) + np.sin(2 * y)
    return [("u", full(np.cos(y), delta * np.cos(x), 0), full(0, 0, s), 2),
            ("phi", full(0, 0, s), full(np.cos(y), delta * np.cos(x) * np.cos(y) * np.cos(z),
                                        delta * np.cos(x) * np.sin(y) * np.sin(z)), 2),
            ("omega", full(0, 0, np.cos(y) + delta * np.cos(x)), full(0, 0, s), 0)]


@pytest.mark.parametrize("prec,delta", [("fp64", 1e-8), ("fp32", 1e-5)])
@pytest.mark.parametrize("nx", SIZES[:-1])
def test_transposed_term_small_parts(nx, prec, delta):
    """Every part of the transposed term to its own precision: the bar of test_transposed_term_line_length for the small
    component alone (a transform rounds the parts of a sequence relative to the larger one: 1e-8 and 1e-3 and more here)."""
    from dnsbox_b200.ops import Box
    ny, nz = 12, 8
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, bandlim=False))
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec, bandlim=False)
    for name, u, c, part in single_parts(nx, ny, nz, delta):
        uh, ch = O.state_u2uhat(g, u), O.state_u2uhat(g, c)
        got = b.rhs_nonlinear_vjp(b.from_numpy(uh), b.from_numpy(ch)).cpu().numpy()
        want = O.rhs_nonlinear_vjp(g, uh, ch)
        assert rel(got[part], want[part]) < 2 * TOL[prec], name
        assert rel(got, want) < 2 * TOL[prec], name
    b.close()


def plane_flow(g, nx, ny, nz, seed):
    """u(x, y), v(x, y), w = 0."""
    rng = np.random.default_rng(seed)
    f = np.broadcast_to(rng.standard_normal((3, 1, ny, nx)), (3, nz, ny, nx)).copy()
    f[2] = 0
    return O.state_dealias(g, O.state_project(g, O.state_u2uhat(g, f)))


@pytest.mark.parametrize("prec,powers", [("fp64", (-300, 300)), ("fp32", (-50, 100))])
@pytest.mark.parametrize("nx", SIZES[:-1])
def test_transposed_term_scales_with_the_cotangent(nx, prec, powers):
    """The transposed term is linear in the cotangent, and a power of two is exact, however far the cotangent is from the
    velocity whose complex sequences it shares; with w = 0 and with a rough field."""
    from dnsbox_b200.ops import Box
    ny, nz = 12, 8
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, bandlim=False))
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec, bandlim=False)
    c = b.from_numpy(rough(g, nx, ny, nz, seed=nx + 1) * 1e-3)
    for uh in (plane_flow(g, nx, ny, nz, seed=nx), rough(g, nx, ny, nz, seed=nx)):
        u = b.from_numpy(uh)
        one = b.rhs_nonlinear_vjp(u, c)
        for k in powers:
            assert torch.equal(b.rhs_nonlinear_vjp(u, c * 2.0 ** k), one * 2.0 ** k), k
    b.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(n, 12, 8) for n in SIZES] + [(96, 192, 96), (192, 96, 128)])
def test_vanishing_w(shape, prec):
    """A velocity without w beside a z vorticity, which share a complex sequence of the x kernels: max |w| is 0."""
    from dnsbox_b200.ops import Box
    nx, ny, nz = shape
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec, bandlim=False, tstep_fix=True, dt=1e-3)
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, bandlim=False))
    u = b.from_numpy(plane_flow(g, nx, ny, nz, seed=nx))
    rec = b.step(u, 1)[0]
    assert rec["umax"][2] == 0.0 and rec["umax"][0] > 0.0
    assert not u[2].abs().max().item()
    b.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny,nz,nbatch", [(96, 96, 96, 2), (96, 48, 48, 8), (192, 48, 96, 3), (192, 192, 192, 2)])
def test_a_box_alone_and_among_others(nx, ny, nz, nbatch, prec):
    """The kernels of a box do not depend on the boxes that share its launch: bit for bit the box alone (the x pass of
    96- and 192-point lines has two kernels)."""
    from dnsbox_b200.ops import Box
    kw = dict(nx=nx, ny=ny, nz=nz, precision=prec, nu=2e-3, bandlim=False, tstep_fix=True, dt=1e-3)
    g = torch.Generator(device="cuda").manual_seed(nx)
    one, batch = Box(**kw), Box(nbatch=nbatch, **kw)
    u = batch.zeros()
    for i in range(nbatch):
        v = one.zeros()
        for c in range(3):
            v[c] = one.r2c(torch.randn(nz, ny, nx, generator=g, device="cuda", dtype=v.dtype.to_real()))
        one.project(v)
        one.dealias(v)
        u[:, i] = v
    first = u[:, 0].clone()
    recs = batch.step(u, 2)
    r = one.step(first, 2)
    assert torch.equal(u[:, 0], first)
    assert [s[0] for s in recs] == r
    one.close()
    batch.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny,nz", [(96, 64, 96), (96, 64, 128), (192, 48, 128), (192, 64, 128)])
def test_x_lines_at_the_split_rule(nx, ny, nz, prec):
    """96- and 192-point lines of boxes of 6144 and of 8192 lines, where the x kernel changes, against the oracle."""
    from dnsbox_b200.ops import Box
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz, bandlim=False))
    uh = rough(g, nx, ny, nz, seed=nx + nz)
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec, bandlim=False)
    got, _ = b.rhs_nonlinear(b.from_numpy(uh))
    assert rel(got.cpu().numpy(), O.rhs_nonlinear(g, uh)) < TOL[prec]
    b.close()


@pytest.mark.parametrize("kcut", [2.5, 6.0, 9.5])
@pytest.mark.parametrize("nz", [8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256])
def test_band_energy_of_every_path(nz, kcut):
    """One band energy: of the operator, the right-hand side and the step record, full and pruned, whatever block adds it
    up (a tail block of pass A, whose threads depend on nz, or a launch of its own); narrow and wide bands."""
    from dnsbox_b200.ops import Box
    kw = dict(nx=24, ny=32, nz=nz, nu=2e-3, kCutOff=kcut, Pin=0.1, bandlim=True, tstep_fix=True, dt=1e-3)
    g = O.Grid(O.Params(nx=24, ny=32, nz=nz, nu=2e-3, kCutOff=kcut, Pin=0.1, bandlim=True))
    uh = rough(g, 24, 32, nz, seed=nz)
    b, full = Box(**kw), Box(prune=False, **kw)
    u, v = b.from_numpy(uh), b.from_numpy(uh)
    want = b.eband(u)
    assert abs(want / O.rhs_eband(g, uh) - 1) < 1e-13
    assert b.rhs_nonlinear(u)[1] == want
    assert b.step(u, 1)[0]["eband"] == want and b.step_pruned()
    assert full.step(v, 1)[0]["eband"] == want and not full.step_pruned()
    b.close()
    full.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("ny,nz", [(8, 8), (12, 96), (96, 128)])
@pytest.mark.parametrize("nx", [8, 12])
def test_transforms_of_short_lines(nx, ny, nz, prec):
    """R2C and C2R whose x lines are two lanes wide, against pocketfft (the round-off bars of the slab transforms)."""
    from dnsbox_b200.ops import Box
    g = O.Grid(O.Params(nx=nx, ny=ny, nz=nz))
    f = np.random.default_rng(nx).standard_normal((nz, ny, nx))
    b = Box(nx=nx, ny=ny, nz=nz, precision=prec)
    tol = 1e-13 if prec == "fp64" else 8e-7
    spec = b.r2c(torch.from_numpy(f).to("cuda", b.zeros().dtype.to_real()))
    assert rel(spec.cpu().numpy(), g.r2c(f)) < tol
    assert rel(b.c2r(spec).cpu().numpy(), f * (nx * ny * nz)) < tol
    b.close()
