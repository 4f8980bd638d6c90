"""Heat conduction with a Dirichlet surface marched on the device (IF-HERK,
test/literate/heatconduction.jl:87-189) against the oracle's dense IF-HERK
march on the same inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import ilm_oracle as O
from geometry import heat_case, oracle_cache


def rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / np.abs(np.asarray(b)).max()


def _setup(dtype, fourier, ds_factor=1.4):
    import torch
    import immersedlayers as il
    og, b = heat_case(ds_factor=ds_factor)
    g = il.PhysicalGrid((-1.28, 1.28), (-1.28, 1.28), og.h)
    prob = il.DirichletHeatConductionProblem(
        g, b, dtype=dtype, phys_params={"diffusivity": 1.0, "Fourier": fourier},
        bc={"exterior": lambda t, x, c, p, m: il.zeros_surface(c), "interior": lambda t, x, c, p, m: il.ones_surface(c)},
        timestep_func=il.timestep_fourier)
    sys = il.construct_system(prob)
    x, y = og.coords(O.NODES_PRIMAL)
    T0 = np.exp(-(x[:, None] ** 2 + y[None, :] ** 2) / 0.2 ** 2)
    u0 = il.init_sol(sys)
    u0.state.set_numpy(T0)
    return il, og, b, sys, u0, T0


@pytest.mark.parametrize("dtype_name,fourier", [("f64", 0.5), ("f64", 1.0), ("f32", 0.5)])
def test_heat_march_matches_oracle(cuda, dtype_name, fourier):
    import torch
    dtype = torch.float64 if dtype_name == "f64" else torch.float32
    il, og, b, sys, u0, T0 = _setup(dtype, fourier)
    integ = il.init(u0, (0.0, 1.0), sys, tol=1e-12, maxiter=500)
    nsteps = 8
    integ.step_(nsteps * integ.dt)
    torch.cuda.synchronize()
    assert abs(integ.t - nsteps * integ.dt) < 1e-15
    oc = oracle_cache(og, b)
    h = og.h
    T_ref, sig_ref = O.heat_march(oc, T0, np.zeros(oc.N), np.ones(oc.N), 1.0, fourier * h * h, nsteps)
    T = il.temperature(integ).numpy_components()
    sig = integ.u.constraint.numpy()
    info = integ.info()
    assert max(info["rel_residual"]) <= 1e-12, info
    if dtype == torch.float64:
        assert rel(T, T_ref) < 1e-10
        assert rel(sig, -sig_ref) < 1e-8   # the reference's constraint force is -R sigma
        # the surface constraint E T = (T+ + T-)/2 holds after every step
        assert np.abs(O.interpolate_scalar(oc, T) - 0.5).max() < 1e-10
    else:
        assert rel(T, T_ref) < 2e-5
        assert rel(sig, -sig_ref) < 2e-3


def test_heat_unit_spacing(cuda):
    """Points one cell apart (stage Schur condition numbers 30-350)."""
    import torch
    il, og, b, sys, u0, T0 = _setup(torch.float64, 0.5, ds_factor=1.0)
    integ = il.init(u0, (0.0, 1.0), sys, tol=1e-12, maxiter=2000)
    integ.advance(6)
    torch.cuda.synchronize()
    oc = oracle_cache(og, b)
    h = og.h
    T_ref, _ = O.heat_march(oc, T0, np.zeros(oc.N), np.ones(oc.N), 1.0, 0.5 * h * h, 6)
    T = il.temperature(integ).numpy_components()
    assert max(integ.info()["rel_residual"]) <= 1e-12
    assert rel(T, T_ref) < 1e-9
    assert np.abs(O.interpolate_scalar(oc, T) - 0.5).max() < 1e-10


def test_heat_dense_points_range_cg(cuda):
    """Points 0.3 h apart (as in the 4096-point configuration, ds ~ 0.25 h):
    the stage Schur complements have condition numbers 1e11-1e12 and the
    constraint data carry real content at those small eigenvalues, so the
    point-wise constraint is ill-posed (the oracle's own temperature moves by
    ~20% near the surface between least-squares cut-offs 1e-6 and 1e-12).
    Policy: CG on the range with an iteration cap.  Checked: the field away
    from the surface layer agrees with the oracle's full least-squares march,
    and the constraint residual is small."""
    import torch
    il, og, b, sys, u0, T0 = _setup(torch.float64, 0.5, ds_factor=0.3)
    integ = il.init(u0, (0.0, 1.0), sys, tol=1e-10, maxiter=200)
    integ.advance(6)
    torch.cuda.synchronize()
    oc = oracle_cache(og, b)
    h = og.h
    T_ref, _ = O.heat_march(oc, T0, np.zeros(oc.N), np.ones(oc.N), 1.0, 0.5 * h * h, 6)
    T = il.temperature(integ).numpy_components()
    x, y = og.coords(O.NODES_PRIMAL)
    far = np.abs(np.hypot(x[:, None], y[None, :]) - 0.4) > 0.1
    assert np.abs(T - T_ref)[far].max() < 1e-2 * np.abs(T_ref).max()
    assert np.isfinite(T).all()
    # the stage residuals stall at the level the cut-off leaves (a few %)
    assert max(integ.info()["rel_residual"]) < 0.25
    assert np.abs(O.interpolate_scalar(oc, T) - 0.5).max() < 5e-2


def test_heat_warm_start_and_restart(cuda):
    """Two advances of 4 steps equal one advance of 8 (the warm-start state
    carries over between calls; the iteration counts drop once warm)."""
    import torch
    il, og, b, sys, u0, T0 = _setup(torch.float64, 0.5)
    a = il.init(u0, (0.0, 1.0), sys, tol=1e-12)
    a.advance(4)
    it_first = a.info()["iterations"]
    a.advance(4)
    it_warm = a.info()["iterations"]
    b8 = il.init(u0, (0.0, 1.0), sys, tol=1e-12)
    b8.advance(8)
    torch.cuda.synchronize()
    assert rel(a.u.state.numpy_components(), b8.u.state.numpy_components()) < 1e-12
    assert sum(it_warm) <= sum(it_first)
    nnz = a.info()["nnz"]
    assert all(n > 0 for n in nnz) and nnz[3] < nnz[2]


def test_heat_rejects_index_scaling_and_large_steps(cuda):
    import torch
    import immersedlayers as il
    og, b = heat_case()
    g = il.PhysicalGrid((-1.28, 1.28), (-1.28, 1.28), og.h)
    for scaling, fo in ((il.IndexScaling, 0.5), (il.GridScaling, 10.0)):
        prob = il.DirichletHeatConductionProblem(
            g, b, scaling=scaling, phys_params={"diffusivity": 1.0, "Fourier": fo},
            bc={"exterior": lambda c, p: np.zeros(len(c)), "interior": lambda c, p: np.ones(len(c))},
            timestep_func=il.timestep_fourier)
        sys = il.construct_system(prob)
        with pytest.raises((ValueError, il._lib.ILMError)):
            il.init(il.init_sol(sys), (0.0, 1.0), sys)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -100])
@pytest.mark.parametrize("fourier", [0.05, 0.5, 4.0])
def test_heat_integrating_factor_tiles(cuda, fourier, scale):
    """The integrating-factor passes over ragged tiles (133 nodes a side, radii
    from 8 to 29, a block of zeros) where no surface term reaches: one step is
    there exp(Fo L) T with zeros outside.  The scaled field leaves the range of
    the float-float taps, so every tap of it is taken in FP64.  Two passes of at
    most 59 rounded FP64 taps, whose own values agree to some 1e-14: 1e-13."""
    import torch
    import immersedlayers as il
    og, b = heat_case(ds_factor=1.4)
    n = [len(c) for c in og.coords(O.NODES_PRIMAL)]
    T0 = scale * np.random.default_rng(5).standard_normal(n)
    T0[30:, 90:] = 0.0
    zero = lambda t, x, c, p, m: il.zeros_surface(c)
    prob = il.DirichletHeatConductionProblem(
        il.PhysicalGrid((-1.28, 1.28), (-1.28, 1.28), og.h), b, dtype=torch.float64,
        phys_params={"diffusivity": 1.0, "Fourier": fourier}, bc={"exterior": zero, "interior": zero},
        timestep_func=il.timestep_fourier)
    sys = il.construct_system(prob)
    u0 = il.init_sol(sys)
    u0.state.set_numpy(T0)
    integ = il.init(u0, (0.0, 1.0), sys, tol=1e-12, maxiter=500)
    integ.advance(1)
    torch.cuda.synchronize()
    T = il.temperature(integ).numpy_components()
    ref = O.apply_if(T0, fourier)
    x, y = og.coords(O.NODES_PRIMAL)
    reach = 0.4 + (3 + O.heat_kernel_1d(fourier).size // 2) * og.h
    free = np.maximum(np.abs(x)[:, None], np.abs(y)[None, :]) > reach
    assert free.sum() > 300
    assert np.abs(T - ref)[free].max() < 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("scale", [2.0 ** -44, 2.0 ** -50, 2.0 ** -59])
def test_heat_integrating_factor_small_values(cuda, scale):
    """A step is linear, and a power of two changes no FP64 rounding: the step of
    a field times `scale` is the step times `scale`.  Spikes of 1 over values of
    2^-18: their FP64 sums are good to 2^-53 2^-18 = 4e-22 away from the spikes;
    float-float taps (on at most 2%) of 48 bits give as much.  1e-18 is far below
    what values cut to 24 bits would leave (2^-18 2^-23 of 2%, 9e-15)."""
    import torch
    out = []
    for s in (1.0, scale):
        il, og, b, sys, u0, _ = _setup(torch.float64, 0.5)
        x, y = og.coords(O.NODES_PRIMAL)
        T0 = 2.0 ** -18 * np.random.default_rng(6).standard_normal((len(x), len(y)))
        T0[::64, ::32] = 1.0
        prob = il.DirichletHeatConductionProblem(
            sys.base_cache.g, b, dtype=torch.float64, phys_params={"diffusivity": 1.0, "Fourier": 0.5},
            bc={"exterior": lambda t, x, c, p, m: il.zeros_surface(c),
                "interior": lambda t, x, c, p, m: il.zeros_surface(c)}, timestep_func=il.timestep_fourier)
        sys = il.construct_system(prob)
        u0 = il.init_sol(sys)
        u0.state.set_numpy(s * T0)
        integ = il.init(u0, (0.0, 1.0), sys, tol=1e-12, maxiter=500)
        integ.advance(1)
        torch.cuda.synchronize()
        out.append(il.temperature(integ).numpy_components() / s)
    r = O.heat_kernel_1d(0.5).size // 2
    away = np.ones(T0.shape, bool)
    i, j = np.arange(T0.shape[0])[:, None], np.arange(T0.shape[1])[None, :]
    away &= (np.minimum(i % 64, 64 - i % 64) > r) | (np.minimum(j % 32, 32 - j % 32) > r)
    reach = 0.4 + (3 + r) * og.h
    away &= np.maximum(np.abs(x)[:, None], np.abs(y)[None, :]) > reach
    assert away.sum() > 300
    assert np.abs(out[0] - out[1])[away].max() < 1e-18
