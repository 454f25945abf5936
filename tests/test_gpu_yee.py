"""Parity of the staggered (Yee) RK3 solver with the reference's own GPU
build of field_solver.cu (oracle/_ref/coffee_refgpu_*, mode "yee"), the only
build the reference has of it, and its properties at full size.

Each parity case runs the same input through the reference's float and
double builds and through coffee_b200 in FP32; the FP32 result must sit
within the float build's own distance from the double build
(tests/helpers.fp32_parity).  The numpy restatement (oracle/yee_oracle.py)
is checked against the double build in the same runs.

The reference's kernel_check_eGTb_thread rescales E in place while its
neighbours read E (a race between GPU threads); the library reads the E of
before the pass everywhere.  The cases compared with the reference keep
|E| < |B|, where the two readings agree; the case where the rescale fires is
compared with the numpy restatement, which reads E the same way.
"""
from __future__ import annotations

import os

import numpy as np
import pytest

from coffee_b200 import problems
from coffee_b200.solver import FieldSolver, SimData, SimEnvironment
from helpers import fp32_parity, rel_l2
from oracle import oracle
from oracle import yee_oracle as yo

pytestmark = pytest.mark.gpu


def _need_refgpu():
    for dt in (np.float32, np.float64):
        if not os.path.exists(oracle.refgpu_binary(dt)):
            pytest.skip(f"{oracle.refgpu_binary(dt)} missing: it takes a checkout of the reference "
                        "(make -C oracle gpuref REF=<checkout>)")


def _run_ours(p, fields32, nsteps, b0=None, time0=0.0):
    env = SimEnvironment(p)
    data = SimData(env, np.float32)
    data.upload(fields32)
    if b0 is not None:
        data.upload_background(b0)
    s = FieldSolver(data, env)
    s.step(time0, nsteps)
    out = data.download()
    s.close()
    data.close()
    env.close()
    return out


def _wave_case():
    p = problems.alfven_params(N=32, guard=2)
    p.dt = 0.3 / 32
    return p, problems.alfven_plane_wave_fields(p, np.float64, yee=True), None


def _mixed_case():
    """x periodic, y and z not, a weak absorbing layer in y and z, a
    non-uniform background field B0 and smooth perturbations with E = -v x B,
    |E| < |B| / 2 throughout: every guard rule and the B0 term."""
    p = problems.alfven_params(N=24, guard=2)
    p.N = [24, 20, 16]
    p.size = [1.0, 20 / 24, 16 / 24]
    p.periodic_boundary = [True, False, False]
    p.pml = [0, 3, 3]
    p.pmllen = 2
    p.sigpml = 0.02
    p.dt = 0.25 / 24
    rng = np.random.default_rng(7)
    shape = (p.N[2] + 4, p.N[1] + 4, p.N[0] + 4)
    d = [p.size[a] / p.N[a] for a in range(3)]
    z, y, x = [(np.arange(shape[2 - a]) - 2) * d[a] for a in (2, 1, 0)]
    Z, Y, X = np.meshgrid(z, y, x, indexing="ij")

    def smooth(amp):
        f = np.zeros(shape)
        for _ in range(4):
            k = rng.integers(1, 3, 3) * 2 * np.pi
            f += amp * rng.standard_normal() * np.sin(k[0] * X + k[1] * Y + k[2] * Z +
                                                      rng.uniform(0, 6.3))
        return f
    b0 = [0.8 + smooth(0.05), smooth(0.05), -0.2 + smooth(0.05)]
    B = [b0[0] + smooth(0.02), 0.2 + b0[1] + smooth(0.02), -0.1 + b0[2] + smooth(0.02)]
    v = [smooth(0.02), smooth(0.02), smooth(0.02)]
    E = [-(v[1] * B[2] - v[2] * B[1]), -(v[2] * B[0] - v[0] * B[2]),
         -(v[0] * B[1] - v[1] * B[0])]
    return p, [*E, *B, np.zeros(shape)], b0


def _pulsar_case():
    p = problems.pulsar_params(N=40, guard=2, half_size=10.0, radius=2.5, omega=0.1, pml=6)
    p.dt = 0.3 * (20.0 / 40)
    return p, problems.pulsar_fields(p, np.float64, yee=True), None


CASES = {"yee_alfven_wave": _wave_case, "yee_mixed_b0": _mixed_case}


@pytest.mark.parametrize("case", sorted(CASES))
def test_yee_matches_reference_gpu_build(case):
    _need_refgpu()
    p, f64, b0 = CASES[case]()
    nsteps = 12
    f32 = [a.astype(np.float32) for a in f64]
    extra64 = list(b0) if b0 is not None else []
    extra32 = [a.astype(np.float32) for a in extra64]
    r64, _, _ = oracle.run_reference_gpu("yee", p, list(f64) + extra64, nsteps)
    r32, _, _ = oracle.run_reference_gpu("yee", p, f32 + extra32, nsteps)
    out = _run_ours(p, f32, nsteps, b0=extra32 or None)
    ok, rep = fp32_parity(out, r32, r64)
    print(f"--- {case}\n{rep}")
    assert ok, f"{case}: FP32 parity with the reference GPU build failed\n{rep}"
    np64 = yo.yee_evolve(p, np.stack(f64), nsteps, B0=np.stack(b0) if b0 is not None else None)
    worst = max(rel_l2(np64[f], r64[f]) for f in range(6))
    print(f"numpy restatement vs reference double build: {worst:.2e}")
    assert worst < 1e-9, f"{case}: numpy restatement departs from the reference ({worst:.2e})"


def _inner(arrays, m):
    return [a[m:-m, m:-m, m:-m] for a in arrays]


def test_yee_pulsar_matches_reference_gpu_build():
    """Rotating star with an absorbing layer.  The reference's double build
    cannot launch its kernel_boundary_pulsar_E_thread on sm_100a (136
    registers x 512 threads per block: "too many resources requested for
    launch"), so the FP64 arm is the restatement.  Near the outer boundary
    the absorbing layer damps B below E and the reference's racy rescale
    acts; the library is compared with the reference's float build on the
    inner box (10 cells from the boundary, |E| < |B| / 2 there) and with the
    restatement everywhere."""
    _need_refgpu()
    p, f64, _ = _pulsar_case()
    nsteps = 12
    f32 = [a.astype(np.float32) for a in f64]
    r32, _, _ = oracle.run_reference_gpu("yee", p, f32, nsteps)
    np64 = list(yo.yee_evolve(p, np.stack(f64), nsteps))
    np32 = list(yo.yee_evolve(p, np.stack(f32), nsteps))
    out = _run_ours(p, f32, nsteps)
    ok, rep = fp32_parity(out, np32, np64)
    print(f"--- against the restatement, whole grid\n{rep}")
    assert ok, rep
    m = p.guard[0] + 10
    ok, rep = fp32_parity(_inner(out, m), _inner(r32, m), _inner(np64, m))
    print(f"--- against the reference float build, inner box\n{rep}")
    assert ok, rep
    worst = max(rel_l2(a, b) for a, b in zip(_inner(np64, m)[:6], _inner(r32, m)[:6]))
    print(f"restatement (FP64) vs reference float build, inner box: {worst:.2e}")
    assert worst < 1e-4


def test_yee_rescale_matches_restatement():
    """|E| > |B| at many points: the |E| <= |B| rescale and the E_par
    cleaning act; FP32 library against the restatement in FP32 and FP64."""
    p = problems.alfven_params(N=24, guard=2)
    p.dt = 0.25 / 24
    rng = np.random.default_rng(11)
    shape = (28, 28, 28)
    B = [0.5 + 0.2 * rng.standard_normal(shape) for _ in range(3)]
    E = [0.6 * rng.standard_normal(shape) for _ in range(3)]
    f64 = [*E, *B, np.zeros(shape)]
    f64 = [a.astype(np.float64) for a in f64]
    nsteps = 4
    np64 = yo.yee_evolve(p, np.stack(f64), nsteps)
    np32 = yo.yee_evolve(p, np.stack([a.astype(np.float32) for a in f64]), nsteps)
    out = _run_ours(p, [a.astype(np.float32) for a in f64], nsteps)
    ok, rep = fp32_parity(out, list(np32), list(np64))
    print(rep)
    assert ok, rep


def _div_cells(p, B):
    """Cell-centred forward-difference div B of staggered B arrays, float64."""
    inv = [p.N[a] / p.size[a] for a in range(3)]
    bx, by, bz = (np.asarray(b, dtype=np.float64) for b in B)
    return ((bx[:-1, :-1, 1:] - bx[:-1, :-1, :-1]) * inv[0] +
            (by[:-1, 1:, :-1] - by[:-1, :-1, :-1]) * inv[1] +
            (bz[1:, :-1, :-1] - bz[:-1, :-1, :-1]) * inv[2])


def test_yee_divb_and_energy_at_full_size():
    """256^3 plane Alfven wave, 20 steps: the staggered update changes the
    cell-centred div B only by FP32 rounding (the divergence of its discrete
    curl vanishes), the library's div B diagnostic agrees with a host
    recomputation, and the wave keeps its energy."""
    p = problems.alfven_params(N=256, guard=2)
    p.dt = 0.3 / 256
    f = problems.alfven_plane_wave_fields(p, np.float32, yee=True)
    env = SimEnvironment(p)
    data = SimData(env, np.float32)
    data.upload(f)
    s = FieldSolver(data, env)
    w0 = s.total_energy("B") + s.total_energy("E")
    s.step(0.0, 20)
    d_lib = s.diag("divB_l2")
    w1 = s.total_energy("B") + s.total_energy("E")
    s.check_finite()
    B1 = data.download(("Bx", "By", "Bz"))
    s.close()
    data.close()
    env.close()
    g = 2
    inner = (slice(g, -g - 1),) * 3
    div0 = _div_cells(p, f[3:6])[inner]
    div1 = _div_cells(p, B1)[inner]
    dx = p.size[0] / p.N[0]
    change = float(np.abs(div1 - div0).max()) * dx
    host_l2 = float(np.sqrt((_div_cells(p, B1)[(slice(g, g + 256),) * 3] ** 2).sum()))
    print(f"max |d(div B)| dx {change:.3e}; div B L2 library {d_lib:.6e} host {host_l2:.6e}; "
          f"energy {w0:.6e} -> {w1:.6e}")
    assert change < 1e-5, change
    assert abs(d_lib - host_l2) <= 1e-3 * host_l2 + 1e-6
    assert abs(w1 - w0) / w0 < 1e-3


def test_yee_rejects_unsupported_configurations():
    from coffee_b200._lib import CoffeeError
    p = problems.alfven_params(N=16, guard=2)
    p.shift_ghost = 1
    env = SimEnvironment(p)
    data = SimData(env, np.float32)
    with pytest.raises(CoffeeError):
        FieldSolver(data, env)
    data.close()
    env.close()
    p = problems.alfven_params(N=16, guard=2)
    env = SimEnvironment(p)
    data = SimData(env, np.float32)
    s = FieldSolver(data, env)
    with pytest.raises(CoffeeError):
        s.set_aux(True)
    s.close()
    data.close()
    env.close()


# ------------------------------------------------------ Kerr-Schild (field_solver_gr)

GR_CASES = {
    # Wald field around a spin-0.9 hole: inner and outer absorbing layers
    "gryee_wald": dict(),
    # no E_par cleaning, no rescale: the current and the layers alone
    "gryee_wald_noclamps": dict(clean_ep=False, check_egb=False),
    # rescale without cleaning: the cleaned D is never stored
    "gryee_wald_check_only": dict(clean_ep=False),
}


@pytest.mark.parametrize("case", sorted(GR_CASES))
def test_gryee_matches_reference_gpu_build(case):
    """field_solver_gr (evolve_fields_gr) against the reference's float and
    double GPU builds; its rescale reads dD and writes D, so it has no race
    and the whole grid is compared."""
    from coffee_b200.solver import FieldSolverGr
    _need_refgpu()
    p = problems.wald_params(N=24, half_size=4.0, a=0.9, pml=4)
    for k, v in GR_CASES[case].items():
        setattr(p, k, v)
    nsteps = 8
    f64 = problems.wald_fields(p, np.float64, yee=True)
    f32 = [a.astype(np.float32) for a in f64]
    r64, _, _ = oracle.run_reference_gpu("gryee", p, f64, nsteps)
    r32, _, _ = oracle.run_reference_gpu("gryee", p, f32, nsteps)
    env = SimEnvironment(p)
    data = SimData(env, np.float32)
    data.upload(f32)
    s = FieldSolverGr(data, env)
    s.step(0.0, nsteps)
    out = data.download()
    s.close()
    data.close()
    env.close()
    ok, rep = fp32_parity(out, r32, r64)
    print(f"--- {case}\n{rep}")
    assert ok, f"{case}: FP32 parity with the reference GPU build failed\n{rep}"
    np64 = yo.gryee_evolve(p, np.stack(f64), nsteps)
    worst = max(rel_l2(np64[f], r64[f]) for f in range(6))
    print(f"numpy restatement vs reference double build: {worst:.2e}")
    assert worst < 1e-9, f"{case}: numpy restatement departs from the reference ({worst:.2e})"


def _run_ours64(cls, p, f64, nsteps, b0=None):
    env = SimEnvironment(p)
    data = SimData(env, np.float64)
    data.upload(f64)
    if b0 is not None:
        data.upload_background(b0)
    s = cls(data, env)
    s.step(0.0, nsteps)
    out = data.download()
    s.close()
    data.close()
    env.close()
    return out


def test_yee_fp64_matches_reference_double_build():
    """The FP64 build of the staggered solver (the two passes) against the
    reference's double build: the same arithmetic in the same precision."""
    _need_refgpu()
    p, f64, b0 = _mixed_case()
    nsteps = 6
    r64, _, _ = oracle.run_reference_gpu("yee", p, list(f64) + list(b0), nsteps)
    out = _run_ours64(FieldSolver, p, f64, nsteps, b0=b0)
    worst = max(rel_l2(out[f], r64[f]) for f in range(6))
    print(f"FP64 library vs reference double build: {worst:.2e}")
    assert worst < 1e-10


def test_gryee_fp64_matches_reference_double_build():
    from coffee_b200.solver import FieldSolverGr
    _need_refgpu()
    p = problems.wald_params(N=16, half_size=3.0, a=0.9, pml=2)
    f64 = problems.wald_fields(p, np.float64, yee=True)
    nsteps = 4
    r64, _, _ = oracle.run_reference_gpu("gryee", p, f64, nsteps)
    out = _run_ours64(FieldSolverGr, p, f64, nsteps)
    worst = max(rel_l2(out[f], r64[f]) for f in range(6))
    print(f"FP64 library vs reference double build: {worst:.2e}")
    assert worst < 1e-10


def test_yee_one_guard_point():
    """guard = 1, the least the staggered stencils need, against the
    restatement."""
    p = problems.alfven_params(N=16, guard=1)
    p.dt = 0.3 / 16
    f64 = problems.alfven_plane_wave_fields(p, np.float64, yee=True)
    nsteps = 6
    np64 = yo.yee_evolve(p, np.stack(f64), nsteps)
    np32 = yo.yee_evolve(p, np.stack([a.astype(np.float32) for a in f64]), nsteps)
    out = _run_ours(p, [a.astype(np.float32) for a in f64], nsteps)
    ok, rep = fp32_parity(out, list(np32), list(np64))
    print(rep)
    assert ok, rep


@pytest.mark.parametrize("n,periodic", [((5, 7, 6), (True, True, True)),
                                        ((33, 4, 9), (True, False, True)),
                                        ((4, 35, 3), (False, True, False)),
                                        ((2, 3, 2), (True, True, True))])
def test_yee_guard_points_of_small_boxes(n, periodic):
    """Every point, guards included, of boxes smaller than a warp's row and
    of all mixes of axes equals the restatement's after two steps (FP64; the
    bound is the growth of 1e-16 roundings of O(1) terms over six substeps)."""
    p = problems.alfven_params(N=8, guard=2)
    p.N = list(n)
    p.size = [m / 40 for m in n]
    p.periodic_boundary = list(periodic)
    p.dt = 0.2 / 40
    rng = np.random.default_rng(11)
    shape = tuple(m + 4 for m in reversed(n))
    U = np.concatenate([0.05 * rng.standard_normal((3, *shape)),
                        np.array([1.0, 0.3, -0.2]).reshape(3, 1, 1, 1) +
                        0.05 * rng.standard_normal((3, *shape)), np.zeros((1, *shape))])
    ref = yo.yee_evolve(p, U.copy(), 2)
    env = SimEnvironment(p)
    data = SimData(env, np.float64)
    data.upload(list(U))
    s = FieldSolver(data, env)
    s.step(0.0, 2)
    out = data.download()
    for o in (s, data, env):
        o.close()
    for c in range(6):
        np.testing.assert_allclose(out[c], ref[c], rtol=0, atol=1e-12)
