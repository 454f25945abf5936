"""Parity of the log-spherical, cylindrical and GR (Kerr-Schild) solvers
with the reference's own GPU build (oracle/_ref/coffee_refgpu_*, compiled
from the reference's field_solver_EZ_spherical.cu,
field_solver_EZ_cylindrical.cu and field_solver_gr_EZ.cu), which is the only
build the reference has of these solvers.

Each case runs the same input through the reference's float and double
builds and through coffee_b200 in FP32; the FP32 result must sit within the
float build's own distance from the double build (tests/helpers.fp32_parity).
The numpy restatements (oracle/axisym_oracle.py, oracle/gr_oracle.py) are
checked against the double build in the same runs.
"""
from __future__ import annotations

import os

import numpy as np
import pytest

from coffee_b200 import problems
from coffee_b200._lib import COFFEE_E_TIMEOUT, CoffeeError
from coffee_b200.solver import FieldSolverEZCylindrical, FieldSolverEZSpherical, \
    FieldSolverGrEZ, SimData, SimEnvironment, SphBatch
from helpers import fp32_parity, rel_l2
from oracle import axisym_oracle as axo
from oracle import gr_oracle
from oracle import oracle

pytestmark = pytest.mark.gpu


def _need_refgpu():
    for dt in (np.float32, np.float64):
        if not os.path.exists(oracle.refgpu_binary(dt)):
            pytest.skip(f"{oracle.refgpu_binary(dt)} missing: it takes a checkout of the reference "
                        "(make -C oracle gpuref REF=<checkout>)")


def _run_ours(cls, p, fields32, nsteps, aux=False, dtype=np.float32):
    env = SimEnvironment(p)
    data = SimData(env, dtype)
    data.upload(fields32)
    solver = cls(data, env)
    if aux:
        solver.set_aux(True)
    solver.step(0.0, nsteps)
    out = data.download()
    auxo = data.download(("Jx", "Jy", "Jz", "divE", "divB")) if aux else None
    solver.close()
    data.close()
    env.close()
    return out, auxo


def _compare(tag, out, r32, r64, np64=None):
    ok, rep = fp32_parity(out, r32, r64)
    print(f"--- {tag}\n{rep}")
    assert ok, f"{tag}: FP32 parity with the reference GPU build failed\n{rep}"
    if np64 is not None:
        worst = max(rel_l2(np64[f], r64[f]) for f in range(7))
        print(f"numpy restatement vs reference double build: {worst:.2e}")
        assert worst < 1e-9, f"{tag}: numpy restatement departs from the reference ({worst:.2e})"


SPH_CASES = {
    # dipole star with a spin perturbation, absorbing layer, geometric KO
    "sph_pulsar": dict(),
    # plain KO, E.B damping in the current, one shifted ghost layer
    "sph_plainko_edotb_shift": dict(KO_geometry=False, use_edotb_damping=True, shift_ghost=1),
}


@pytest.mark.parametrize("case", sorted(SPH_CASES))
def test_logsph_matches_reference_gpu_build(case):
    _need_refgpu()
    p = problems.sph_pulsar_params(nr=64, nth=32, guard=4, omega=0.25)
    p.tp_start, p.tp_end, p.dw0, p.thp1, p.thp2 = 0.0, 0.5, 0.1, 0.6, 1.2
    for k, v in SPH_CASES[case].items():
        setattr(p, k, v)
    nsteps = 24
    f64 = problems.sph_pulsar_fields(p, np.float64)
    f32 = [a.astype(np.float32) for a in f64]
    r64, _, _ = oracle.run_reference_gpu("sph", p, f64, nsteps)
    r32, _, _ = oracle.run_reference_gpu("sph", p, f32, nsteps)
    np64 = axo.sph_evolve(p, np.stack([a[0] for a in f64]), nsteps)
    out, _ = _run_ours(FieldSolverEZSpherical, p, f32, nsteps)
    _compare(case, out, r32, r64, [a[None] for a in np64])


CYL_CASES = {
    "cyl_pulsar": dict(),
    "cyl_noclamps": dict(clean_ep=False, check_egb=False, KOeps=0.3),
}


@pytest.mark.parametrize("case", sorted(CYL_CASES))
def test_cylindrical_matches_reference_gpu_build(case):
    _need_refgpu()
    p = problems.cyl_pulsar_params(nR=64, nz=128, guard=3)
    p.tp_start, p.tp_end, p.dw0, p.rpert1, p.rpert2 = 0.0, 2.0, 0.05, 3.0, 6.0
    for k, v in CYL_CASES[case].items():
        setattr(p, k, v)
    nsteps = 24
    f64 = problems.cyl_pulsar_fields(p, np.float64)
    f32 = [a.astype(np.float32) for a in f64]
    r64, _, _ = oracle.run_reference_gpu("cyl", p, f64, nsteps)
    r32, _, _ = oracle.run_reference_gpu("cyl", p, f32, nsteps)
    np64 = axo.cyl_evolve(p, np.stack([a[0] for a in f64]), nsteps)
    out, _ = _run_ours(FieldSolverEZCylindrical, p, f32, nsteps)
    _compare(case, out, r32, r64, [a[None] for a in np64])


GR_CASES = {
    # Wald field around a spin-0.9 hole: outer and inner absorbing layers
    "gr_wald": dict(),
    # without the divergence cleaning terms, one shifted ghost layer
    "gr_wald_noclean_shift": dict(divB_clean=False, shift_ghost=1, guard=[4, 4, 4]),
}


@pytest.mark.parametrize("case", sorted(GR_CASES))
def test_gr_matches_reference_gpu_build(case):
    _need_refgpu()
    p = problems.wald_params(N=40, half_size=5.0, a=0.9, pml=6)
    for k, v in GR_CASES[case].items():
        setattr(p, k, v)
    nsteps = 16
    f64 = problems.wald_fields(p, np.float64)
    f32 = [a.astype(np.float32) for a in f64]
    r64, _, _ = oracle.run_reference_gpu("gr", p, f64, nsteps)
    r32, _, _ = oracle.run_reference_gpu("gr", p, f32, nsteps)
    np64 = gr_oracle.gr_evolve(p, np.stack(f64), nsteps)
    out, _ = _run_ours(FieldSolverGrEZ, p, f32, nsteps)
    _compare(case, out, r32, r64, list(np64))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_gr_eh_from_the_writing_kernel_is_bitwise(dtype, monkeypatch):
    """E and H written by the stage and KO kernels for the next kernel (with
    one E, H pass per call) give bitwise the fields of an E, H pass before
    every stage, over calls of several steps and single steps, with the
    inner and outer absorbing layers active."""
    p = problems.wald_params(N=40, half_size=5.0, a=0.9, pml=6)
    f = [a.astype(dtype) for a in problems.wald_fields(p, np.float64)]

    def run(per_stage):
        monkeypatch.setenv("COFFEE_GR_EH_PER_STAGE", "1" if per_stage else "0")
        env = SimEnvironment(p)
        data = SimData(env, dtype)
        data.upload(f)
        solver = FieldSolverGrEZ(data, env)
        solver.step(0.0, 5)
        solver.step(0.0, 1)
        solver.step(0.0, 3)
        out = data.download()
        solver.close()
        data.close()
        env.close()
        return out

    a, b = run(False), run(True)
    for k in range(7):
        assert np.array_equal(a[k], b[k]), k


def test_gr_tiled_stage_is_bitwise(monkeypatch):
    """The FP32 stage streamed through shared-memory tiles gives bitwise the
    fields of the per-point stage kernel: an 80^3 Wald run (two z chunks of
    the tiled kernel, a ragged last one), both absorbing layers, the
    near-horizon metric table, over several calls."""
    p = problems.wald_params(N=80, half_size=10.0, a=0.9, pml=8)
    f = [a.astype(np.float32) for a in problems.wald_fields(p, np.float64)]

    def run(untiled):
        monkeypatch.setenv("COFFEE_GR_TILED", "0" if untiled else "1")
        env = SimEnvironment(p)
        data = SimData(env, np.float32)
        data.upload(f)
        solver = FieldSolverGrEZ(data, env)
        solver.set_aux(True)
        solver.step(0.0, 3)
        solver.step(0.0, 2)
        out = data.download()
        aux = data.download(("Jx", "Jy", "Jz", "divE", "divB"))
        solver.close()
        data.close()
        env.close()
        return out, aux

    (a, xa), (b, xb) = run(False), run(True)
    for k in range(7):
        assert np.array_equal(a[k], b[k]), k
    for k in range(5):
        assert np.array_equal(xa[k], xb[k]), ("aux", k)


FLAT_CASES = {
    "flat_pulsar": lambda: problems.pulsar_params(N=40, guard=3, half_size=10.0, radius=2.5,
                                                  omega=0.1, pml=6),
    "flat_alfven_periodic": lambda: problems.alfven_params(N=32, guard=3),
}


@pytest.mark.parametrize("case", sorted(FLAT_CASES))
def test_flat_gpu_semantics_matches_reference_gpu_build(case):
    """COFFEE_SEM_GPU_REF against the reference's own field_solver_EZ.cu."""
    from coffee_b200.solver import run_flat
    _need_refgpu()
    p = FLAT_CASES[case]()
    nsteps = 12
    if p.problem == 0:
        f64 = problems.alfven_fields(p, np.float64)
    else:
        f64 = problems.pulsar_fields(p, np.float64)
    f32 = [a.astype(np.float32) for a in f64]
    r64, _, _ = oracle.run_reference_gpu("ez", p, f64, nsteps)
    r32, _, _ = oracle.run_reference_gpu("ez", p, f32, nsteps)
    out, _ = run_flat(p, f32, nsteps, semantics="gpu")
    _compare(case, out, r32, r64)


def test_logsph_rejects_short_theta_guard():
    """guard[1] = 3 with theta reaching pi: the reference's axis boundary
    would write past the array; the library refuses the configuration."""
    p = problems.sph_pulsar_params(nr=32, nth=16, guard=4)
    p.guard = [4, 3, 0]
    env = SimEnvironment(p)
    data = SimData(env, np.float32)
    with pytest.raises(RuntimeError, match="guard"):
        FieldSolverEZSpherical(data, env)


def _batch_runs(dtype, nsteps=7):
    """Three log-spherical runs of different sizes, spins and layers: their
    single-run results after nsteps steps, their initial fields, and a
    (env, data, solver) of each for a batch."""
    cfgs = [dict(nr=64, nth=32, omega=0.2, pml=8), dict(nr=96, nth=48, omega=0.3, pml=0),
            dict(nr=48, nth=24, omega=0.1, pml=6)]
    singles, inits, runs = [], [], []
    for k, cfg in enumerate(cfgs):
        p = problems.sph_pulsar_params(guard=4, **cfg)
        if k == 0:
            p.tp_start, p.tp_end, p.dw0, p.thp1, p.thp2 = 0.0, 0.5, 0.1, 0.6, 1.2
        f = problems.sph_pulsar_fields(p, dtype)
        out, _ = _run_ours(FieldSolverEZSpherical, p, f, nsteps, dtype=dtype)
        singles.append(out)
        inits.append(f)
        env = SimEnvironment(p)
        data = SimData(env, dtype)
        data.upload(f)
        runs.append((env, data, FieldSolverEZSpherical(data, env)))
    return singles, inits, runs


def _check_batch(runs, singles):
    for k, (env, data, solver) in enumerate(runs):
        got = data.download()
        for f in range(7):
            assert np.array_equal(got[f], singles[k][f]), f"run {k} field {f} differs"


def _close_runs(batch, runs):
    batch.close()
    for env, data, solver in runs:
        solver.close()
        data.close()
        env.close()


def test_logsph_batch_equals_single_runs():
    """One launch per phase over runs of different sizes, spins and layers
    gives bitwise the results of stepping each run alone."""
    singles, _, runs = _batch_runs(np.float32)
    batch = SphBatch([r[2] for r in runs])
    info = batch.info()  # the autotuner's choice: any candidate gives the same fields
    assert info["tile"] in ([32, 8], [64, 4], [128, 2], [16, 16]) and info["first_stage_ms"] > 0
    batch.step(3)  # captures the step graph, replays it 3 times
    batch.step(4)  # replays it from the new times
    _check_batch(runs, singles)
    _close_runs(batch, runs)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_logsph_persistent_batch_equals_single_runs(dtype):
    """The persistent mode (one cooperative launch per call, grid-wide
    barriers between the phases) gives bitwise the single runs' results."""
    singles, _, runs = _batch_runs(dtype)
    batch = SphBatch([r[2] for r in runs])
    batch.set_persistent(True)
    batch.step(3)
    batch.step(4)
    _check_batch(runs, singles)
    _close_runs(batch, runs)


def test_logsph_persistent_batch_wait_limit():
    """A barrier wait that runs out ends the persistent launch with
    COFFEE_E_TIMEOUT (one CTA leaves out its first arrival, so the others
    wait for it until the 1 ms limit); the context stays usable and the next
    calls, from the initial fields again, give the single runs' results."""
    singles, inits, runs = _batch_runs(np.float32)
    batch = SphBatch([r[2] for r in runs])
    batch.set_persistent(True)
    batch.set_wait_limit(1_000_000, stall_block=0)
    with pytest.raises(CoffeeError) as err:
        batch.step(2)
    assert err.value.code == COFFEE_E_TIMEOUT and "grid barrier 0" in str(err.value)
    batch.set_wait_limit(2_000_000_000, stall_block=-1)
    for (env, data, solver), f in zip(runs, inits):
        data.upload(f)
    batch.times[:] = 0.0
    batch.step(7)
    _check_batch(runs, singles)
    _close_runs(batch, runs)


@pytest.mark.parametrize("nr,nth,shift,theta", [(33, 4, 0, (0.0, 1.0)), (20, 7, 1, (0.0, 1.0)),
                                                (40, 9, 0, (0.0, 0.5)), (17, 12, 2, (0.3, 0.8)),
                                                (70, 35, 0, (0.5, 1.0))])
def test_logsph_axis_rows(nr, nth, shift, theta):
    """The axis boundary written by the rows next to an axis: every point,
    guards included, equals the restatement's after three steps (FP64), with
    both axes, either or none on the grid, rows beyond the axis in the update
    box (shift_ghost) and as few rows between the axes as are accepted."""
    p = problems.sph_pulsar_params(nr=nr, nth=nth, guard=4 + shift, pml=4)
    p.shift_ghost = shift
    p.lower[1], p.size[1] = theta[0] * np.pi, (theta[1] - theta[0]) * np.pi
    p.dt *= 0.5
    U = np.stack(problems.sph_pulsar_fields(p, np.float64))
    rng = np.random.default_rng(3)
    U[:6] += 0.02 * rng.standard_normal(U[:6].shape) * np.abs(U[3])
    ref = axo.sph_evolve(p, U.copy(), 3)
    env = SimEnvironment(p)
    data = SimData(env, np.float64)
    data.upload(list(U))
    s = FieldSolverEZSpherical(data, env)
    s.step(0.0, 3)
    out = data.download()
    for o in (s, data, env):
        o.close()
    for f in range(7):
        # the metric terms of the rows beside the axis, 1 / (r^3 sin), amplify
        # FP64 roundings by at most 1e4 on these grids
        scale = np.abs(ref[f]).max() + 1e-30
        np.testing.assert_allclose(out[f][0], ref[f], rtol=0, atol=1e-11 * scale)


def _rounding(cls, p, fields, evolve, nsteps):
    """Distance of an FP32 run from the FP64 restatement over that of the FP32
    restatement (plain operations, no fused multiply-adds), per field."""
    f = [np.asarray(a, dtype=np.float32) for a in fields]
    U = np.stack([a.reshape(a.shape[-2:]) if evolve is not gr_oracle.gr_evolve else a for a in f])
    ref, plain = evolve(p, U.astype(np.float64), nsteps), evolve(p, U, nsteps)
    out, _ = _run_ours(cls, p, [a.reshape((1,) * (3 - a.ndim) + a.shape) for a in f], nsteps)
    return [rel_l2(out[c].reshape(ref[c].shape), ref[c]) / rel_l2(plain[c], ref[c])
            for c in range(7)]


def _waves(p, rng, ndim=2):
    """Seven random sums of three plane waves on p's grid."""
    n = [np.arange(p.N[a] + 2 * p.guard[a]) / p.N[a] for a in reversed(range(ndim))]
    x = np.meshgrid(*n, indexing="ij")[::-1]
    return [sum(rng.uniform(0.3, 1) * np.sin(2 * np.pi * sum(rng.integers(1, 4) * q for q in x) +
                                             rng.uniform(0, 6.3)) for _ in range(3))
            for _ in range(7)]


def test_logsph_rounding():
    """The sums of the log-spherical stage and KO pass round no more than they
    have to.  Four seeds, mean: B_theta 0.979, P 0.812; with the metric and
    1 / sqrt(gamma) rounded into the difference weights 1.029 and 0.829."""
    r = []
    for seed in range(4):
        p = problems.sph_pulsar_params(nr=300, nth=170)
        f = problems.sph_pulsar_fields(p, np.float64)
        w = _waves(p, np.random.default_rng(seed))
        scale = np.abs(f[3]) + np.abs(f[4])
        r.append(_rounding(FieldSolverEZSpherical, p,
                           [(a + 0.03 * scale * b)[0] for a, b in zip(f, w)], axo.sph_evolve, 4))
    r = np.mean(r, 0)
    print(r)
    assert r[4] < 1.0 and r[6] < 0.82


def test_cylindrical_rounding():
    """The same of the cylindrical solver, a wave field that is smooth on the
    axis: E_z 0.741, E_phi 0.777; with 1 / delta and 1 / R rounded into the
    weights 0.765 and 0.804."""
    r = []
    for seed in range(4):
        p = problems.cyl_pulsar_params(nR=170, nz=300, radius=0.02)
        p.b0 = 1e-3
        w = _waves(p, np.random.default_rng(seed))
        R = (np.arange(p.N[0] + 2 * p.guard[0]) - p.guard[0]) * p.size[0] / p.N[0]
        odd = R / (np.abs(R) + 2.0)
        r.append(_rounding(FieldSolverEZCylindrical, p,
                           [0.05 * w[0] * odd, 0.05 * w[1], 0.05 * w[2] * odd, 0.1 * w[3] * odd,
                            1 + 0.1 * w[4], 0.1 * w[5] * odd, 0.01 * w[6]], axo.cyl_evolve, 4))
    r = np.mean(r, 0)
    print(r)
    assert r[1] < 0.753 and r[2] < 0.79


@pytest.mark.parametrize("tau", [0.83, 1.3])
@pytest.mark.parametrize("solver", ["logsph", "cyl"])
def test_p_over_tau_is_the_rounded_quotient(solver, tau):
    """P alone, the time step too small for anything else to reach it: five
    stages of dP = A dP - P / tau, P += B dP in FP32 with fused sums and a
    correctly rounded quotient, bit for bit."""
    if solver == "logsph":
        p, cls, box = problems.sph_pulsar_params(nr=64, nth=40), FieldSolverEZSpherical, (8, 24)
        f = problems.sph_pulsar_fields(p, np.float32)
    else:
        p, cls, box = problems.cyl_pulsar_params(nR=64, nz=60), FieldSolverEZCylindrical, (16, 30)
        f = problems.cyl_pulsar_fields(p, np.float32)
    p.tau, p.dt, p.KOeps = float(np.float32(tau)), 1e-12, 0.0
    f[6] = np.random.default_rng(1).uniform(1, 2, f[6].shape).astype(np.float32)
    A = [0, -0.4178904745, -1.192151694643, -1.697784692471, -1.514183444257]
    B = [0.1496590219993, 0.3792103129999, 0.8229550293869, 0.6994504559488, 0.1530572479681]
    # (an FMA through FP64: the products are exact, and a sum that rounds twice is one in 1e8)
    fma = lambda x, y, z: (x.astype(np.float64) * np.float64(np.float32(y)) + z).astype(np.float32)
    P = f[6].copy()
    d = np.zeros_like(P)
    for a, b in zip(A, B):
        d = fma(d, a, -(P / np.float32(tau)))
        P = fma(d, b, P)
    out, _ = _run_ours(cls, p, list(f), 1)
    sl = (0, slice(box[0], -box[0]), slice(box[1], -box[0]))
    assert np.array_equal(out[6][sl], P[sl]), int((out[6][sl] != P[sl]).sum())


def test_gr_rounding():
    """The same of the Kerr-Schild solver, with spacings that differ: P 0.907;
    with 1 / 12 rounded into each axis' 1 / delta and KO sums that start from the
    point's own -60 0.918."""
    r = []
    for seed in range(4):
        p = problems.wald_params(N=40, half_size=12.0, a=0.9, pml=6)
        p.size = [p.size[0], p.size[1] * 0.83, p.size[2] * 1.27]
        p.lower = [-s / 2 - 0.5 * s / 40 for s in p.size]
        w = _waves(p, np.random.default_rng(seed), 3)
        f = problems.wald_fields(p, np.float64)
        r.append(_rounding(FieldSolverGrEZ, p,
                           [a + (0.1 if c != 6 else 0.01) * b for c, (a, b) in enumerate(zip(f, w))],
                           gr_oracle.gr_evolve, 4))
    r = np.mean(r, 0)
    print(r)
    assert r[6] < 0.9125


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_gr_without_cleaning_p_moves_nothing(value):
    """With divB_clean off D and B do not depend on P, also where P is not a
    finite number."""
    p = problems.wald_params(N=24, half_size=5.0, a=0.9, pml=4)
    p.divB_clean = False
    f = [a.astype(np.float32) for a in problems.wald_fields(p, np.float64)]
    ref, _ = _run_ours(FieldSolverGrEZ, p, f, 2)
    f[6] = f[6].copy()
    f[6][9, 14, 20] = value
    out, _ = _run_ours(FieldSolverGrEZ, p, f, 2)
    for c in range(6):
        assert np.array_equal(out[c], ref[c]), c


@pytest.mark.parametrize("n", [(33, 30, 21), (40, 37, 52)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_gr_matches_the_restatement(n, dtype):
    """Boxes with ragged edges, both layers, the near-horizon table and calls
    of one and several steps: FP64 to 1e-12 (some hundred roundings), FP32
    within the FP32 restatement's own distance."""
    p = problems.wald_params(N=40, half_size=5.0, a=0.9, pml=4)
    d = p.size[0] / 40
    p.N = list(n)
    p.size, p.lower = [d * m for m in n], [-d * (m // 2 + 0.5) for m in n]
    f64 = problems.wald_fields(p, np.float64)
    U = np.stack(f64)
    U[:6] += 0.02 * np.stack(_waves(p, np.random.default_rng(4), 3))[:6]
    ref = gr_oracle.gr_evolve(p, U.astype(dtype).astype(np.float64), 4)
    env = SimEnvironment(p)
    data = SimData(env, dtype)
    data.upload(list(U.astype(dtype)))
    solver = FieldSolverGrEZ(data, env)
    solver.step(0.0, 1)
    solver.step(0.0, 3)
    out = data.download()
    for o in (solver, data, env):
        o.close()
    if dtype == np.float64:
        assert max(rel_l2(out[c], ref[c]) for c in range(7)) < 1e-12
    else:
        ok, rep = fp32_parity(out, gr_oracle.gr_evolve(p, U.astype(dtype), 4), ref)
        assert ok, rep
