"""Parity of the CUDA field update (through the C ABI) with the oracle.

In its default arithmetic the FP32 CPU-semantics solver computes every
operation of the reference float build in that build's order and rounding,
so where no star or absorbing layer acts its fields must equal the float
build's bit for bit (0 differing points).  Everything else in FP32 (the star
and absorbing boundaries, the GPU semantics, the fast arithmetic) is held to
the bar of helpers.fp32_parity: within max(2e-5, 4 x noise) relative L2 of
the reference float build, per field, where `noise` is the float build's own
distance from the same algorithm in FP64, and no less accurate than the
float build against that FP64 run (up to 2x + 2e-5).  FP64 results must
match the reference FP64 build to 1e-10.
"""
import numpy as np
import pytest

from coffee_b200 import problems
from coffee_b200.solver import FieldSolverEZ, SimData, SimEnvironment, run_flat
from helpers import (NAMES, count_differing, fp32_parity, golden_cases, interior, load_golden,
                     rel_l2, wide_box_case)
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", golden_cases())
def test_golden_fp32(name):
    p, d = load_golden(name)
    aux = "aux_f32" in d
    out, auxo = run_flat(p, list(d["in_f32"]), int(d["steps"]), time0=float(d["time0"]),
                         semantics="cpu", aux=aux)
    ok, rep = fp32_parity(out, d["out_f32"], d["out_f64_l16"])
    assert ok, rep
    if aux:
        sl = interior(p)
        for f in range(5):
            assert rel_l2(auxo[f][sl], d["aux_f32"][f][sl]) < 2e-4, (name, f)


EXACT_CASES = ("alfven16", "noclean16", "turb16")


@pytest.mark.parametrize("name", EXACT_CASES)
def test_golden_fp32_bit_for_bit(name):
    """The float build's fields, J, divE and divB, bit for bit."""
    p, d = load_golden(name)
    aux = "aux_f32" in d
    out, auxo = run_flat(p, list(d["in_f32"]), int(d["steps"]), time0=float(d["time0"]),
                         semantics="cpu", aux=aux)
    for f in range(7):
        assert count_differing(out[f], d["out_f32"][f]) == 0, \
            (name, f, rel_l2(out[f], d["out_f32"][f]))
    if aux:
        sl = interior(p)
        for f in range(5):
            assert count_differing(auxo[f][sl], d["aux_f32"][f][sl]) == 0, (name, "aux", f)


@pytest.mark.parametrize("name", golden_cases())
def test_golden_fp32_fast_arithmetic(name):
    p, d = load_golden(name)
    out, _ = run_flat(p, list(d["in_f32"]), int(d["steps"]), time0=float(d["time0"]),
                      semantics="cpu", arithmetic="fast")
    ok, rep = fp32_parity(out, d["out_f32"], d["out_f64_l16"])
    assert ok, rep


def test_wide_box_bit_for_bit():
    """Both branches of the taper's tanh (a box around the origin) against
    the restatement, which equals the reference float build bit for bit
    (tests/test_oracle.py), and against that build where it is built."""
    p, f32 = wide_box_case()
    out, _ = run_flat(p, f32, 3)
    ref, _ = oracle.run_port(p, f32, 3, taper_lanes=16)
    for f in range(7):
        assert count_differing(out[f], ref[f]) == 0, (f, rel_l2(out[f], ref[f]))
    if oracle.reference_available(np.float32):
        refb, _, _ = oracle.run_reference(p, f32, 3)
        for f in range(7):
            assert count_differing(out[f], refb[f]) == 0, f


@pytest.mark.parametrize("name", golden_cases())
def test_golden_fp64(name):
    p, d = load_golden(name)
    f64 = [a.astype(np.float64) for a in d["in_f32"]]
    out, _ = run_flat(p, f64, int(d["steps"]), time0=float(d["time0"]), semantics="cpu")
    for f in range(7):
        assert rel_l2(out[f], d["out_f64"][f]) < 1e-10, (name, f, rel_l2(out[f], d["out_f64"][f]))


def _check_vs_port(p, f32, steps, semantics, t0=0.0):
    sem = oracle.SEM_CPU_REF if semantics == "cpu" else oracle.SEM_GPU_REF
    ref32, _ = oracle.run_port(p, f32, steps, time0=t0, semantics=sem, taper_lanes=16)
    ref64, _ = oracle.run_port(p, [a.astype(np.float64) for a in f32], steps, time0=t0,
                               semantics=sem, taper_lanes=16)
    out, _ = run_flat(p, f32, steps, time0=t0, semantics=semantics)
    ok, rep = fp32_parity(out, ref32, ref64)
    assert ok, rep
    # guard points hold exactly what the kernels wrote: compare them too
    for f in range(7):
        assert rel_l2(out[f], ref32[f]) <= max(1e-4, 8 * rel_l2(ref32[f], ref64[f])), f


@pytest.mark.parametrize("semantics", ["cpu", "gpu"])
def test_alfven_both_semantics(semantics):
    p = problems.alfven_params(32)
    _check_vs_port(p, problems.alfven_fields(p, np.float32), 6, semantics)


@pytest.mark.parametrize("semantics", ["cpu", "gpu"])
def test_pulsar_absorbing_both_semantics(semantics):
    p = problems.pulsar_params(N=32, half_size=8.0, radius=2.0, omega=0.1, b0=1.0, pml=6)
    p.q11 = 0.05
    p.q12 = 0.02
    p.p1 = 0.3
    _check_vs_port(p, problems.pulsar_fields(p, np.float32), 4, semantics, t0=0.3)


def test_mixed_boundaries_noncubic():
    p = problems.turbulence_params(16)
    p.N = [48, 16, 32]
    p.size = [3.0, 1.0, 2.0]
    p.periodic_boundary = [True, False, True]
    p.pml = [0, 3, 0]
    p.pmllen = 2
    _check_vs_port(p, problems.turbulence_fields(p, np.float32), 5, "cpu")


def test_shift_ghost():
    p = problems.alfven_params(16)
    p.guard = [5, 5, 5]
    p.shift_ghost = 2
    p.periodic_boundary = [True, False, True]
    _check_vs_port(p, problems.alfven_fields(p, np.float32), 3, "gpu")


def test_no_cleaning_no_damping():
    p = problems.turbulence_params(32)
    p.divB_clean = False
    p.use_edotb_damping = False
    p.KOeps = 0.1
    p.clean_ep = False
    p.check_egb = False
    for sem in ("cpu", "gpu"):
        _check_vs_port(p, problems.turbulence_fields(p, np.float32), 4, sem)


def test_config1_alfven128_100_steps():
    """The Alfven-wave configuration at full size and length: 128^3 + 3
    guards, periodic, dt = dx/2, 100 steps, all 7 fields, against the
    reference float build when it is built here (else the restatement, which
    equals it bit for bit): every field within the stated bound of 1e-5
    relative L2, and in fact bit for bit.  The error against the same
    algorithm in FP64 is reported."""
    p = problems.alfven_params(128)
    f32 = problems.alfven_fields(p, np.float32)
    if oracle.reference_available(np.float32):
        ref32, _, _ = oracle.run_reference(p, f32, 100)
    else:
        ref32, _ = oracle.run_port(p, f32, 100, taper_lanes=16)
    ref64, _ = oracle.run_port(p, [a.astype(np.float64) for a in f32], 100, taper_lanes=16)
    out, _ = run_flat(p, f32, 100)
    for f in range(7):
        e32, e64 = rel_l2(out[f], ref32[f]), rel_l2(out[f], ref64[f])
        print(f"field {f}: vs float build {e32:.2e}, vs FP64 {e64:.2e}, "
              f"differing points {count_differing(out[f], ref32[f])}")
        assert e32 <= 1e-5, (f, e32)
        assert count_differing(out[f], ref32[f]) == 0, f


def test_config1_fast_arithmetic():
    """The same configuration in the regrouped (fast) arithmetic: within the
    FP32 noise bar of the reference float build."""
    p = problems.alfven_params(128)
    f32 = problems.alfven_fields(p, np.float32)
    ref32, _ = oracle.run_port(p, f32, 100, taper_lanes=16)
    ref64, _ = oracle.run_port(p, [a.astype(np.float64) for a in f32], 100, taper_lanes=16)
    out, _ = run_flat(p, f32, 100, arithmetic="fast")
    ok, rep = fp32_parity(out, ref32, ref64)
    print(rep)
    assert ok, rep


@pytest.mark.parametrize("name", ["alfven16", "turb16", "wide"])
def test_energy_diagnostics_bit_for_bit(name):
    """The CPU build's energy-change diagnostics (dU_EgtB, dU_Epar, dU_KO and
    the _cum sums from zero) after 3 steps: against the restatement (itself
    bit for bit the reference float build, tests/test_oracle.py) and against
    the reference where it is built, bit for bit on the interior."""
    if name == "wide":
        p, f32 = wide_box_case()
    else:
        p, d = load_golden(name)
        f32 = list(d["in_f32"])
    out, extra = run_flat(p, f32, 3, energy_diag=True)
    dg = [np.zeros_like(f32[0]) for _ in range(6)]
    ref, _ = oracle.run_port(p, f32, 3, taper_lanes=16, diag=dg)
    sl = interior(p)
    for f in range(7):
        assert count_differing(out[f], ref[f]) == 0, (name, f)
    for k in range(6):
        assert count_differing(extra[k][sl], dg[k][sl]) == 0, (name, "dU", k)
    if oracle.reference_available(np.float32):
        _, _, info = oracle.run_reference(p, f32, 3, diag=True)
        for k in range(6):
            assert count_differing(extra[k][sl], info["diag"][k][sl]) == 0, (name, "ref dU", k)


def test_fp64_with_the_float_builds_taper_lanes():
    """FP64 with the float build's 16 taper lanes (coffee_solver_set_taper_lanes)
    is the float build's algorithm without FP32 rounding: it matches the
    restatement in FP64 with 16 lanes (the fixtures' out_f64_l16)."""
    from coffee_b200.solver import FieldSolverEZ, SimData, SimEnvironment
    p, d = load_golden("alfven16")
    env = SimEnvironment(p)
    data = SimData(env, np.float64)
    data.upload([a.astype(np.float64) for a in d["in_f32"]])
    s = FieldSolverEZ(data, env, "cpu")
    s.set_taper_lanes(16)
    s.step(float(d["time0"]), int(d["steps"]))
    out = data.download()
    s.close()
    data.close()
    env.close()
    for f in range(7):
        assert rel_l2(out[f], d["out_f64_l16"][f]) < 1e-12, f


def _ragged_case(n, tiny=False, star=False, dtype=np.float32):
    """A periodic box of any size with smooth waves on B = x-hat (or a star with
    an absorbing layer); with `tiny`, E and P fall from 1 to below the smallest
    normal number across the box, zeros included."""
    if star:
        p = problems.pulsar_params(N=n[0], half_size=8.0, radius=2.1, pml=5)
        d = p.size[0] / p.N[0]
        p.N, p.size = list(n), [d * m for m in n]
        p.p1, p.p3 = 0.6, 0.8
    else:
        p = problems.alfven_params(8)
        p.N = list(n)
        p.size = [m / 32 for m in n]
        p.dt = 0.4 / 32
    g = p.guard
    x = [(np.arange(p.N[a] + 2 * g[a]) - g[a]) / p.N[a] * 2 * np.pi for a in range(3)]
    Z, Y, X = np.meshgrid(x[2], x[1], x[0], indexing="ij")
    if star:
        f = problems.pulsar_fields(p, np.float64)
        f[0:3] = [0.1 * f[3 + (c + 1) % 3] * np.sin(X + c) for c in range(3)]
    else:
        f = [0.2 * np.sin(X + Y + c) * np.cos(Z - c) for c in range(3)]
        f += [(1.0 if c == 0 else 0.0) + 0.3 * np.cos(X - Z + 2 * c) * np.sin(Y + c)
              for c in range(3)]
        f.append(0.05 * np.sin(X + Z))
    if tiny:
        fall = 10.0 ** (-46.0 * (0.5 - 0.5 * np.cos(Z)))
        f = [a if 3 <= c < 6 else a * fall for c, a in enumerate(f)]
    return p, [a.astype(dtype) for a in f]


# FP32 boxes: KO streams above 2.2 million points (the fifth) and the stage above 12
# million (the last)
@pytest.mark.parametrize("n,tiny", [((6, 7, 8), False), ((33, 6, 9), False), ((33, 6, 9), True),
                                    ((31, 40, 20), True), ((161, 129, 107), False),
                                    ((161, 129, 107), True), ((229, 231, 228), True),
                                    ((230, 229, 229), False)])
def test_flat_boxes_of_any_size_bit_for_bit(n, tiny):
    """FP32 boxes with ragged edges in every direction, on both sides of the
    one-point-per-thread limits and with rows of even and odd length, equal the
    restatement bit for bit, also where quotients and derivatives leave the
    range of the straight-line division."""
    p, f = _ragged_case(n, tiny)
    ref, _ = oracle.run_port(p, f, 2, semantics=0, taper_lanes=16)
    out, _ = run_flat(p, f, 2)
    for c in range(7):
        assert count_differing(out[c], ref[c]) == 0, NAMES[c]


@pytest.mark.parametrize("n", [(33, 20, 9), (129, 97, 103)])
@pytest.mark.parametrize("semantics,arithmetic", [("cpu", "fast"), ("gpu", "reference")])
def test_flat_boxes_of_any_size_regrouped(n, semantics, arithmetic):
    """The regrouped arithmetic on the same grids: within FP32 rounding of the
    FP64 restatement (2e-6 relative L2: some tens of roundings over ten stages)."""
    p, f = _ragged_case(n)
    ref, _ = oracle.run_port(p, [a.astype(np.float64) for a in f], 2,
                             semantics=0 if semantics == "cpu" else 1, taper_lanes=16)
    out, _ = run_flat(p, f, 2, semantics=semantics, arithmetic=arithmetic)
    for c in range(7):
        assert rel_l2(out[c], ref[c]) < 2e-6, NAMES[c]


@pytest.mark.parametrize("n,star", [((33, 20, 9), False), ((201, 207, 203), False),
                                    ((40, 42, 41), True), ((72, 70, 69), True)])
def test_flat_fp64_and_star_of_any_size(n, star):
    """FP64 (both kernels) within 1e-12 of the restatement, and the star with its
    absorbing layer in FP32 within the float build's own bar (2e-5)."""
    p, f = _ragged_case(n, star=star, dtype=np.float64)
    ref, _ = oracle.run_port(p, f, 2, semantics=0, taper_lanes=8)
    out, _ = run_flat(p, f, 2)
    for c in range(7):
        assert rel_l2(out[c], ref[c]) < 1e-12, NAMES[c]
    if star:
        f = [a.astype(np.float32) for a in f]
        ref, _ = oracle.run_port(p, f, 2, semantics=0, taper_lanes=16)
        out, _ = run_flat(p, f, 2)
        for c in range(7):
            assert rel_l2(out[c], ref[c]) < 2e-5, NAMES[c]


def test_p_over_tau_beyond_the_straight_line_range():
    """P / tau of 2^64 and more, with P and tau each in the range of the
    straight-line division: bit for bit, and finite, as the IEEE division gives it
    (no cleaning, so that P moves nothing else)."""
    p = problems.alfven_params(16)
    p.divB_clean = False
    p.tau = float(np.float32(6e-5))
    f = problems.alfven_fields(p, np.float32)
    f[6] = (1.12e15 * np.linspace(0.99, 1.0, f[6].size).reshape(f[6].shape)).astype(np.float32)
    ref, _ = oracle.run_port(p, f, 1, semantics=0, taper_lanes=16)
    out, _ = run_flat(p, f, 1)
    assert np.isfinite(ref[6]).all()
    for c in range(7):
        assert count_differing(out[c], ref[c]) == 0, NAMES[c]


@pytest.mark.parametrize("n,periodic", [((3, 4, 5), (True, True, True)),
                                        ((5, 9, 3), (True, False, True)),
                                        ((3, 3, 40), (True, True, True)),
                                        ((34, 4, 6), (False, True, True))])
@pytest.mark.parametrize("energy_diag", [False, True])
def test_periodic_axes_of_fewer_than_two_guard_widths(n, periodic, energy_diag):
    """A point of such an axis has guard images on both sides: every point,
    the guards of the periodic axes included, bit for bit, with both kinds of
    kernels."""
    p, f = _ragged_case((6, 6, 6))
    p.N, p.size, p.periodic_boundary = list(n), [m / 32 for m in n], list(periodic)
    rng = np.random.default_rng(5)
    shape = tuple(m + 6 for m in reversed(n))
    f = [(0.05 * rng.standard_normal(shape) + (1.0 if c == 3 else 0.0)).astype(np.float32)
         for c in range(7)]
    ref, _ = oracle.run_port(p, f, 2, semantics=0, taper_lanes=16)
    out, _ = run_flat(p, f, 2, energy_diag=energy_diag)
    box = tuple(slice(None) if q else slice(3, -3) for q in reversed(periodic))
    for c in range(7):
        assert count_differing(out[c][box], ref[c][box]) == 0, NAMES[c]


@pytest.mark.parametrize("semantics,arithmetic", [("cpu", "reference"), ("cpu", "fast"),
                                                  ("gpu", "reference")])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_without_cleaning_p_moves_nothing(semantics, arithmetic, value):
    """With divB_clean off E and B do not depend on P, also where P is not a
    finite number."""
    p, f = _ragged_case((33, 20, 9))
    p.divB_clean = False
    ref, _ = run_flat(p, f, 2, semantics=semantics, arithmetic=arithmetic)
    f[6] = f[6].copy()
    f[6][7, 11, 20] = value
    out, _ = run_flat(p, f, 2, semantics=semantics, arithmetic=arithmetic)
    for c in range(6):
        assert count_differing(out[c], ref[c]) == 0, NAMES[c]


def _run_kernels(p, f, streaming, semantics="cpu", arithmetic="reference"):
    env = SimEnvironment(p)
    data = SimData(env, f[0].dtype)
    data.upload(f)
    solver = FieldSolverEZ(data, env, semantics)
    solver.set_arithmetic(arithmetic)
    solver.set_streaming(streaming)
    solver.set_aux(True)
    solver.step(0.0, 2)
    out = data.download() + data.download(("Jx", "Jy", "Jz", "divE", "divB"))
    for o in (solver, data, env):
        o.close()
    return out


# rows of odd and even length, a partial last tile in x and y, one z chunk and several
# with a partial last group of planes
@pytest.mark.parametrize("n", [(33, 20, 9), (40, 42, 41), (37, 17, 131), (64, 29, 72)])
@pytest.mark.parametrize("star", [False, True])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("semantics,arithmetic", [("cpu", "reference"), ("cpu", "fast"),
                                                  ("gpu", "reference")])
def test_streaming_kernels_on_small_grids(n, star, dtype, semantics, arithmetic):
    """The streaming kernels, which larger grids run, against those of one point
    per thread, which small ones run: bit for bit in the reference arithmetic; in
    the regrouped one within the roundings of two steps: some tens of 2^-24 or
    2^-53, relative L2, and 100 times that for J, the divergences and P, which with
    the star is a sum of div B from 0 on: each is a difference of terms of |B| / dx
    that cancel to the dipole's truncation error, 1e-2 of them."""
    p, f = _ragged_case(n, star=star, dtype=dtype)
    a = _run_kernels(p, f, False, semantics, arithmetic)
    b = _run_kernels(p, f, True, semantics, arithmetic)
    eps = 2e-6 if dtype == np.float32 else 2e-14
    for c in range(12):
        if arithmetic == "reference" and semantics == "cpu":
            assert count_differing(a[c], b[c]) == 0, c
        else:
            assert rel_l2(a[c], b[c]) < (eps if c < 6 else 100 * eps), c


def test_energy_diagnostics_with_a_star():
    """The FP32 stage kernel of runs with both the boundary code and the
    diagnostics gives the fields of a run without the diagnostics, bit for bit."""
    for n in ((40, 42, 41), (37, 30, 70)):
        p, f = _ragged_case(n, star=True)
        a, _ = run_flat(p, f, 2)
        b, dg = run_flat(p, f, 2, energy_diag=True)
        for c in range(7):
            assert count_differing(a[c], b[c]) == 0, NAMES[c]
        assert all(np.isfinite(d).all() for d in dg)
