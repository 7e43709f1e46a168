"""The reference's compiled model (collective V with spin flips) on the
two-pass flip path: parity with the FP64 oracle, the reference's golden FP32
energy trace (examples/outputEnergy.txt, tol 1e-5 as in CMakeLists.txt:1102-1115)
and flip couplings on the spin-glass model."""
import numpy as np
import pytest

from helix_b200 import capi
from helix_b200 import systems as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize("dim", [4, 8, 32, 128])
def test_legacy_model_rhs_and_steps_match_oracle(dim):
    p = S.legacy_spin_glass(dim)
    o = O.Oracle(p)
    with capi.Context(p) as ctx:
        assert ctx.size == 10
        assert ctx.stage_path == "flip"
        rng = np.random.default_rng(dim)
        x = rng.standard_normal((10, dim, dim)) + 1j * rng.standard_normal((10, dim, dim))
        ctx.set_state(x)
        got = ctx.rhs()
        want = o.rhs(x)
        assert np.max(np.abs(got - want)) <= 1e-12 * max(1.0, np.max(np.abs(want)))
        ctx.set_state(np.concatenate([S.initial_rho0(dim)[None], np.zeros((9, dim, dim))]))
        rho, en = ctx.step_trace(15)
    rho_ref, en_ref = o.run(15, trace=True)
    assert np.max(np.abs(rho - rho_ref)) <= TOL
    assert np.max(np.abs(en - en_ref)) <= TOL
    o.close()


def test_legacy_compiled_default_energy_trace(golden, tmp_path):
    """d = 1024, 10 ADOs, dt = 0.1: all 1980 steps against all 1981 rows of the
    reference's golden trace (FP32 reference, tolerance 1e-5), the written
    outputEnergy.txt against the golden lines, and 2 steps against the FP64 oracle."""
    g = golden("legacy_energy_trace.json")
    want = np.array(g["energy"])
    assert want.shape == (1981,)
    steps = want.size - 1
    p = S.legacy_spin_glass(1024)
    with capi.Context(p) as ctx:
        assert ctx.stage_path == "flip"
        e0, tr = ctx.observables()
        assert abs(e0 - want[0]) < 1e-5 and abs(tr - 1.0) < 1e-14
        rho, en = ctx.step_trace(2, rho0=True)
        _, en_rest = ctx.step_trace(steps - 2, rho0=False)
    energies = np.concatenate([[e0], en, en_rest])
    assert np.max(np.abs(energies - want)) < 1e-5
    # the file: same line count, the time column byte for byte, energies within 1e-5
    path = tmp_path / "outputEnergy.txt"
    capi.write_energy_trace(str(path), np.arange(steps + 1) * p.dt, energies)
    lines = path.read_text().splitlines()
    assert len(lines) == want.size
    for mine, ref_t, ref_e in zip(lines, g["time"], want):
        t_txt, e_txt = mine.split(" ")
        assert float(t_txt) == pytest.approx(ref_t, abs=1e-12)
        assert abs(float(e_txt) - ref_e) < 1e-5
    for mine, ref_line in zip(lines, g["lines"]):
        assert mine.split(" ")[0] == ref_line.split(" ")[0]
    o = O.Oracle(p)
    rho_ref, en_ref = o.run(2, trace=True)
    o.close()
    assert np.max(np.abs(rho - rho_ref)) <= TOL
    assert np.max(np.abs(en - en_ref)) <= TOL


def test_flip_coupling_on_spin_glass_matches_oracle():
    """A transverse part in per-spin couplings (V_j = sz_j + 0.3 sx_j) selects the flip path for d = 16."""
    p = S.spin_glass(4, seed=5, depth=2, K=1, h=0.8, dt=0.01)
    for j, b in enumerate(p.baths):
        f = np.zeros(4)
        f[j] = 0.3
        b.v_flip = f
    o = O.Oracle(p)
    rho_ref, en_ref = o.run(20, trace=True)
    with capi.Context(p) as ctx:
        rho, en = ctx.step_trace(20)
    assert np.max(np.abs(rho - rho_ref)) <= TOL
    assert np.max(np.abs(en - en_ref)) <= TOL
    o.close()


def test_large_dim_diagonal_coupling_matches_oracle():
    """d = 128 (> 64) with diagonal couplings (band kernels of hx_large.cu)."""
    p = S.spin_glass(7, seed=3, depth=1, K=1, h=0.5, dt=0.01)
    o = O.Oracle(p)
    rho_ref, en_ref = o.run(5, trace=True)
    with capi.Context(p) as ctx:
        rho, en = ctx.step_trace(5)
    assert np.max(np.abs(rho - rho_ref)) <= TOL
    assert np.max(np.abs(en - en_ref)) <= TOL
    o.close()


def _flip_rhs_exact(u, rows, edges, nu, baths, shift):
    """sum of -i [H, u_n] - g_n u_n - i sum_up [V, u_up] in long double, the operators' diagonals without `shift`,
    which no commutator sees.  baths: (first mode, diagonal, flips); the first entry is H.  Also the sum of the
    absolute values of the coefficients of any element."""
    ld = np.clongdouble
    d = u.shape[-1]
    bits = range(d.bit_length() - 1)
    r = np.arange(d)

    def comm(v, w, x):
        v = (v - shift).astype(np.longdouble)
        y = (v[:, None] - v[None, :]) * x
        for i in bits:
            y = y + np.longdouble(w[i]) * (x[:, r ^ (1 << i), :] - x[:, :, r ^ (1 << i)])
        return y

    def norm(v, w):
        return float(np.max(v) - np.min(v) + 2 * np.sum(np.abs(w)))

    M, H = rows.shape[1], rows.shape[0]
    x = u.astype(ld)
    g = (rows * nu).sum(axis=1).astype(np.longdouble)
    out = -1j * comm(*baths[0][1:], x) - g[:, None, None] * x
    size = norm(*baths[0][1:]) + float(g.max())
    for k, (m0, v, w) in enumerate(baths[1:]):
        m1 = baths[k + 2][0] if k + 2 < len(baths) else M
        for m in range(m0, m1):
            up = edges[:, m]
            ok = up < H
            s = np.zeros_like(x)
            s[ok] = x[up[ok]]
            out = out - 1j * comm(v, w, s)
            size += norm(v, w)
    return out, size


@pytest.mark.parametrize("n", [1, 3, 4, 5, 7, 8])
def test_large_common_part_of_the_diagonals_costs_no_digits(n):
    """H and V_j with a common 2^24 on their diagonals, which no commutator sees
    (bath strengths of 1e-40 leave nothing else of V_j): right-hand side, and
    one step (whole steps in one launch at d <= 32).  Every term is a difference
    times a coefficient, so the error of a right-hand side is at most one
    rounding per operation (64 is more than any element has) of the sum of the
    coefficients times the largest element, and a step's Taylor sum adds those
    of its stages to the rounding of the base."""
    shift, eps = 2.0 ** 24, 2.0 ** -53
    p = S.spin_glass(n, seed=90 + n, depth=2, K=1, h=0.6, dt=0.005)
    p.baths = p.baths[:2]
    rng = np.random.default_rng(n)
    p.h_diag = shift + rng.uniform(-2.0, 2.0, p.dim)
    p.h_flip = rng.uniform(0.2, 1.0, n)
    nu, offsets = [], []
    for b in p.baths:
        b.v_diag = shift + rng.uniform(-1.0, 1.0, p.dim)
        b.v_flip = rng.uniform(0.2, 0.6, n)
        b.zeta = 1e-40
        offsets.append(len(nu))
        nu += list(O.bath_coefficients(b.beta, b.gamma, b.zeta, b.K)["nu"])
    rows, edges = capi.hierarchy_tables(len(nu), p.max_depth)
    M = len(nu)
    rows, edges = np.asarray(rows).reshape(-1, M), np.asarray(edges).reshape(-1, 2 * M)
    ops = [(0, p.h_diag, p.h_flip)] + [(o, b.v_diag, b.v_flip) for o, b in zip(offsets, p.baths)]
    x = rng.standard_normal((len(rows), p.dim, p.dim)) + 1j * rng.standard_normal((len(rows), p.dim, p.dim))

    def rhs(u):
        return _flip_rhs_exact(u, rows, edges, np.array(nu), ops, shift)

    with capi.Context(p) as ctx:
        assert ctx.stage_path == "flip" and ctx.get_info().kernels_per_step == (1 if n <= 5 else 8)
        ctx.set_state(x)
        got = ctx.rhs()
        want, size = rhs(x)
        big = np.max(np.abs(x))
        assert np.max(np.abs(got - want)) <= 64 * eps * size * big
        ctx.step(1)
        total, term, bound = x.astype(np.clongdouble), x.astype(np.clongdouble), 4 * eps * big
        for k in range(1, 5):
            term = rhs(term)[0] * (np.longdouble(p.dt) / k)
            total = total + term
            bound += 64 * eps * big * (p.dt * size) ** k / float(np.prod(range(1, k + 1)))
        assert np.max(np.abs(ctx.state() - total)) <= bound


@pytest.mark.parametrize("n", [1, 2])
def test_thousands_of_small_slabs_take_the_two_passes(n):
    """Couplings with flips at d = 2 and 4: 2925 ADOs run whole steps in one
    launch, 3654 a launch per pass, where barriers over that many CTAs took 72 us a
    step and two passes take 42; both as the oracle has it."""
    for depth, size, per_step in ((24, 2925, 1), (26, 3654, 8)):
        p = S.spin_glass(n, seed=7 + n, depth=depth, K=2, h=0.6, dt=0.002)
        p.baths = p.baths[:1]
        p.baths[0].v_flip = np.full(n, 0.3)
        o = O.Oracle(p)
        rho_ref, en_ref = o.run(3, trace=True)
        o.close()
        with capi.Context(p) as ctx:
            assert ctx.stage_path == "flip" and ctx.size == size and ctx.get_info().kernels_per_step == per_step
            rho, en = ctx.step_trace(3)
        assert np.max(np.abs(rho - rho_ref)) <= TOL and np.max(np.abs(en - en_ref)) <= TOL
