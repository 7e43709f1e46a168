"""The small-slab stage kernels against the oracle: small_kernel (hx_small.cu,
d <= 16 with sigma_z couplings, batched neighbour gathers; the default for
those shapes), its one-launch-per-step form small_step_kernel (the stages of
a step separated by grid barriers; HX_SMALL_STEP=0 selects one launch per
stage) and the generic stage_kernel they replace (HX_SMALL_STAGE=0).  RHS
within 1e-12 relative and trajectories within 1e-10 max-abs, the tolerances
of the other parity tests; the two small forms give the same bits."""
import math

import numpy as np
import pytest

from helix_b200 import capi
from helix_b200 import systems as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-10
RHS_TOL = 1e-12


@pytest.mark.parametrize("path", ["small", "generic"])
@pytest.mark.parametrize("n", [1, 2, 3, 4])
def test_small_slab_rhs(monkeypatch, n, path):
    monkeypatch.setenv("HX_SMALL_STAGE", "1" if path == "small" else "0")
    p = S.spin_glass(n, seed=40 + n, depth=3, K=2, h=0.8)
    o = O.Oracle(p)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((o.size, p.dim, p.dim)) + 1j * rng.standard_normal((o.size, p.dim, p.dim))
    want = o.rhs(x)
    o.close()
    with capi.Context(p) as ctx:
        assert ctx.stage_path == path
        ctx.set_state(x)
        got = ctx.rhs()
    assert np.max(np.abs(got - want)) <= RHS_TOL * max(1.0, np.max(np.abs(want)))


def test_small_kernel_c1_trajectory(monkeypatch):
    """C1 (d = 16, 12 modes, L = 3: 455 ADOs): 1000 steps of rho_0(t) and <H>(t)."""
    monkeypatch.setenv("HX_SMALL_STAGE", "1")
    p = S.spin_glass(4, seed=2024, depth=3, K=2, h=1.0, dt=0.01)
    steps = 1000
    o = O.Oracle(p)
    rho_ref, en_ref = o.run(steps, trace=True)
    o.close()
    with capi.Context(p) as ctx:
        assert ctx.size == 455 and ctx.stage_path == "small"
        rho, en = ctx.step_trace(steps)
    assert np.max(np.abs(rho - rho_ref)) <= TOL
    assert np.max(np.abs(en - en_ref)) <= TOL


@pytest.mark.parametrize("n,depth,K,order", [(4, 3, 2, 4), (4, 3, 3, 4), (2, 3, 2, 4), (3, 4, 2, 3), (4, 2, 2, 2)])
def test_small_step_kernel_matches_stage_launches(monkeypatch, n, depth, K, order):
    """One launch per step against one launch per stage: identical states
    after 25 steps (the per-ADO arithmetic is the same), including 969 ADOs
    at d = 16 (several ADOs per CTA) and Horner orders 2 and 3."""
    monkeypatch.setenv("HX_SMALL_STAGE", "1")
    p = S.spin_glass(n, seed=300 + n + depth, depth=depth, K=K, h=0.9, dt=0.01)
    steps = 25
    out = {}
    for form in ("step", "stage"):
        monkeypatch.setenv("HX_SMALL_STEP", "1" if form == "step" else "0")
        with capi.Context(p, order=order) as ctx:
            assert ctx.stage_path == "small"
            kps = ctx.get_info().kernels_per_step
            assert kps == (1 if form == "step" else order)
            rho, en = ctx.step_trace(steps)
            out[form] = (rho, en, ctx.state())
    for a, b in zip(out["step"], out["stage"]):
        assert np.array_equal(a, b)
    o = O.Oracle(p)
    rho_ref, _ = o.run(5, order=order, trace=True)
    o.close()
    assert np.max(np.abs(out["step"][0][:5] - rho_ref)) <= TOL


def test_small_step_kernel_replays_from_a_captured_graph(monkeypatch):
    """The step kernel's grid barrier keeps no host-side count: a CUDA graph
    captured from one hx_ctx_step replays into the same states as steps
    launched one by one."""
    import torch

    monkeypatch.setenv("HX_SMALL_STAGE", "1")
    monkeypatch.setenv("HX_SMALL_STEP", "1")
    p = S.spin_glass(4, seed=2024, depth=3, K=2, h=1.0, dt=0.01)
    steps = 7
    with capi.Context(p) as ref:
        assert ref.get_info().kernels_per_step == 1
        ref.step(steps)
        want = ref.state()
    stream = torch.cuda.Stream()
    with capi.Context(p) as ctx:
        ctx.set_stream(stream.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.step(1)
        for _ in range(steps):
            graph.replay()
        torch.cuda.synchronize()
        ctx.sync()
        got = ctx.state()
        del graph
    assert np.array_equal(got, want)


def test_step_kernel_wait_timeout_is_reported_and_the_context_recovers(monkeypatch):
    """Failure detection without a GPU fault: the injected step waits at its
    first grid barrier for an arrival that never comes, gives up after a short
    poll limit and reports DeviceWaitTimeout; rho is untouched, so the context
    then steps on exactly as one that never failed."""
    monkeypatch.setenv("HX_SMALL_STAGE", "1")
    monkeypatch.setenv("HX_SMALL_STEP", "1")
    p = S.spin_glass(4, seed=2024, depth=3, K=2, h=1.0, dt=0.01)
    with capi.Context(p) as ref:
        ref.step(5)
        want = ref.state()
    with capi.Context(p) as ctx:
        before = ctx.state()
        ctx.inject_wait_timeout()
        ctx.step(1)
        with pytest.raises(capi.HxError) as e:
            ctx.sync()
        assert e.value.status == "DeviceWaitTimeout"
        assert np.array_equal(ctx.state(), before)
        ctx.step(5)
        ctx.sync()
        assert np.array_equal(ctx.state(), want)
    monkeypatch.setenv("HX_SMALL_STEP", "0")
    with capi.Context(p) as plain:  # one launch per stage: no grid-barrier waits to run out
        with pytest.raises(capi.HxError) as e:
            plain.inject_wait_timeout()
        assert e.value.status == "UnsupportedExecution"


@pytest.mark.parametrize("collective", [False, True])
@pytest.mark.parametrize("n,baths,K,depth", [
    (1, 1, 1, 3),   # 10 ADOs at d = 2: one CTA
    (3, 2, 1, 2),   # 15 ADOs, 960 elements: one CTA
    (3, 1, 1, 4),   # 15 ADOs with one bath
    (3, 3, 0, 3),   # 20 ADOs, 1280 elements: the smallest grids, 4 ADOs per CTA
    (4, 3, 1, 4),   # 210 ADOs at d = 16: two slabs per CTA
    (4, 2, 3, 4),   # 495 ADOs, up to 16 entries each
    (4, 4, 3, 3),   # 969 ADOs: several slabs per CTA one after the other, all entries staged
    (4, 4, 6, 2),   # 28 modes, 435 ADOs: more entries than the staging area holds at once
])
def test_whole_step_runs_match_oracle(n, baths, K, depth, collective):
    """Whole steps in one launch, sigma_z and general diagonal couplings, with
    and without records: the trajectory against the oracle, and the recorded
    run equal to the unrecorded one."""
    p = S.spin_glass(n, seed=70 + n, depth=depth, K=K, h=0.8, dt=0.01)
    p.baths = p.baths[:baths]
    if collective:
        rng = np.random.default_rng(n)
        for b in p.baths:
            b.v_diag = rng.uniform(-0.7, 0.7, p.dim)
    steps = 4
    o = O.Oracle(p)
    rho_ref, en_ref = o.run(steps, trace=True)
    want = o.state()
    o.close()
    with capi.Context(p) as a, capi.Context(p) as b:
        # general couplings at d = 16: one round of four slabs in each of 147 CTAs, else a launch per stage
        one = not (collective and n == 4 and a.size > 588)
        assert a.get_info().kernels_per_step == (1 if one else 4)
        rho, en = a.step_trace(steps)
        b.step(steps)
        b.sync()
        assert np.array_equal(a.state(), b.state())
        assert np.max(np.abs(a.state() - want)) <= TOL
    assert np.max(np.abs(rho - rho_ref)) <= TOL
    assert np.max(np.abs(en - en_ref)) <= TOL


@pytest.mark.parametrize("n,baths,K,depth,order,collective", [
    (5, 1, 0, 1, 4, False),   # 2 ADOs
    (5, 5, 2, 2, 4, False),   # 136 ADOs: one per SM, kept in registers
    (5, 4, 3, 2, 3, True),    # 153 ADOs: just more than one per SM
    (5, 5, 1, 3, 2, False),   # 286 ADOs
    (5, 3, 3, 3, 4, True),    # 455 ADOs, general diagonal couplings
    (6, 6, 0, 1, 4, False),   # 7 ADOs at d = 64
    (6, 4, 2, 2, 4, True),    # 91 ADOs
    (6, 5, 2, 2, 4, False),   # 136 ADOs
    (6, 6, 2, 2, 2, False),   # 190 ADOs: two per CTA
])
def test_packed_whole_step_runs_match_oracle(n, baths, K, depth, order, collective):
    """Whole steps in one launch on Hermitian-packed slabs (d = 32, 64): the
    trajectory against the oracle, the recorded run equal to the unrecorded
    one, and to one step at a time."""
    p = S.spin_glass(n, seed=90 + n, depth=depth, K=K, h=0.8, dt=0.005)
    p.baths = p.baths[:baths]
    if collective:
        rng = np.random.default_rng(n)
        for b in p.baths:
            b.v_diag = rng.uniform(-0.7, 0.7, p.dim)
    steps = 3
    o = O.Oracle(p)
    rho_ref, en_ref = o.run(steps, order=order, trace=True)
    want = o.state()
    o.close()
    with capi.Context(p, order=order) as a, capi.Context(p, order=order) as b:
        assert a.hermitian_packed and a.get_info().kernels_per_step == 1
        rho, en = a.step_trace(steps)
        for _ in range(steps):
            b.step(1)
        b.sync()
        assert np.array_equal(a.state(), b.state())
        assert np.max(np.abs(a.state() - want)) <= TOL
        assert abs(a.observables()[0] - en[-1]) == 0.0
    assert np.max(np.abs(rho - rho_ref)) <= TOL
    assert np.max(np.abs(en - en_ref)) <= TOL


def _run_problem(kind, n, baths, K, depth):
    p = S.spin_glass(n, seed=60 + n, depth=depth, K=K, h=0.8, dt=0.005)
    p.baths = p.baths[:baths]
    rng = np.random.default_rng(n)
    for b in p.baths:
        if kind != "spin":
            b.v_diag = rng.uniform(-0.7, 0.7, p.dim)
        if kind == "flip":
            b.v_flip = rng.uniform(0.1, 0.4, n)
    return p


@pytest.mark.parametrize("kind,n,baths,K,depth", [
    ("spin", 2, 2, 1, 2),         # 15 ADOs at d = 4: one CTA without barriers, unless a wait is to run out
    ("collective", 1, 1, 1, 3),   # 10 ADOs at d = 2, the same with a general diagonal coupling
    ("collective", 4, 2, 3, 4),   # 495 ADOs at d = 16
    ("spin", 5, 5, 2, 2),         # 136 ADOs at d = 32, one per SM
    ("spin", 5, 5, 1, 3),         # 286 ADOs at d = 32, two CTAs per SM
    ("collective", 6, 4, 2, 2),   # 91 ADOs at d = 64
    ("spin", 6, 6, 2, 2),         # 190 ADOs at d = 64, two per CTA
    ("flip", 2, 1, 2, 3),         # 20 ADOs at d = 4, couplings with flips
    ("flip", 5, 1, 2, 4),         # 35 ADOs at d = 32
])
def test_waits_of_every_run_kernel_are_reported_and_recovered_from(kind, n, baths, K, depth):
    """A wait that runs out in any kernel of whole steps, in a run of several
    steps and with more steps enqueued behind it: reported once, rho and the
    count of steps are those of before, and the context goes on as one that
    never failed."""
    p = _run_problem(kind, n, baths, K, depth)
    with capi.Context(p) as ref, capi.Context(p) as ctx:
        assert ctx.get_info().kernels_per_step == 1
        ref.step(2)
        before = ref.state()
        ctx.step(2)
        for traced in (False, True):
            assert np.array_equal(ctx.state(), before) and ctx.get_info().steps_done == 2
            ctx.inject_wait_timeout()
            with pytest.raises(capi.HxError) as e:
                if traced:
                    ctx.step_trace(3)
                else:
                    ctx.step(3)
                    if n >= 4:  # (with one CTA there is no barrier for later steps to stop at)
                        ctx.step(1)
                    ctx.sync()
            assert e.value.status == "DeviceWaitTimeout"
        assert np.array_equal(ctx.state(), before) and ctx.get_info().steps_done == 2
        rho, _ = ctx.step_trace(3)
        assert np.array_equal(rho, ref.step_trace(3)[0])
        assert np.array_equal(ctx.state(), ref.state()) and ctx.get_info().steps_done == 5


@pytest.mark.parametrize("kind,n,baths,K,depth,per_step", [
    ("spin", 4, 2, 1, 3, 4), ("spin", 5, 5, 2, 2, 8), ("flip", 2, 1, 2, 3, 8), ("flip", 5, 1, 2, 4, 8),
])
def test_small_step_variable_leaves_every_run_out(monkeypatch, kind, n, baths, K, depth, per_step):
    """HX_SMALL_STEP=0 when a context is made: a launch per pass of a stage,
    for couplings with flips too, and the same trajectory."""
    p = _run_problem(kind, n, baths, K, depth)
    with capi.Context(p) as ctx:
        assert ctx.get_info().kernels_per_step == 1
        want, _ = ctx.step_trace(4)
    monkeypatch.setenv("HX_SMALL_STEP", "0")
    with capi.Context(p) as ctx:
        assert ctx.get_info().kernels_per_step == per_step
        got, _ = ctx.step_trace(4)
        with pytest.raises(capi.HxError) as e:
            ctx.inject_wait_timeout()
        assert e.value.status == "UnsupportedExecution"
    assert np.max(np.abs(got - want)) <= TOL


# ---- rounding: against the same sums in long double


def _rhs_sums(p, rows, edges, x, real, cplx):
    """The right-hand side in the given precision: every operator's terms summed by themselves, then added."""
    d, H, M, r = p.dim, len(rows), rows.shape[1], np.arange(p.dim)
    ext = np.concatenate([x, np.zeros((1, d, d), x.dtype)])

    def apply(op, y, sign):  # [op, y] or {op, y}
        diag, flips, matrix = op
        if matrix is None:
            out = (diag[:, None] + sign * diag[None, :]).astype(real) * y
            for i, w in enumerate(flips):
                if w != 0.0:
                    out = out + real(w) * (y[:, r ^ (1 << i), :] + sign * y[:, :, r ^ (1 << i)])
            return out
        left, right = np.zeros_like(y), np.zeros_like(y)
        for i, k in zip(*np.nonzero(matrix)):
            left[:, i, :] += cplx(matrix[i, k]) * y[:, k, :]
            right[:, :, k] += y[:, :, i] * cplx(matrix[i, k])
        return left + sign * right

    def operator(diag, flips, csr):
        if csr is None:
            return np.asarray(diag, real), np.zeros(0) if flips is None else np.asarray(flips), None
        ptr, col, val = csr
        m = np.zeros((d, d), np.complex128)
        for i in range(d):
            np.add.at(m, (i, col[ptr[i]:ptr[i + 1]]), val[ptr[i]:ptr[i + 1]])
        return None, None, m

    ham = operator(p.h_diag, p.h_flip, p.h_csr_explicit)
    plain = ham[2] is None and all(b.v_csr is None and b.v_flip is None for b in p.baths)
    g = np.zeros(H, real)
    table = np.zeros((d, d), np.clongdouble)  # every term that multiplies the element itself, rounded once
    total, entries = np.zeros_like(x), np.zeros_like(x)
    o = 0
    for b in p.baths:
        c = O.bath_coefficients(b.beta, b.gamma, b.zeta, b.K)
        op = operator(b.v_diag, b.v_flip, b.v_csr)
        n = rows[:, o:o + b.K + 1]
        g += (n * c["nu"]).sum(axis=1).astype(real)
        weight = (n * c["nu"] * np.array([c["ktheta_c_im"], *c["kphi_im"]])).astype(real)
        up = [ext[np.minimum(edges[:, o + k], H)] for k in range(b.K + 1)]
        down = [ext[np.minimum(edges[:, M + o + k], H)] for k in range(b.K + 1)]
        theta = (n[:, 0] * c["nu"][0] * c["ktheta_a"]).astype(real)[:, None, None]
        if plain:
            v = np.asarray(b.v_diag, np.longdouble)
            dv, sv = v[:, None] - v[None, :], v[:, None] + v[None, :]
            table -= c["kxi"] * dv * dv + 1j * c["kxi_counter_im"] * sv * dv
            for k in range(b.K + 1):
                entries = entries - 1j * (dv.astype(real) * up[k])
                w = -1j * weight[:, k, None, None] * dv.astype(real) - (theta * sv.astype(real) if k == 0 else 0)
                entries = entries + w * down[k]
        else:
            s = np.zeros_like(x)
            for k in range(b.K + 1):
                s = s + up[k] + weight[:, k, None, None] * down[k]
            comm = apply(op, x, -1)
            t = -1j * s - real(c["kxi"]) * comm
            a = -1j * real(c["kxi_counter_im"]) * comm - theta * down[0]
            total = total + (apply(op, t, -1) + apply(op, a, 1))
        o += b.K + 1
    if plain:
        e = np.asarray(p.h_diag, np.longdouble)
        table -= 1j * (e[:, None] - e[None, :])
        flips = apply((np.zeros(d, real), p.h_flip, None), x, -1)
        return ((table.astype(cplx) - g[:, None, None]) * x - 1j * flips) + entries
    return (-1j * apply(ham, x, -1) - g[:, None, None] * x) + total


def _step_sums(rhs, x, dt, real):
    """One step, F = x + dt/1 L(x + dt/2 L(x + dt/3 L(x + dt/4 L x)))."""
    y = x
    for k in (4, 3, 2, 1):
        y = x + real(dt) / real(k) * rhs(y)
    return y


def _distance(a, b):
    return float(np.sqrt((np.abs(a - b) ** 2).sum()))


@pytest.mark.parametrize("kind,n,baths,K,depth", [
    ("flip", 2, 1, 2, 3), ("flip", 3, 2, 1, 3), ("flip", 5, 3, 1, 2),  # whole steps in one launch
    ("flip", 6, 2, 1, 3), ("flip", 7, 1, 2, 3),                        # two passes
    ("sparse", 3, 2, 1, 3), ("sparse", 5, 5, 1, 2), ("sparse", 6, 2, 2, 4),  # a slab per CTA
    ("sparse", 7, 2, 0, 2),                                                  # two passes
    ("spin", 7, 7, 0, 2), ("spin", 8, 3, 0, 2), ("collective", 7, 2, 1, 2),  # a CTA per tile
])
def test_no_more_rounding_than_term_by_term_sums(kind, n, baths, K, depth):
    """Right-hand side and one step of length 1/4 against long double, from a
    random Hermitian state.  The measure is the error of plain double-precision
    sums on the host, every operator's terms by themselves: the kernels have a
    rounding fewer per product, and half as much again is left for the order in
    which they add the parts (a quarter with diagonal couplings, which have
    three parts only)."""
    bar = 1.5 if kind in ("flip", "sparse") else 1.25
    p = _rounding_problem(kind, n, baths, K, depth)
    M = sum(b.K + 1 for b in p.baths)
    rows, edges = capi.hierarchy_tables(M, p.max_depth)
    rng = np.random.default_rng(17)
    x = rng.standard_normal((len(rows), p.dim, p.dim)) + 1j * rng.standard_normal((len(rows), p.dim, p.dim))
    x = x + x.conj().transpose(0, 2, 1)

    def exact(y):
        return _rhs_sums(p, rows, edges, y, np.longdouble, np.clongdouble)

    def plain(y):
        return _rhs_sums(p, rows, edges, y, np.float64, np.complex128)

    with capi.Context(p) as ctx:
        ctx.set_state(x)
        rhs = ctx.rhs()
        ctx.step(1)
        state = ctx.state()
    xl = x.astype(np.clongdouble)
    want = exact(xl)
    assert _distance(rhs, want) <= bar * _distance(plain(x), want)
    want = _step_sums(exact, xl, p.dt, np.longdouble)
    assert _distance(state, want) <= bar * _distance(_step_sums(plain, x, p.dt, np.float64), want)


def _rounding_problem(kind, n, baths, K, depth):
    p = S.sparse_problem(n, seed=70 + n, depth=depth, K=K, dt=0.25) if kind == "sparse" else _run_problem(kind, n, n, K, depth)
    p.baths, p.dt = p.baths[:baths], 0.25
    return p


def test_observables_of_sparse_operators_are_summed_pairwise():
    """The trace of rho_0 at d = 512, summed by 64 blocks, against the exact sum
    over 24 steps.  At 1.5 a sum by halves has roundings of 0.54 units of 2^-53
    of it in the root mean square; adding the blocks one after the other, 21 of
    them above 1 and 21 above 1/2, has 2.0.  The bar is between the two."""
    p = S.sparse_problem(9, seed=3, depth=1, K=0, dt=0.01)
    p.baths = p.baths[:2]
    rng = np.random.default_rng(5)
    with capi.Context(p) as ctx:
        assert ctx.stage_path == "csr"
        x = np.zeros((ctx.size, 512, 512), np.complex128)
        w = rng.uniform(0.5, 1.5, 512)
        x[0] = np.diag(1.5 * w / w.sum())
        ctx.set_state(x)
        err = []
        for _ in range(24):
            ctx.step(1)
            want = math.fsum(np.real(np.diagonal(ctx.rho0())))
            err.append((np.real(ctx.observables()[1]) - want) / want * 2.0 ** 53)
    assert np.sqrt(np.mean(np.square(err))) <= 1.1


@pytest.mark.parametrize("n,K,depth,size", [(1, 2, 16, 969), (1, 2, 17, 1140), (2, 2, 20, 1771), (2, 2, 21, 2024)])
def test_many_small_slabs_of_sparse_operators_match_oracle(n, K, depth, size):
    """Sparse operators at d = 2 and 4, on both sides of the number of ADOs from
    which the two passes take over from a slab per CTA."""
    p = S.sparse_problem(n, seed=20 + n, depth=depth, K=K, dt=0.002)
    p.baths = p.baths[:1]
    o = O.Oracle(p)
    rho_ref, en_ref = o.run(3, trace=True)
    o.close()
    with capi.Context(p) as ctx:
        assert ctx.stage_path == "csr" and ctx.size == size
        rho, en = ctx.step_trace(3)
    assert np.max(np.abs(rho - rho_ref)) <= TOL and np.max(np.abs(en - en_ref)) <= TOL


@pytest.mark.parametrize("kind,n,depth", [("spin", 2, 80), ("spin", 3, 37), ("spin", 4, 5), ("spin", 4, 40),
                                          ("collective", 3, 20)])
def test_one_mode_runs_whole_steps_in_one_launch(kind, n, depth):
    """A single mode gives an ADO two neighbours at most: the staging area then
    holds all of them, however few, and whole steps run in one launch."""
    p = _run_problem(kind, n, 1, 0, depth)
    o = O.Oracle(p)
    rho_ref, en_ref = o.run(5, trace=True)
    o.close()
    with capi.Context(p) as ctx:
        assert ctx.size == depth + 1 and ctx.get_info().kernels_per_step == 1
        rho, en = ctx.step_trace(5)
    assert np.max(np.abs(rho - rho_ref)) <= TOL and np.max(np.abs(en - en_ref)) <= TOL
