"""The device-resident serving loop (sp_server_*): results against the
oracle's finite-difference tangent (micro/src/homogenize.c:59-94), the same
request alone and in a mix of concurrent requests, the replay driver, and
admission by HBM budget."""
import ctypes as C
import time

import numpy as np
import pytest

import madmax_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def geoms():
    rng = np.random.default_rng(17)
    out = []
    for n in (3, 4, 5, 6, 4, 8):
        ratio = float(np.exp(rng.uniform(np.log(2), np.log(100))))
        out.append(mb.rve_desc(n, float(rng.uniform(0.1, 0.35)), (1e9, 1e9 * ratio),
                               (float(rng.uniform(0.2, 0.35)), float(rng.uniform(0.2, 0.35)))))
    return out


def oracle_fd(d, eps):
    m = O.cube_mesh(d.n[0])
    et = O.fiber_types(m, [1, 1], d.radius)
    Cm, s0 = O.fd_tangent(m, et, (d.E[0], d.E[1]), (d.nu[0], d.nu[1]), eps, rtol=1e-12,
                          lin_rtol=1e-13)
    return s0, Cm


@pytest.mark.parametrize("op", [mb.SP_OP_STENCIL, mb.SP_OP_ELL])
def test_serve_matches_oracle(op):
    G = geoms()
    s = mb.Server(G, op=op)
    s.start()
    rng = np.random.default_rng(1)
    reqs = [(int(rng.integers(0, len(G))), rng.normal(0, 1e-3, 6)) for _ in range(12)]
    tickets = [s.submit(g, e) for g, e in reqs]
    for tk, (g, e) in zip(tickets, reqs):
        st, tg, info = s.wait(tk)
        assert info.status == 0 and info.relres <= 1e-8
        s0, Cm = oracle_fd(G[g], e)
        assert np.abs(st - s0).max() <= 1e-8 * np.abs(s0).max()
        assert np.abs(tg - Cm).max() <= 1e-7 * np.abs(Cm).max()
    s.stop()
    s.close()


def test_same_result_alone_and_in_mix():
    G = geoms()
    e = np.array([1e-3, -5e-4, 2e-4, 3e-4, 0.0, -1e-4])
    a = mb.Server(G)
    a.start()
    st_alone, tg_alone, _ = a.wait(a.submit(3, e))
    a.stop()
    a.close()
    b = mb.Server(G)
    b.start()
    rng = np.random.default_rng(2)
    burst = [b.submit(int(rng.integers(0, len(G))), rng.normal(0, 1e-3, 6)) for _ in range(20)]
    mine = b.submit(3, e)
    burst += [b.submit(int(rng.integers(0, len(G))), rng.normal(0, 1e-3, 6)) for _ in range(20)]
    st_mix, tg_mix, info = b.wait(mine)
    for tk in burst:
        assert b.wait(tk)[2].status == 0
    b.stop()
    b.close()
    # warm starts differ between the two runs: equal within the solve tolerance
    assert np.abs(st_mix - st_alone).max() <= 2e-8 * np.abs(st_alone).max()
    assert np.abs(tg_mix - tg_alone).max() <= 2e-7 * np.abs(tg_alone).max()


def test_replay_poisson_latencies():
    G = geoms()
    s = mb.Server(G)
    rng = np.random.default_rng(3)
    n = 200
    t_arr = np.cumsum(rng.exponential(1.0 / 2000.0, size=n))
    geo = rng.integers(0, len(G), size=n)
    eps = rng.normal(0, 1e-3, size=(n, 6))
    td, st, tg, info = s.replay(geo, eps, t_arr, timeout=120)
    lat = td - t_arr
    assert (lat > 0).all()
    assert all(i.status == 0 for i in info)
    # spot-check a few against the oracle
    for i in (0, 57, 199):
        s0, Cm = oracle_fd(G[geo[i]], eps[i])
        assert np.abs(st[i] - s0).max() <= 1e-8 * np.abs(s0).max()
    s.stop()
    s.close()


def test_budget_refusal_and_bad_geometry():
    G = geoms()
    descs = (mb.sp_rve_desc * len(G))(*G)
    o = mb.server_opts(hbm_budget=1 << 20)
    h = mb._vp()
    assert mb.lib().sp_server_create(len(G), descs, C.byref(o), C.byref(h)) == mb.SP_ERR_BUDGET
    s = mb.Server(G)
    s.start()
    t = C.c_longlong()
    e = np.zeros(6)
    assert mb.lib().sp_server_submit(s.h, len(G), mb.ptr(e), C.byref(t)) == mb.SP_ERR_RANGE
    s.stop()
    s.close()


def test_repeated_and_zero_strain_requests_converge():
    """A warm start that already solves the request (the same strain again)
    stops at once, and a zero strain (zero right-hand side of the base load
    case) is answered with zero stress: the stopping rule is relative to the
    right-hand side, not to the warm start's residual."""
    G = geoms()
    s = mb.Server(G)
    s.start()
    e = np.array([2e-4, -1e-4, 3e-4, 0.0, 1e-4, -2e-4])
    st1, tg1, i1 = s.wait(s.submit(2, e))
    st2, tg2, i2 = s.wait(s.submit(2, e))
    z = np.zeros(6)
    st0, tg0, i0 = s.wait(s.submit(2, z))
    st0b, tg0b, i0b = s.wait(s.submit(2, z))
    s.stop()
    s.close()
    for i in (i1, i2, i0, i0b):
        assert i.status == 0 and i.relres <= 1e-8
    assert i2.inner_its < i1.inner_its
    assert np.abs(st2 - st1).max() <= 2e-8 * np.abs(st1).max()
    assert np.abs(st0).max() <= 1e-9 * np.abs(st1).max()
    assert np.abs(tg0 - tg1).max() <= 1e-7 * np.abs(tg1).max()
    assert np.abs(tg0b - tg1).max() <= 1e-7 * np.abs(tg1).max()


def test_warm_last_mode_solves_every_request():
    """SP_WARM_LAST: each request starts from the geometry's last solution
    of each load case (no prediction), runs CG to 1e-8, and keeps its
    solution as the next start; results match the oracle."""
    G = geoms()
    s = mb.Server(G, warm_start=mb.SP_WARM_LAST)
    s.start()
    rng = np.random.default_rng(8)
    reqs = [(g, rng.normal(0, 1e-3, 6)) for g in (2, 5, 2, 5, 2)]
    res = [s.wait(s.submit(g, e)) for g, e in reqs]
    s.stop()
    s.close()
    for (st, tg, info), (g, e) in zip(res, reqs):
        assert info.status == 0 and info.relres <= 1e-8 and info.outer_its > 0
        s0, Cm = oracle_fd(G[g], e)
        assert np.abs(st - s0).max() <= 1e-8 * np.abs(s0).max()
        assert np.abs(tg - Cm).max() <= 1e-7 * np.abs(Cm).max()
    bad = mb.server_opts(warm_start=7)
    descs = (mb.sp_rve_desc * len(G))(*G)
    h = mb._vp()
    assert mb.lib().sp_server_create(len(G), descs, C.byref(bad), C.byref(h)) == mb.SP_ERR_ARG


def test_idle_loop_returns_and_is_relaunched():
    """Every device wait of the serving loop is bounded: with a small
    idle_spin_limit the loop returns by itself once its queue stays empty
    (the host sees its stream idle), and the next submit relaunches it; the
    answers before and after match the oracle."""
    G = geoms()
    s = mb.Server(G, idle_spin_limit=1000)
    s.start()
    e1 = np.array([3e-4, -1e-4, 2e-4, 0.0, 1e-4, -2e-4])
    st1, tg1, i1 = s.wait(s.submit(1, e1))
    deadline = time.time() + 20.0
    on, n1, _ = s.status()
    while on and time.time() < deadline:
        time.sleep(0.01)
        on, n1, _ = s.status()
    assert not on and n1 == 1
    e2 = np.array([-2e-4, 4e-4, 1e-4, 2e-4, 0.0, 1e-4])
    st2, tg2, i2 = s.wait(s.submit(3, e2))
    _, n2, sub = s.status()
    s.stop()
    s.close()
    assert n2 == 2 and sub == 2
    for st, tg, info, g, e in ((st1, tg1, i1, 1, e1), (st2, tg2, i2, 3, e2)):
        assert info.status == 0 and info.relres <= 1e-8
        s0, Cm = oracle_fd(G[g], e)
        assert np.abs(st - s0).max() <= 1e-8 * np.abs(s0).max()
        assert np.abs(tg - Cm).max() <= 1e-7 * np.abs(Cm).max()


# --------------------------------------- message_t coupling (micro side) ---

def fake_transport(inbox):
    """In-memory stand-in for the MPI transport: recv pops the next queued
    message, send records the reply."""
    sent = []

    def recv(msg, ctx):
        if not inbox:
            return 1
        C.memmove(msg, C.byref(inbox.pop(0)), C.sizeof(mb.sp_message))
        return 0

    def send(msg, ctx):
        m = mb.sp_message()
        C.memmove(C.byref(m), msg, C.sizeof(mb.sp_message))
        sent.append(m)
        return 0

    return mb.MESSAGE_RECV(recv), mb.MESSAGE_SEND(send), sent


def message(action, strain=None):
    m = mb.sp_message()
    m.action, m.num_voigt = action, 6
    if strain is not None:
        m.strain_mac[:] = list(strain)
    return m


@pytest.mark.parametrize("mode", [mb.SP_MICRO_SOLVE, mb.SP_MICRO_LINEAR])
def test_micro_message_loop_matches_oracle(mode):
    """The request loop of micro/src/main.c:114-153 over message_t: stress,
    tangent and density requests answered from the serving loop, END ends
    the loop unanswered; results against the oracle's FD tangent."""
    G = geoms()
    s = mb.Server(G)
    s.start()
    h = mb._vp()
    mb.check(mb.lib().sp_micro_create(s.h, 4, mode, 1e7, C.byref(h)), "sp_micro_create")
    e = np.array([4e-4, -2e-4, 1e-4, 3e-4, -1e-4, 2e-4])
    inbox = [message(mb.SP_ACTION_MICRO_CALC_STRESS, e), message(mb.SP_ACTION_MICRO_CALC_C_TANGENT, e),
             message(mb.SP_ACTION_MICRO_CALC_RHO), message(mb.SP_ACTION_MICRO_END)]
    recv, send, sent = fake_transport(inbox)
    n = C.c_longlong()
    mb.check(mb.lib().sp_micro_serve(h, recv, send, None, C.byref(n)), "sp_micro_serve")
    assert n.value == 4 and len(sent) == 3 and not inbox
    assert [m.action for m in sent] == [1, 2, 3]
    stress = np.array(sent[0].stress_ave[:])
    tangent = np.array(sent[1].c_tangent_ave[:]).reshape(6, 6)
    assert sent[2].rho == 1e7
    s0, Cm = oracle_fd(G[4], e)
    _, C0 = oracle_fd(G[4], np.zeros(6))
    if mode == mb.SP_MICRO_SOLVE:
        assert np.abs(stress - s0).max() <= 1e-8 * np.abs(s0).max()
        assert np.abs(tangent - Cm).max() <= 1e-7 * np.abs(Cm).max()
    else:
        # the reference's linear path: C from the FD tangent around zero, sigma = C eps
        assert np.abs(tangent - C0).max() <= 1e-7 * np.abs(C0).max()
        assert np.abs(stress - C0 @ e).max() <= 1e-7 * np.abs(C0 @ e).max()
    req = C.c_longlong()
    mb.lib().sp_micro_requests(h, C.byref(req))
    assert req.value == (2 if mode == mb.SP_MICRO_SOLVE else 1)
    bad = message(9)
    assert mb.lib().sp_micro_handle(h, C.byref(bad)) == mb.SP_ERR_ARG
    bad = message(mb.SP_ACTION_MICRO_CALC_STRESS, e)
    bad.num_voigt = 3
    assert mb.lib().sp_micro_handle(h, C.byref(bad)) == mb.SP_ERR_ARG
    mb.lib().sp_micro_destroy(h)
    s.stop()
    s.close()


# ---------------------------------------------- element-mode request loop ---

MODE_GEOMS = [
    ((5, 7, 3), (6, 6, 6)),        # 64 threads, eight tasks to an SM
    ((12, 12, 12), (9, 10, 11)),   # 160 threads, three to an SM
    ((16, 16, 15),),               # 256 threads, two to an SM
    ((17, 12, 20), (8, 8, 8)),     # 512 threads, p and q on chip
    ((24, 20, 20), (32, 10, 31)),  # p on chip; a layer of one strip
    ((31, 32, 9), (32, 32, 32)),   # strips of rows, no vector on chip
    ((4, 4, 4), (5, 5, 33)),       # beyond the range: the block-stencil loop
    ((6, 6, 6), (3, 3, 1)),        # no interior node: the block-stencil loop
]


def mode_desc(n, k):
    edge = 1.0 / 8 if k % 2 else np.array([0.125, 0.12, 0.13])
    return mb.rve_desc(n, 0.2, (1e9, 1e9 * (5 + 9 * k)), (0.3, 0.2), list(np.array(n) * edge))


def exact_tangents(D):
    """Effective tangents by the FP64 batch of assembled operators (linear materials:
    the stress of strain e is C e, and the finite-difference tangent is C)."""
    b = mb.Batch(D, nrhs=6, precision=mb.SP_PREC_FP64, op=mb.SP_OP_ELL, rtol=1e-11)
    eye = np.ascontiguousarray(np.broadcast_to(np.eye(6), (len(D), 6, 6)))
    Cs = np.swapaxes(b.homogenize(eye)[0], 1, 2).copy()
    b.close()
    return Cs


@pytest.mark.parametrize("k", range(len(MODE_GEOMS)))
def test_serve_classes_match_batch(k):
    """Requests one after the other on every class of the loop, against the
    effective tangent.  Solves to 1e-8 of the right-hand side's norm; the
    tangent divides a difference of stresses by 0.005, about 2 |eps|."""
    D = [mode_desc(n, i + k) for i, n in enumerate(MODE_GEOMS[k])]
    Cs = exact_tangents(D)
    rng = np.random.default_rng(k)
    s = mb.Server(D)
    s.start()
    for g in [i % len(D) for i in range(4)]:
        e = rng.normal(0, 1e-3, 6)
        st, tg, info = s.wait(s.submit(g, e))
        assert info.status == 0 and info.relres <= 1e-8
        ref = Cs[g] @ e
        assert np.abs(st - ref).max() <= 2e-8 * np.abs(ref).max()
        assert np.abs(np.array(tg).reshape(6, 6) - Cs[g]).max() <= 2e-7 * np.abs(Cs[g]).max()
    s.stop()
    s.close()


@pytest.mark.parametrize("n,warm,opts", [
    ((6, 6, 6), 0, {}), ((12, 12, 12), 0, {}), ((24, 24, 24), 0, {}), ((6, 6, 6), 1, {}),
    ((6, 6, 6), 0, {"ctas_per_sm": 2}), ((6, 6, 6), 1, {"op": mb.SP_OP_ELL}),
    ((5, 5, 33), 0, {})])
def test_concurrent_cold_requests_on_one_geometry(n, warm, opts):
    """Requests that arrive together on a geometry without a stored solution,
    then again: while one stores its solutions the others start from none or
    from whole ones, never from a mixture."""
    d = mode_desc(n, 1)
    Cm = exact_tangents([d])[0]
    rng = np.random.default_rng(3)
    nreq = 12 if n[0] > 12 else 40
    for fresh in range(3):
        s = mb.Server([d], warm_start=mb.SP_WARM_LAST if warm else mb.SP_WARM_PREDICT, **opts)
        s.start()
        for again in range(3):
            E = rng.normal(0, 1e-3, (nreq, 6))
            tk = [s.submit(0, e) for e in E]
            for t, e in zip(tk, E):
                st, tg, info = s.wait(t)
                assert info.status == 0 and info.relres <= 1e-8
                ref = Cm @ e
                assert np.abs(st - ref).max() <= 2e-8 * np.abs(ref).max()
                assert np.abs(np.array(tg).reshape(6, 6) - Cm).max() <= 2e-7 * np.abs(Cm).max()
        s.stop()
        s.close()


def test_slow_requests_after_a_burst():
    """CTAs that took tickets past the end of a burst keep them while requests
    come one by one, for many times the idle limit in all, and across a loop
    that left and was relaunched: every request is answered."""
    d = mode_desc((6, 6, 6), 1)
    Cm = exact_tangents([d])[0]
    rng = np.random.default_rng(9)
    s = mb.Server([d], idle_spin_limit=2000)
    s.start()

    def ask(n):
        E = rng.normal(0, 1e-3, (n, 6))
        for t, e in [(s.submit(0, e), e) for e in E]:
            st, _, info = s.wait(t)
            ref = Cm @ e
            assert info.status == 0 and np.abs(st - ref).max() <= 2e-8 * np.abs(ref).max()

    for gap in (0.0, 5e-4, 2e-3, 3e-2):
        ask(300)
        for _ in range(60 if gap < 1e-2 else 5):
            time.sleep(gap)
            ask(1)
    s.stop()
    s.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("warm", [mb.SP_WARM_PREDICT, mb.SP_WARM_LAST])
@pytest.mark.parametrize("opts", [{}, {"ctas_per_sm": 2}, {"op": mb.SP_OP_ELL}])
def test_non_finite_request_does_not_outlast_its_answer(opts, warm, bad):
    """A request with a non-finite strain, on a geometry without and with a
    stored solution, is answered as not converged; the requests after it on the
    same geometry are solved as if it had not been there."""
    d = mode_desc((6, 6, 6), 1)
    Cm = exact_tangents([d])[0]
    rng = np.random.default_rng(4)
    s = mb.Server([d], warm_start=warm, **opts)
    s.start()
    for k in range(3):
        e = rng.normal(0, 1e-3, 6)
        e[(1, 3, 0)[k]] = bad
        info = s.wait(s.submit(0, e))[2]
        assert info.status == mb.SP_ERR_NOCONV and np.isnan(info.relres)
        for _ in range(2):
            e = rng.normal(0, 1e-3, 6)
            st, tg, info = s.wait(s.submit(0, e))
            assert info.status == 0 and info.relres <= 1e-8
            ref = Cm @ e
            assert np.abs(st - ref).max() <= 2e-8 * np.abs(ref).max()
            assert np.abs(np.array(tg).reshape(6, 6) - Cm).max() <= 2e-7 * np.abs(Cm).max()
    s.stop()
    s.close()


@pytest.mark.parametrize("n", [(6, 6, 6), (12, 12, 12), (24, 24, 24)])
def test_request_that_misses_in_some_load_cases_is_kept(n):
    """A base strain far below the stored one: its load case misses the
    prediction, the six of eps + 0.005 e_i meet it.  The request's solutions
    become the geometry's store all the same, so that later requests of that
    size are predicted."""
    d = mode_desc(n, 1)
    Cm = exact_tangents([d])[0]
    rng = np.random.default_rng(6)
    s = mb.Server([d])
    s.start()
    big, small = rng.normal(0, 1e-3, 6), rng.normal(0, 1e-9, 6)
    first = s.wait(s.submit(0, big))[2]
    second = s.wait(s.submit(0, small))[2]
    assert first.inner_its > second.inner_its > 0
    for _ in range(3):
        e = small * rng.uniform(0.9, 1.1)
        st, tg, info = s.wait(s.submit(0, e))
        assert info.status == 0 and info.inner_its == 0
        ref = Cm @ e
        assert np.abs(st - ref).max() <= 2e-8 * np.abs(ref).max()
        assert np.abs(np.array(tg).reshape(6, 6) - Cm).max() <= 2e-7 * np.abs(Cm).max()
    s.stop()
    s.close()


@pytest.mark.parametrize("scale,strain", [(1.0, 1e-14), (1.0, 1e-18), (1e-6, 1e-10)])
@pytest.mark.parametrize("warm", [mb.SP_WARM_PREDICT, mb.SP_WARM_LAST])
def test_small_strains_and_lengths(warm, scale, strain):
    """Strains at the round-off level of an unloaded point, and edges of
    micrometres in SI units: the residual norms that steer CG are squares far
    below the smallest FP32 number.  One geometry of each place the vectors
    may lie in."""
    D = []
    for n in ((6, 6, 6), (24, 20, 20), (31, 32, 9)):
        D.append(mb.rve_desc(n, 0.2, (1e9, 2e10), (0.3, 0.2), list(np.array(n) / 8.0)))
    Cs = exact_tangents(D)
    for d in D:
        for k in range(3):
            d.len[k] *= scale
        d.radius *= scale
    rng = np.random.default_rng(12)
    s = mb.Server(D, warm_start=warm)
    s.start()
    for g in (0, 1, 2, 0, 1, 2):
        e = rng.normal(0, strain, 6)
        st, tg, info = s.wait(s.submit(g, e))
        assert info.status == 0 and info.relres <= 1e-8
        ref = Cs[g] @ e
        assert np.abs(st - ref).max() <= 2e-8 * np.abs(ref).max()
        assert np.abs(np.array(tg).reshape(6, 6) - Cs[g]).max() <= 2e-7 * np.abs(Cs[g]).max()
    s.stop()
    s.close()
