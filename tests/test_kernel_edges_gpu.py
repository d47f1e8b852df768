"""The force kernels at the sizes where their tiles, ranges and queues can go
wrong, against the FP64 oracle.  Tolerances: the per-particle bounds of the
other parity tests (acceleration and potential 1e-6, jerk 1e-5), which the FP32
pair math on hi/lo differences with double-single or FP64 sums meets at any size:
relative to the value where its terms mostly add up, to the sum of the terms'
sizes (_sizes) where they may cancel; neighbour lists identical."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from parity import rel_err_vec

pytestmark = pytest.mark.gpu


# tile of 128 bodies, i-tile of 128 (256 once ni >= 4736), order from 1e9 pairs
@pytest.mark.parametrize("n,i0,ni", [(127, 0, 127), (257, 129, 128), (4736, 0, 4736), (5001, 265, 4735),
                                     (33000, 0, 30304), (33000, 2696, 30304), (40007, 14997, 25010),
                                     (65537, 65537 - 15361, 15361), (40960, 0, 40960)])
def test_potential_ranges(nb6, orc, n, i0, ni):
    """Ranges of the set on both sides of the rule that orders it, at its
    start, inside and at its end, whole and ragged tiles."""
    from nb6b200 import ics
    cl = ics.plummer(n, seed=n + i0, imf=True)
    x = cl.pos.copy()
    x[i0] = x[(i0 + 1) % n]                       # a coincident pair
    p = nb6.gpupot(cl.mass, x, istart=i0 + 1, ni=ni)
    sel = np.unique(np.concatenate([[0, ni - 1], np.random.default_rng(n).integers(0, ni, 300)]))
    po = np.array([orc.pot(cl.mass, x, i0 + 1 + int(k), 1)[0] for k in sel])
    assert np.all(p > 0)
    assert rel_err_vec(p[sel], po).max() <= 1e-6


# 32 samples per CTA and round; 296 CTAs, so a second round from 9,473 samples
@pytest.mark.parametrize("n", [31, 32, 33, 1000, 9472, 9473, 20011])
def test_mlp_gradient_sample_counts(n):
    """The gradient's sample streams at full and ragged rounds against the
    FP64 oracle: within 2e-5 of its norm (FP32 sums over the batch)."""
    import mlp_oracle as M
    from nb6b200 import mlp
    rng = np.random.default_rng(n)
    model = np.zeros(M.NPARAM + M.NNORM, dtype=np.float32)
    model[:M.NPARAM] = rng.normal(size=M.NPARAM) * 0.15
    model[M.NPARAM + M.IN:M.NPARAM + 2 * M.IN] = 1.0
    model[-1] = 0.5
    mlp.set_model(model)
    x = rng.normal(size=(n, 5)).astype(np.float32)
    y = rng.normal(size=n).astype(np.float32)
    g, loss = mlp.grad(x, y)
    gr, lr = M.grad(model, x, y)
    assert abs(loss - lr) <= 1e-5 * lr
    assert np.linalg.norm(g - gr) <= 2e-5 * np.linalg.norm(gr)


@pytest.fixture(scope="module")
def shuffled(tmp_path_factory):
    """The order std::shuffle gives 0..n-1 with a std::mt19937 of `seed`."""
    d = tmp_path_factory.mktemp("shuffle")
    (d / "s.cpp").write_text("""#include <algorithm>
#include <numeric>
#include <random>
extern "C" void order(int n, unsigned seed, int *p) {
    std::iota(p, p + n, 0);
    std::mt19937 gen(seed);
    std::shuffle(p, p + n, gen);
}""")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", str(d / "s.so"), str(d / "s.cpp")], check=True)
    lib = C.CDLL(str(d / "s.so"))

    def order(n, seed):
        p = np.empty(n, dtype=np.int32)
        lib.order(n, seed, p.ctypes.data_as(C.c_void_p))
        return p
    return order


# 32 samples per four CTAs, one round; 145 CTAs sum the parameters, more CTAs
# hold the samples from a batch of 1,153; 1,024 steps per launch; two launches
# a step once the CTAs no longer fit (4,736 here at the latest: 4 per SM)
@pytest.mark.parametrize("n,batch", [(1, 1), (1030, 1), (700, 33), (3000, 256), (4100, 1000), (4000, 1152),
                                     (4000, 1184), (20011, 2500), (11000, 3552), (15000, 4737)])
def test_mlp_training_steps(shuffled, n, batch):
    """One epoch against Adam on the FP64 oracle's gradients.  A gradient
    within 2e-5 of its norm turns the sign of about that share of its elements,
    which moves a parameter by two learning rates: 1% of the parameters' change
    (bound 2%).  The mean loss follows to 1e-3; a second run gives the same
    bits."""
    import mlp_oracle as M
    from nb6b200 import mlp
    rng = np.random.default_rng(n + batch)
    model = np.zeros(M.NPARAM + M.NNORM, dtype=np.float32)
    model[:M.NPARAM] = rng.normal(size=M.NPARAM) * 0.15
    model[M.NPARAM + M.IN:M.NPARAM + 2 * M.IN] = 1.0
    model[-1] = 1.0
    x = rng.normal(size=(n, 5)).astype(np.float32)
    y = (x[:, 0] - 0.3 * x[:, 1] * x[:, 2] + 0.1 * rng.normal(size=n)).astype(np.float32)
    lr = 1e-5 if n // batch > 100 else 1e-4
    runs = []
    for _ in range(2):
        mlp.set_model(model)
        hist = mlp.train(x, y, epochs=1, batch=batch, lr=lr, seed=5)
        runs.append((mlp.get_model(), hist))
    np.testing.assert_array_equal(runs[0][0], runs[1][0])
    np.testing.assert_array_equal(runs[0][1], runs[1][1])
    got, hist = runs[0]
    nm = got[M.NPARAM:].astype(np.float64)
    xs = x.astype(np.float64)
    std = np.sqrt(np.maximum(xs.var(0), 1e-12))
    np.testing.assert_allclose(nm[:5], xs.mean(0), atol=1e-6)
    np.testing.assert_allclose(nm[5:10], 1 / std, rtol=1e-6)
    order = shuffled(n, 5)
    w = model[:M.NPARAM].astype(np.float64)
    b1, b2, one = np.float32(0.9), np.float32(0.999), np.float32(1)
    m1, m2, losses = np.zeros(M.NPARAM), np.zeros(M.NPARAM), []
    for t in range(1, n // batch + 1):
        s = order[(t - 1) * batch:t * batch]
        g, loss = M.grad64(M.bf16_round(w).astype(np.float64), nm, x[s], y[s])
        losses.append(loss)
        m1 = b1 * m1 + (one - b1) * g
        m2 = b2 * m2 + (one - b2) * g * g
        w = w - lr * (m1 / (1 - float(b1) ** t)) / (np.sqrt(m2 / (1 - float(b2) ** t)) + 1e-8)
    assert abs(hist[0] - np.mean(losses)) <= 1e-3 * np.mean(losses) + 1e-12
    assert np.linalg.norm(got[:M.NPARAM] - w) <= 0.02 * np.linalg.norm(w - model[:M.NPARAM])


def test_mlp_moments_of_unusable_columns():
    """A NaN or an infinity among the samples shows in the stored moments of its
    column, mean and scale (the variance is a NaN), and in no other; a constant
    column has the least variance, 1e-12."""
    import mlp_oracle as M
    from nb6b200 import mlp
    rng = np.random.default_rng(4)
    n = 2500
    x, y = rng.normal(size=(n, 5)).astype(np.float32), rng.normal(size=n).astype(np.float32)
    x[1700, 1], x[3, 2], x[:, 3] = np.nan, np.inf, 2.0
    model = np.zeros(M.NPARAM + M.NNORM, dtype=np.float32)
    model[M.NPARAM + M.IN:M.NPARAM + 2 * M.IN] = 1.0
    model[-1] = 1.0
    mlp.set_model(model)
    mlp.train(x, y, epochs=0, batch=100, lr=1e-3, seed=1)
    mean, scale = np.split(mlp.get_model()[M.NPARAM:M.NPARAM + 10], 2)
    assert np.isnan(mean[1]) and np.isnan(scale[1])
    assert np.isposinf(mean[2]) and np.isnan(scale[2])
    assert mean[3] == 2.0 and scale[3] == np.float32(1e6)
    ok = x[:, [0, 4]].astype(np.float64)
    np.testing.assert_allclose(mean[[0, 4]], ok.mean(0), atol=1e-6)
    np.testing.assert_allclose(scale[[0, 4]], 1 / ok.std(0), rtol=1e-6)


def _sizes(m, x, v, xi, vi, near):
    """Sums of the sizes of one body's acceleration and jerk terms over the
    bodies that are not its neighbours."""
    d, w = x - xi, v - vi
    r2 = (d * d).sum(1)
    use = (r2 > 0) & ~np.isin(np.arange(len(m)), near)
    d, w, r2, m = d[use], w[use], r2[use], m[use]
    r = np.sqrt(r2)
    return (m / r2).sum(), (m / (r * r2) * (np.sqrt((w * w).sum(1)) + 3 * np.abs((d * w).sum(1)) / r)).sum()


def _shells(n, seed):
    """n bodies, of which the first 40 sit at the centre of dense shells: most
    pairs of theirs lie within 1% of their radius, inside and outside."""
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    v = 0.3 * rng.normal(size=(n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    x[:40] *= 0.02
    u = rng.normal(size=(n - 40, 3))
    u /= np.sqrt((u * u).sum(1))[:, None]
    x[40:] = u * (0.5 * (1.0 + 0.02 * rng.uniform(-1, 1, n - 40)))[:, None]
    return m, x, v


@pytest.mark.parametrize("variant", [11, 12, 13, -1, -2, -4, -8])
@pytest.mark.parametrize("n", [200, 257, 1291])
def test_candidate_queue_band_and_overflow(nb6, orc, variant, n):
    """Candidate queues that fill on nearly every pair: bodies whose pairs
    crowd the slack band about the radius (candidates that are no neighbours
    give their force back), rows that list every body, rows that overflow,
    and a ragged last tile whose padding is within reach."""
    m, x, v = _shells(n, n)
    ni = 67
    h2 = np.full(ni, 0.25)
    h2[41:45] = 100.0              # every body a neighbour
    h2[45:47] = 1.0e31             # and the padding slots within reach
    h2[47:50] = 0.0                # no neighbour at all
    dtr = np.zeros(ni)
    dtr[50:] = 2.0 ** -6
    cap = 1300 if n < 1000 else 400
    raw = nb6.lib
    raw.nb6_regf_tune_(C.byref(C.c_int(variant)), C.byref(C.c_int(0)))
    try:
        nb6.gpunb_open(n, 0)
        nb6.gpunb_send(m, x, v)
        for mf in (0, 1):
            hh = h2 * n if mf else h2
            acc, jrk, pot, lst = nb6.gpunb_regf(hh, dtr, x[:ni], v[:ni], cap + 1, cap, mf)
            oa, oj, op, ol = orc.regf(m, x, v, hh, dtr, x[:ni], v[:ni], cap + 1, cap, mf)
            np.testing.assert_array_equal(lst[:, 0], ol[:, 0])
            for r in range(ni):
                k = max(int(ol[r, 0]), 0)
                np.testing.assert_array_equal(lst[r, 1:1 + k], ol[r, 1:1 + k])
            # FP32 sums of n terms against the sum of their sizes
            for r in range(ni):
                if ol[r, 0] < 0:
                    continue
                if np.isnan(oa[r]).any():   # radius zero: the body acts on itself
                    assert h2[r] == 0.0 and np.isnan(acc[r]).any()
                    continue
                sa, sj = _sizes(m, x, v, x[r], v[r], ol[r, 1:1 + max(int(ol[r, 0]), 0)])
                assert np.abs(acc[r] - oa[r]).max() <= 1e-6 * sa
                assert np.abs(jrk[r] - oj[r]).max() <= 1e-5 * sj
                assert abs(pot[r] - op[r]) <= 1e-6 * abs(op[r]) + 1e-300
    finally:
        raw.nb6_regf_tune_(C.byref(C.c_int(0)), C.byref(C.c_int(0)))
        nb6.gpunb_close()


@pytest.mark.parametrize("ni,nj,slices", [(200, 1024, 500), (5, 1024, 500), (1500, 2050, 77), (9000, 9000, 3),
                                          (3, 1025, 70000)])
def test_forced_slices_on_the_tuning_call(nb6, orc, ni, nj, slices):
    """A forced slice count with the variant left to the tuner, on the first
    call of its bucket: the partials have room for the variant that wins, more
    slices than bodies (or than a grid holds) are accepted, and a second call,
    which no longer tunes, gives the same bits."""
    from nb6b200 import ics
    cl = ics.plummer(nj, seed=nj, imf=True)
    h2 = cl.h2(0)[:ni]
    raw, geom = nb6.lib, (C.c_int * 3)()
    raw.nb6_regf_tune_(C.byref(C.c_int(0)), C.byref(C.c_int(slices)))
    raw.nb6_regf_autotune_(C.byref(C.c_int(-1)))
    try:
        nb6.gpunb_open(nj, 0)
        nb6.gpunb_send(cl.mass, cl.pos, cl.vel)
        runs = []
        for _ in range(2):
            runs.append(nb6.gpunb_regf(h2, cl.dtr[:ni], cl.pos[:ni], cl.vel[:ni], 512, 400, 0))
            raw.nb6_regf_last_geometry_(geom)
            most = -(-nj // 128) if geom[0] > 0 else nj
            assert geom[2] == min(slices, most, 65535)
    finally:
        raw.nb6_regf_tune_(C.byref(C.c_int(0)), C.byref(C.c_int(0)))
        raw.nb6_regf_autotune_(C.byref(C.c_int(-1)))
        nb6.gpunb_close()
    for a, b in zip(*runs):
        np.testing.assert_array_equal(a, b)
    acc, jrk, pot, lst = runs[0]
    oa, oj, op, ol = orc.regf(cl.mass, cl.pos, cl.vel, h2, cl.dtr[:ni], cl.pos[:ni], cl.vel[:ni], 512, 400, 0)
    np.testing.assert_array_equal(lst, ol)
    assert rel_err_vec(acc, oa).max() <= 1e-6
    assert rel_err_vec(jrk, oj).max() <= 1e-5
    assert rel_err_vec(pot, op).max() <= 1e-6


@pytest.mark.parametrize("cap", [31, 400, 512, 700])
def test_list_rows_at_register_widths(nb6, orc, cap):
    """List rows whose count falls on either side of the widths the sort
    takes in registers (32 .. 512 ids) and in shared memory, with and without
    room in the row; the caller's row past the count is left alone."""
    n = 1100
    rng = np.random.default_rng(cap)
    m = np.full(n, 1.0 / n)
    x = np.zeros((n, 3))
    x[:, 0] = rng.permutation(n)          # body at rank k: k neighbours within k + 1/2 of the first
    v = np.zeros((n, 3))
    at0 = int(np.argmin(x[:, 0]))
    counts = np.array([1, 2, 30, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 399, 400, 401, 511, 512,
                       513, 699, 700, 701, 1100])
    h2 = (counts - 0.5) ** 2
    ni = len(counts)
    xi, vi, dtr = np.repeat(x[at0:at0 + 1], ni, 0), np.zeros((ni, 3)), np.zeros(ni)
    nb6.gpunb_open(n, 0)
    try:
        nb6.gpunb_send(m, x, v)
        acc, jrk, pot, lst = nb6.gpunb_regf(h2, dtr, xi, vi, cap + 1, cap, 0)
    finally:
        nb6.gpunb_close()
    order = np.argsort(x[:, 0])
    for r, c in enumerate(counts):
        if c > cap:
            assert lst[r, 0] == -c
            assert np.all(lst[r, 1:] == 0)
        else:
            assert lst[r, 0] == c
            np.testing.assert_array_equal(lst[r, 1:1 + c], np.sort(order[:c]))
            assert np.all(lst[r, 1 + c:] == 0)


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("ni", [1, 3, 255, 256, 257, 292, 293, 8193])
def test_irregular_rounds_and_call_sizes(nb6, orc, mode, ni):
    """Lists on either side of the walk's rounds of 32 and of the row's end,
    and calls on either side of the sizes that pass their addresses with the
    launch and write their results in place.  FP64 sums of at most 199 terms:
    1e-10 relative leaves four digits for cancellation."""
    n, lmax = 600, 200
    rng = np.random.default_rng(ni)
    lens = np.array([0, 1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 191, 192, 193, 199])
    lists = np.zeros((n, lmax), dtype=np.int32)
    for i in range(n):
        k = int(lens[i % len(lens)])
        lists[i, 0] = k
        lists[i, 1:1 + k] = np.sort(rng.choice(np.delete(np.arange(1, n + 1), i), k, replace=False))
    x0, v0, f2, fd6 = (rng.normal(size=(n, 3)) for _ in range(4))
    m, t0 = rng.uniform(0.5, 1.5, n) / n, -rng.integers(0, 16, n) / 2048.0
    addr = (rng.permutation(max(n, ni))[:ni] % n + 1).astype(np.int32)
    nb6.irr_open(n, lmax, 0)
    try:
        nb6.lib.nb6_irr_pv_(C.byref(C.c_int(mode)))
        nb6.irr_set_jp_all(x0, v0, f2, fd6, m, t0)
        for i in range(n):
            nb6.irr_set_list(i + 1, lists[i])
        for _ in range(2):       # the second call has nothing staged before it
            acc, jrk, nnbid = nb6.irr_firr_vec(1.0 / 2048, addr)
            oa, oj, oid = orc.firr(1.0 / 2048, addr, x0, v0, f2, fd6, m, t0, lists)
            ok = lists[addr - 1, 0] > 0
            np.testing.assert_array_equal(nnbid, oid)
            assert np.all(acc[~ok] == 0) and np.all(jrk[~ok] == 0)
            if ok.any():
                assert rel_err_vec(acc[ok], oa[ok]).max() <= 1e-10
                assert rel_err_vec(jrk[ok], oj[ok]).max() <= 1e-10
    finally:
        nb6.lib.nb6_irr_pv_(C.byref(C.c_int(1)))
        nb6.irr_close(0)


def test_failed_segmented_call_leaves_the_callers_arrays(nb6, orc):
    """A segmented call in stages against a j set with a NaN in its last
    segment: the status is reported and no row of the caller's arrays is
    touched; a good set sent afterwards gives the oracle's rows."""
    import nb6b200
    rng = np.random.default_rng(8)
    nc, nseg = 300, 70
    n, cap = nc * nseg, 60
    x, v = rng.normal(size=(n, 3)), 0.3 * rng.normal(size=(n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    j0 = (nc * np.arange(nseg + 1)).astype(np.int32)
    iseg = np.repeat(np.arange(nseg), nc).astype(np.int32)
    h2, dtr = np.full(n, 0.2), np.full(n, 2.0 ** -6)
    bad = x.copy()
    bad[n - 1, 1] = np.nan
    nb6b200.set_abort_on_error(False)
    nb6.gpunb_open(n, 0)
    try:
        nb6b200.last_status()
        nb6.gpunb_send(m, bad, v)
        for o in nb6.regf_seg(h2, dtr, x, v, iseg, j0, cap + 1, cap, 0):
            assert not o.any()
        assert nb6b200.last_status() == 3
        geom = (C.c_int * 3)()
        nb6.lib.nb6_regf_last_geometry_(geom)
        assert geom[2] >= 8 * geom[1]      # rounds enough for stages
        nb6.gpunb_send(m, x, v)
        out = nb6.regf_seg(h2, dtr, x, v, iseg, j0, cap + 1, cap, 0)
        assert nb6b200.last_status() == 0
    finally:
        nb6b200.set_abort_on_error(True)
        nb6.gpunb_close()
    for c in (0, 34, nseg - 1):
        s = slice(j0[c], j0[c + 1])
        ol = orc.regf(m[s], x[s], v[s], h2[s], dtr[s], x[s], v[s], cap + 1, cap, 0)[3]
        np.testing.assert_array_equal(out[3][s], ol)


@pytest.mark.parametrize("cap,mf", [(20, 0), (60, 0), (60, 1), (600, 0)])
def test_segmented_many_items(nb6, orc, cap, mf):
    """A segmented call of many work items per CTA, whose rows reach the
    caller in stages while later ones compute (cap 20 and 60): ragged segments,
    groups of one to four, a lone body, an empty segment in between, rows that
    overflow (cap 20), rows longer than the kernel sorts itself (cap 600),
    radii that scale with the bodies' masses (mf 1); every row against the
    oracle of its segment."""
    rng = np.random.default_rng(cap)
    ns = np.concatenate([rng.integers(250, 420, 66), [0, 1, 2, 3]])
    rng.shuffle(ns)
    j0 = np.concatenate([[0], np.cumsum(ns)]).astype(np.int32)
    n = int(j0[-1])
    x, v = rng.normal(size=(n, 3)), 0.3 * rng.normal(size=(n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    iseg = np.repeat(np.arange(len(ns)), ns).astype(np.int32)
    h2 = rng.uniform(0.2, 0.8, n) ** 2 * (n if mf else 1)
    dtr = np.full(n, 2.0 ** -6)
    nb6.gpunb_open(n, 0)
    try:
        nb6.gpunb_send(m, x, v)
        for _ in range(2):
            acc, jrk, pot, lst = nb6.regf_seg(h2, dtr, x, v, iseg, j0, cap + 1, cap, mf)
            geom = (C.c_int * 3)()
            nb6.lib.nb6_regf_last_geometry_(geom)
            if cap <= 512:                # eight rounds of items: in stages
                assert geom[2] > 7 * geom[1]
            for c in range(len(ns)):
                s = slice(j0[c], j0[c + 1])
                if ns[c] == 0:
                    continue
                oa, oj, op, ol = orc.regf(m[s], x[s], v[s], h2[s], dtr[s], x[s], v[s], cap + 1, cap, mf)
                np.testing.assert_array_equal(lst[s], ol)
                ok = (np.abs(oa).sum(1) > 0) & (ol[:, 0] >= 0)
                if ok.any():
                    assert rel_err_vec(acc[s][ok], oa[ok]).max() <= 1e-5
                    assert rel_err_vec(pot[s][ok], op[ok]).max() <= 1e-6
                for r in np.flatnonzero(ok)[::5]:
                    sa, sj = _sizes(m[s], x[s], v[s], x[s][r], v[s][r], ol[r, 1:1 + ol[r, 0]])
                    assert np.abs(acc[s][r] - oa[r]).max() <= 1e-6 * sa
                    assert np.abs(jrk[s][r] - oj[r]).max() <= 1e-5 * sj
    finally:
        nb6.gpunb_close()


def test_kernel_times_of_small_and_large_calls(nb6):
    """The kernel time of a call that stamps its own (small) and of one timed
    by events (large), alternating: more than zero, within the call's wall
    time, and the large one's not left over from the small one."""
    import time

    from nb6b200 import ics
    lib = nb6.lib

    def timed(call, ms):
        t = time.perf_counter()
        call()
        wall = 1e3 * (time.perf_counter() - t)
        got = float(ms())
        assert 0.0 < got <= wall
        return got

    big, small = ics.plummer(40960, seed=3), ics.plummer(300, seed=4)
    nb6.gpupot(big.mass, big.pos)
    for _ in range(2):
        a = timed(lambda: nb6.gpupot(small.mass, small.pos), lib.nb6_pot_last_kernel_ms_)
        b = timed(lambda: nb6.gpupot(big.mass, big.pos), lib.nb6_pot_last_kernel_ms_)
        assert b > a
    n, zero = 20000, np.zeros((20000, 3))
    cl = ics.plummer(n, seed=5)
    rng = np.random.default_rng(6)
    nb6.irr_open(n, 64, 0)
    try:
        nb6.irr_set_jp_all(cl.pos, cl.vel, zero, zero, cl.mass, np.zeros(n))
        for i in range(n):
            nb6.irr_set_list(i + 1, np.concatenate([[40], rng.integers(1, n + 1, 40)]).astype(np.int32))
        few, many = np.arange(1, 101, dtype=np.int32), np.arange(1, n + 1, dtype=np.int32)
        nb6.irr_firr_vec(0.0, many)
        for _ in range(2):
            a = timed(lambda: nb6.irr_firr_vec(0.0, few), lib.nb6_irr_last_kernel_ms_)
            b = timed(lambda: nb6.irr_firr_vec(0.0, many), lib.nb6_irr_last_kernel_ms_)
            assert b > a
    finally:
        nb6.irr_close(0)


@pytest.mark.parametrize("kind", ["segments", "j-parallel"])
def test_long_sums(nb6, kind):
    """Active bodies far outside a compact clump of bodies of one mass: every
    thread adds nearly the same term again and again, and its FP32 sum drifts
    the same way in all of them.  A sum of N equal terms is off by at most N / 2
    half-ulps of its value: 32 terms in a segmented call, 128 in a j-parallel
    one, and six more half-ulps for the terms."""
    seg = kind == "segments"
    nseg, nc, na = (2, 65536, 6000) if seg else (1, 262144, 6000)
    rng = np.random.default_rng(7)
    n, ni = nseg * nc, nseg * na
    x, v, m = 1e-6 * rng.normal(size=(n, 3)), 1e-6 * rng.normal(size=(n, 3)), np.full(n, 1.0 / nc)
    xi = np.zeros((ni, 3))
    xi[:, 0] = np.tile(1.0 + np.arange(na) / na, nseg)
    xi[:, 1] = 0.3 * xi[:, 0]
    vi = np.tile([0.0, 0.7, 0.0], (ni, 1))
    h2, dtr = np.full(ni, 1e-4), np.full(ni, 2.0 ** -10)
    nb6.gpunb_open(n, 0)
    try:
        nb6.gpunb_send(m, x, v)
        if seg:
            out = nb6.regf_seg(h2, dtr, xi, vi, np.repeat(np.arange(nseg), na), np.arange(nseg + 1) * nc, 64, 50, 0)
        else:
            nb6.lib.nb6_regf_tune_(C.byref(C.c_int(-1)), C.byref(C.c_int(0)))
            out = nb6.gpunb_regf(h2, dtr, xi, vi, 64, 50, 0)
    finally:
        nb6.lib.nb6_regf_tune_(C.byref(C.c_int(0)), C.byref(C.c_int(0)))
        nb6.gpunb_close()
    bound = ((32 if seg else 128) / 2 + 6) * 2.0 ** -24
    for k in range(0, ni, 250):
        s = slice(k // na * nc, (k // na + 1) * nc)
        dx, dv = x[s] - xi[k], v[s] - vi[k]
        r2 = (dx * dx).sum(1)
        mr3 = m[s] / (r2 * np.sqrt(r2))
        al = -3.0 * (dx * dv).sum(1) / r2
        for got, ref in ((out[0][k], (mr3[:, None] * dx).sum(0)),
                         (out[1][k], (mr3[:, None] * (dv + al[:, None] * dx)).sum(0)),
                         (out[2][k:k + 1], (m[s] / np.sqrt(r2)).sum(keepdims=True))):
            assert np.linalg.norm(got - ref) <= bound * np.linalg.norm(ref)
        assert out[3][k, 0] == 0


def test_close_gives_the_device_memory_back(nb6):
    """A session over a set larger than any before it, through every layout and
    kernel form of the regular force: what it took on the device is free again
    after the close (but for what the context keeps for its kernels: a first,
    small session loads those; allocations come in units of 2 MB)."""
    import torch
    rng = np.random.default_rng(3)

    def session(n):
        x, v, m = rng.normal(size=(n, 3)), 0.1 * rng.normal(size=(n, 3)), np.full(n, 1.0 / n)
        ni = 300
        h2, dtr = np.full(ni, 1e-4), np.full(ni, 2.0 ** -8)
        nb6.gpunb_open(n, 0)
        try:
            nb6.gpunb_send(m, x, v)
            for variant in (11, 13, 12, -4, 1, 11):
                nb6.lib.nb6_regf_tune_(C.byref(C.c_int(variant)), C.byref(C.c_int(0)))
                last = nb6.gpunb_regf(h2, dtr, x[:ni], v[:ni], 512, 400, 0)
            iseg, j0 = np.repeat([0, 1], ni // 2), np.array([0, n // 2, n])
            nb6.regf_seg(h2, dtr, x[:ni], v[:ni], iseg, j0, 512, 400, 0)
        finally:
            nb6.lib.nb6_regf_tune_(C.byref(C.c_int(0)), C.byref(C.c_int(0)))
            nb6.gpunb_close()
        return last

    session(40000)
    free = torch.cuda.mem_get_info()[0]
    n = 1500000
    state = rng.bit_generator.state
    first = session(n)
    assert free - torch.cuda.mem_get_info()[0] <= 8 << 20
    rng.bit_generator.state = state
    for a, b in zip(first, session(n)):     # and a session after it starts afresh
        np.testing.assert_array_equal(a, b)
