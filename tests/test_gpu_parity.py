"""GPU parity: eps bit for bit, counts exactly, estimates within 1e-10 nats.

Against (1) the golden vectors made by the live reference (cKDTree) and (2)
the CPU oracle at sizes that have no fixture, for every kernel variant: the
FP32 filter with FP64 recheck (default) and all-FP64 (plain), each as brute
force and as sorted slab.
"""

import numpy as np
import pytest

from ennemi_gb300 import _entropy_estimators as E
from ennemi_gb300 import _native as N
from conftest import estimator_cases, inputs_of, outputs_of

pytestmark = pytest.mark.gpu

CASES = estimator_cases()
VARIANTS = {
    "fp32": 0,
    "fp32-brute": N.FORCE_BRUTE,
    "fp32-slab": N.FORCE_SLAB,
    "fp32-grid": N.FORCE_GRID,
    "fp32-ctagrid": N.FORCE_GRID | N.FORCE_CTA_GRID,
    "fp32-rank": N.FORCE_RANK,
    "fp64-brute": N.PLAIN_FP64 | N.FORCE_BRUTE,
    "fp64-slab": N.PLAIN_FP64 | N.FORCE_SLAB,
    "fp64-grid": N.PLAIN_FP64 | N.FORCE_GRID,
}
SLOTS = {"mi": ["nx", "ny"], "cmi": ["nxz", "nyz", "nz"], "semi": ["n"],
         "csemi": ["nxz", "nyz", "nz"], "ent": [],
         "dent": ["c"], "dmi": ["cxy", "cx", "cy"], "dcmi": ["cxyz", "cxz", "cyz", "cz"]}
TOL = 1e-10  # nats


def make_task(kind, k, inp):
    if kind == "mi":
        return E.mi_task(inp["x"], inp["y"], k)
    if kind == "cmi":
        return E.cmi_task(inp["x"], inp["y"], inp["z"], k)
    if kind == "semi":
        return E.semidiscrete_task(inp["x"], inp["y"], k)
    if kind == "csemi":
        return E.conditional_semidiscrete_task(inp["x"], inp["y"], inp["z"], k)
    if kind == "dent":
        return E.discrete_entropy_task(inp["x"])
    if kind == "dmi":
        return E.discrete_mi_task(inp["x"], inp["y"])
    if kind == "dcmi":
        return E.discrete_cmi_task(inp["x"], inp["y"], inp["z"])
    return E.entropy_task(inp["x"], k)


def same_value(a, b, tol=TOL):
    if np.isnan(a) or np.isnan(b):
        return np.isnan(a) and np.isnan(b)
    if np.isinf(a) or np.isinf(b):
        return a == b
    return abs(a - b) <= tol


def check_internals(i, kind, n, eps_ref, counts_ref):
    if eps_ref is not None:
        eps = N.fetch(i, 0, n)
        assert np.array_equal(eps.view(np.uint64), np.asarray(eps_ref, np.float64).view(np.uint64)), \
            f"eps differs at {np.flatnonzero(eps != eps_ref)[:10]}"
    for s, name in enumerate(SLOTS[kind]):
        c = N.fetch(i, 1 + s, n)
        ref = np.asarray(counts_ref[name]).astype(np.int64)
        assert np.array_equal(c, ref), f"{name} differs at {np.flatnonzero(c != ref)[:10]}"


@pytest.mark.parametrize("variant", list(VARIANTS))
@pytest.mark.parametrize("case", CASES, ids=[c["name"] for c in CASES])
def test_golden_estimators(case, variant):
    kind, k = str(case["kind"]), int(case["k"])
    inp = inputs_of(case)
    task = make_task(kind, k, inp)
    vals = N.run_tasks([task], flags=VARIANTS[variant] | N.KEEP_INTERNALS)
    gold = outputs_of(case)
    check_internals(0, kind, task.n, gold.get("eps"), gold)
    assert same_value(vals[0], float(case["value"])), (vals[0], float(case["value"]))


@pytest.mark.parametrize("variant", ["fp32", "fp64-slab", "fp32-grid", "fp32-rank"])
def test_golden_all_in_one_batch(variant):
    tasks = [make_task(str(c["kind"]), int(c["k"]), inputs_of(c)) for c in CASES]
    vals = N.run_tasks(tasks, flags=VARIANTS[variant] | N.KEEP_INTERNALS)
    for i, c in enumerate(CASES):
        gold = outputs_of(c)
        check_internals(i, str(c["kind"]), tasks[i].n, gold.get("eps"), gold)
        assert same_value(vals[i], float(c["value"])), c["name"]


def _oracle_case(O, kind, k, inp):
    with np.errstate(all="ignore"):
        if kind == "mi":
            return O.ksg_mi(inp["x"], inp["y"], k)
        if kind == "cmi":
            return O.cmi(inp["x"], inp["y"], inp["z"], k)
        if kind == "semi":
            return O.semidiscrete_mi(inp["x"], inp["y"], k)
        if kind == "csemi":
            return O.conditional_semidiscrete_mi(inp["x"], inp["y"], inp["z"], k)
        return O.entropy(inp["x"], k)


def _medium_cases():
    rng = np.random.default_rng(2024)
    n = 20000
    g = rng.multivariate_normal([0, 0], [[1, 0.6], [0.6, 1]], size=n)
    yield "mi_gauss_20k", "mi", 3, dict(x=g[:, 0], y=g[:, 1])
    t = rng.standard_t(3, size=n)
    yield "mi_t3_lognormal_20k", "mi", 3, dict(x=t, y=np.exp(rng.normal(size=n)) + 0.1 * t)
    c3 = rng.multivariate_normal([0, 0, 0], [[1, .5, .4], [.5, 1, .4], [.4, .4, 1]], size=n)
    yield "cmi_gauss3_20k", "cmi", 3, dict(x=c3[:, 0], y=c3[:, 1], z=c3[:, 2:])
    c4 = rng.normal(size=(12000, 4))
    yield "cmi_dz2_12k_k5", "cmi", 5, dict(x=c4[:, 0], y=c4[:, 1] + c4[:, 0], z=c4[:, 2:])
    cls = rng.choice(5, p=[0.5, 0.2, 0.2, 0.08, 0.02], size=n)
    yield "semi_x2_5cls_20k", "semi", 3, dict(x=rng.normal(size=(n, 2)) + cls[:, None] * 0.3, y=cls)
    cls2 = (rng.uniform(size=15000) * 3).astype(int)
    yield "csemi_15k", "csemi", 2, dict(x=rng.normal(size=15000) + cls2, y=cls2,
                                          z=rng.normal(size=(15000, 1)))
    yield "ent_3d_20k", "ent", 3, dict(x=rng.normal(size=(n, 3)))
    yield "ent_1d_20k_k40", "ent", 40, dict(x=rng.normal(size=n))
    yield "mi_k40_8k", "mi", 40, dict(x=g[:8000, 0], y=g[:8000, 1])
    yield "mi_rounded_20k", "mi", 3, dict(x=np.round(g[:, 0], 2), y=np.round(g[:, 1], 2))
    yield "ent_9d_3k", "ent", 4, dict(x=rng.normal(size=(3000, 9)))
    big = rng.normal(size=(5000, 2))
    yield "mi_huge_unsafe32_5k", "mi", 3, dict(x=1e300 * big[:, 0], y=big[:, 1])
    # nested-cell grids (d >= 3): generic d, heavy ties, K = 8, 4-D counts
    yield "ent_5d_12k", "ent", 3, dict(x=rng.normal(size=(12000, 5)))
    c3r = np.round(c3, 1)
    yield "cmi_rounded3_20k", "cmi", 3, dict(x=c3r[:, 0], y=c3r[:, 1], z=c3r[:, 2:])
    yield "ent_3d_k7_20k", "ent", 7, dict(x=rng.standard_t(4, size=(n, 3)))
    c6 = rng.normal(size=(10000, 5))
    yield "cmi_dz3_10k", "cmi", 3, dict(x=c6[:, 0], y=c6[:, 1] + 0.5 * c6[:, 2], z=c6[:, 2:])
    # walk kNN / key-range counts: exact duplicates (K-th distance 0, counts
    # with negative radius), K = 8 in 2-D, a job just above the grid size
    dup = rng.integers(0, 40, size=(20000, 2)).astype(np.float64)
    yield "mi_duplicates_20k", "mi", 3, dict(x=dup[:, 0], y=dup[:, 1])
    yield "mi_k7_20k", "mi", 7, dict(x=g[:, 0], y=g[:, 1] ** 3)
    yield "mi_4100", "mi", 3, dict(x=g[:4100, 0], y=g[:4100, 1])
    yield "cmi_dup_z_15k", "cmi", 3, dict(x=c3[:15000, 0], y=c3[:15000, 1],
                                           z=np.round(c3[:15000, 2:], 0))
    # ball ends from FP32 brackets: values far below the FP32 normal range
    # (bracket holds everything -> exact path), scales spread over 40 decades,
    # and balls whose left end crosses zero
    yield "mi_tiny_scales_12k", "mi", 3, dict(x=1e-30 * g[:12000, 0], y=1e-42 * g[:12000, 1])
    spread = 10.0 ** rng.uniform(-20, 20, size=n)
    yield "mi_spread_scales_20k", "mi", 3, dict(x=g[:, 0] * spread, y=g[:, 1])
    near0 = np.concatenate([rng.uniform(-1e-3, 1e-3, size=10000), rng.normal(size=10000)])
    yield "cmi_near_zero_20k", "cmi", 3, dict(x=near0, y=near0[::-1] + 0.1 * g[:, 1],
                                               z=np.abs(near0)[:, None])


MEDIUM = list(_medium_cases())


@pytest.mark.parametrize("variant", ["fp32", "fp32-brute", "fp32-slab", "fp32-ctagrid", "fp64-grid"])
@pytest.mark.parametrize("case", MEDIUM, ids=[c[0] for c in MEDIUM])
def test_medium_against_oracle(oracle, case, variant):
    name, kind, k, inp = case
    ref_value, ref = _oracle_case(oracle, kind, k, inp)
    task = make_task(kind, k, inp)
    vals = N.run_tasks([task], flags=VARIANTS[variant] | N.KEEP_INTERNALS)
    check_internals(0, kind, task.n, ref["eps"], ref)
    assert same_value(vals[0], ref_value), (vals[0], ref_value)


def test_ball_count_radius_on_exact_distances(oracle):
    """Radii equal to exact coordinate distances of dyadic data: every
    boundary is a tie that the inclusive test keeps."""
    rng = np.random.default_rng(11)
    for d in [1, 2]:
        pts = rng.integers(-4000, 4000, size=(9000, d)) / 64.0
        r = rng.integers(0, 200, size=9000) / 64.0
        r[::50] = 0.0
        r[7::50] = -0.0
        cnt = N.ball_count(pts, r)
        assert np.array_equal(cnt, oracle.ball_count(pts, r)), d


def test_primitives_against_oracle(oracle):
    rng = np.random.default_rng(5)
    for d in [1, 2, 3, 6]:
        pts = rng.normal(size=(7000, d))
        for k in [1, 3, 50]:
            eps = N.knn_eps(pts, k)
            assert np.array_equal(eps, oracle.knn_eps(pts, k)), (d, k)
        r = np.abs(rng.normal(0.05, 0.05, size=7000))
        r[::97] = -1e-13
        r[5] = np.inf
        cnt = N.ball_count(pts, r)
        assert np.array_equal(cnt, oracle.ball_count(pts, r)), d


@pytest.mark.parametrize("data", ["normal", "rounded", "huge"])
@pytest.mark.parametrize("d", [2, 3, 4, 5])
def test_warp_list_knn(oracle, d, data):
    """K at the edges of the list sizes and of the compiled classes, at the
    smallest grid size, one point below it and odd sizes above; near ties that
    overflow the list, and values that rule out the FP32 screen."""
    rng = np.random.default_rng(10 * d)
    sizes = [4095, 4096, 9001] if data == "normal" else [4097]
    for n in sizes:
        pts = rng.normal(size=(n, d)) * np.linspace(1.0, 3.0, d)
        if data == "rounded":
            pts = np.round(pts, 0 if d > 3 else 1)
        elif data == "huge":
            pts[:, 0] *= 1e300
        for k in [3, 7, 8, 15, 16, 31, 32, 63, 64, 127, 128]:
            eps = N.knn_eps(pts, k)
            assert np.array_equal(eps, oracle.knn_eps(pts, k)), (n, k)
    few = rng.normal(size=(40, d))
    for k in [32, 38, 39, 40, 127]:
        assert np.array_equal(N.knn_eps(few, k), oracle.knn_eps(few, k)), k


def _noisy_levels(n, d, rng, step):
    """Columns of a few levels with 1e-10 of noise: FP32 cannot tell a level's points apart."""
    return np.round(rng.normal(size=(n, d)) / step) * step + 1e-10 * rng.normal(size=(n, d))


@pytest.mark.parametrize("d", [2, 3, 4, 5])
@pytest.mark.parametrize("n", [333, 2000, 5001])
def test_crowded_queries(oracle, n, d):
    """More near ties than a list holds, over all points and over grids, with
    exact ties among them, at the edges of the list sizes."""
    pts = _noisy_levels(n, d, np.random.default_rng(n + d), 0.8)
    pts[1:-1:5] = pts[2::5][: len(pts[1:-1:5])]
    crowded = 0
    for k in [1, 3, 7, 8, 15, 16, 31, 32, 63, 64, 127]:
        assert np.array_equal(N.knn_eps(pts, k), oracle.knn_eps(pts, k)), k
        crowded += N.context(0).stats()["knn_deferred"]
    assert crowded > n // 4


@pytest.mark.parametrize("n,d,k", [(20_000, 2, 20), (20_000, 2, 50), (20_000, 3, 20)])
def test_crowded_queries_cost_a_sweep_not_eight(n, d, k):
    """The warp list's searches over noisy levels take no longer than those of
    the tiles that it replaces (K <= 32), or eight times as long as over normal
    data (device times)."""
    rng = np.random.default_rng(n + k)
    ctx = N.context(0)

    def device_ms(pts, flags):
        best = np.inf
        for _ in range(4):
            N.knn_eps(pts, k, flags=flags | N.TIMING)
            best = min(best, ctx.timings()["knn"])
        return best

    crowded = device_ms(_noisy_levels(n, d, rng, 0.8), 0)
    assert ctx.stats()["knn_deferred"] > n // 2
    if k < 32:
        assert crowded < device_ms(_noisy_levels(n, d, rng, 0.8), N.FORCE_CTA_GRID)
    else:
        assert crowded < 8 * device_ms(rng.normal(size=(n, d)), 0)


@pytest.mark.parametrize("data", ["normal", "dyadic", "duplicates", "huge"])
@pytest.mark.parametrize("d", [3, 4, 5])
def test_leaf_counts(oracle, d, data):
    """Ball counts over leaf boxes: the smallest grid, odd sizes, radii from
    nothing to everything in one item (leaf lists that overflow), boundaries
    on exact distances, and values that rule out the FP32 screen."""
    rng = np.random.default_rng(100 + d)
    for n in [4096, 4097, 9001]:
        pts = rng.normal(size=(n, d)) * np.linspace(1.0, 2.0, d)
        r = np.abs(rng.normal(0.3, 0.2, size=n))
        if data == "dyadic":
            pts = rng.integers(-300, 300, size=(n, d)) / 64.0
            r = rng.integers(0, 120, size=n) / 64.0
        elif data == "duplicates":
            pts = rng.integers(0, 6, size=(n, d)).astype(np.float64)
            r = rng.integers(0, 4, size=n) - 1e-12
        elif data == "huge":
            pts[:, 1] *= 1e300
            r[::2] *= 1e300
        r[::97] = -1e-13
        r[1::97] = 0.0
        r[2::97] = np.inf
        r[3::97] = 1e3
        r[4::97] = np.nan
        r[5::97] = -0.0
        assert np.array_equal(N.ball_count(pts, r), oracle.ball_count(pts, r)), n


@pytest.mark.parametrize("data", ["normal", "dyadic", "duplicates", "fine", "tiny", "huge"])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 2049, 9001, 311_295, 311_297, 400_003])
def test_window_counts(n, data):
    """1-D ball counts through windows of the sorted values: a few points and
    the first sizes of each block span, balls from nothing to everything (ends
    inside the window, past its edge and past the segment), boundaries on exact
    distances, and values that an FP32 bracket cannot tell apart or hold."""
    rng = np.random.default_rng(n)
    x = rng.normal(size=n)
    r = np.abs(rng.normal(0.0, 3.0 / np.sqrt(n), size=n))
    if data == "dyadic":
        x = rng.integers(-3000, 3000, size=n) / 64.0
        r = rng.integers(0, 120, size=n) / 64.0
    elif data == "duplicates":
        x = rng.integers(0, 6, size=n).astype(np.float64)
        r = rng.integers(0, 4, size=n) - 1e-12
    elif data == "fine":
        x = 1.0 + x * 1e-9
        r *= 1e-9
    elif data == "tiny":
        x *= 1e-42
        r *= 1e-42
    elif data == "huge":
        x[::2] *= 1e300
        r[::3] *= 1e300
    r[::97] = -1e-13
    r[1::97] = 0.0
    r[2::97] = np.inf
    r[3::97] = 1e3
    r[4::97] = np.nan
    r[5::97] = -0.0
    r[6::97] = 0.5
    got = N.ball_count(x[:, None], r)
    rows = np.unique(np.concatenate([np.arange(min(n, 40)), np.argsort(x)[[0, -1]], rng.integers(0, n, 160)]))
    for i in rows:
        assert got[i] == np.count_nonzero(np.abs(x - x[i]) <= r[i]), i


@pytest.mark.parametrize("n", [300, 9001, 180_000])
def test_window_counts_on_noisy_levels(n):
    """Brackets with no, a few and thousands of values that FP32 cannot tell apart."""
    rng = np.random.default_rng(n)
    x = np.round(rng.normal(size=n), 1) + 1e-10 * rng.normal(size=n)
    x[:: 7] += rng.normal(size=len(x[:: 7]))
    r = rng.choice([1e-10, 3e-9, 0.1, 0.1 + 1e-10, 0.05], size=n)
    got = N.ball_count(x[:, None], r)
    for i in [*range(60), *rng.integers(0, n, 200)]:
        assert got[i] == np.count_nonzero(np.abs(x - x[i]) <= r[i]), i


def test_window_counts_on_noisy_levels_keep_pace():
    """Device times of the 1-D counts, against those of continuous columns: the
    exact search of each end and a short walk before it (3.6 times; with a long
    one 5.7)."""
    rng = np.random.default_rng(4)
    ctx = N.context(0)

    def counts_ms(step):
        x = [rng.normal(size=180_000) for _ in range(8)]
        if step:
            x = [np.round(v / step) * step + 1e-10 * rng.normal(size=len(v)) for v in x]
        tasks = [N.Task(N.MI, 3, [x[i]], [x[i + 1]]) for i in range(0, 8, 2)]
        best = np.inf
        for _ in range(5):
            N.run_tasks(tasks, flags=N.TIMING)
            best = min(best, ctx.timings()["count_1d"])
        return best

    assert counts_ms(0.1) < 4.5 * counts_ms(0.0)


def _code_columns(data, n, rng):
    x = rng.normal(size=n)
    if data == "offset":
        x += 1e6
    elif data == "near":      # short runs of equal codes, out of order
        x = rng.permutation(np.concatenate([x[: n // 4] + j * 2.0 ** -40 for j in range(4)] + [x[: n % 4]]))
    elif data == "levels":    # long runs of equal values
        x = np.round(x * 2.0)
    elif data == "zeros":     # both zeros
        x = np.where(rng.random(n) < 0.5, np.copysign(0.0, x), x)
    elif data == "cluster":   # a long run of equal codes, out of order
        x[: n // 50] = 3.0 + rng.permutation(n // 50) * 2.0 ** -40
    elif data == "twins":     # runs around the longest that is repaired
        x = rng.permutation(np.concatenate([v + rng.permutation(m) * 2.0 ** -45 for m in (31, 32, 33, 34)
                                            for v in rng.normal(size=n // 8 // m)] + [x])[:n])
    elif data == "huge":
        x[::3] *= 1e300
    elif data == "tiny":
        x *= 1e-300
    elif data == "cauchy":
        x = rng.standard_cauchy(size=n)
    elif data == "outlier":
        x[n // 2] = 1e7
    elif data == "one_huge":  # everything else shares a code
        x[0] = 1e308
    return x


@pytest.mark.parametrize("data", ["normal", "offset", "near", "levels", "zeros", "cluster", "twins", "huge",
                                  "tiny", "cauchy", "outlier", "one_huge"])
def test_code_sort_equals_the_digit_sort(data):
    """A batch large enough for the code sort returns, for segments of one
    point up to several tiles, exactly what each of its tasks returns alone."""
    rng = np.random.default_rng(17)
    sizes = [5, 40, 2047, 2049, 4096, 4097, 60_001, 500_000, 500_003]
    tasks = []
    for n in sizes:
        x = _code_columns(data, n, rng)
        tasks.append(N.Task(N.MI, 3, [x], [0.5 * x + rng.normal(size=n)]))
    ctx = N.context(0)
    both = N.run_tasks(tasks, flags=N.KEEP_INTERNALS)
    # "twins": runs too long to repair both in their codes and in 48 key bits
    assert ctx.stats()["sort_passes"] == (8 if data == "twins" else 4)
    kept = [[N.fetch(t, w, n) for w in (0, 1, 2)] for t, n in enumerate(sizes)]
    for t, n in enumerate(sizes):
        alone = N.run_tasks([tasks[t]], flags=N.KEEP_INTERNALS)
        assert ctx.stats()["sort_passes"] != 4
        assert np.array_equal(alone[0], both[t], equal_nan=True), n
        for w in (0, 1, 2):
            assert np.array_equal(N.fetch(0, w, n), kept[t][w], equal_nan=True), (n, w)


@pytest.mark.parametrize("n", [300, 9001])
@pytest.mark.parametrize("d", [1, 2, 3])
def test_counts_about_points_that_are_not_finite(d, n):
    """No point lies within a finite distance of an infinite or NaN one, itself
    included; such points are in no finite ball."""
    rng = np.random.default_rng(n + d)
    pts = rng.normal(size=(n, d))
    pts[[5, 6, 7, n // 2], d - 1] = [np.inf, -np.inf, np.nan, np.inf]
    r = np.abs(rng.normal(0.3, 0.2, size=n))
    r[9] = 0.0
    for flags in (0, N.FORCE_BRUTE, N.FORCE_RANK if d == 2 else N.FORCE_GRID):
        got = N.ball_count(pts, r, flags=flags)
        for i in [*range(40), n // 2, n - 1]:
            with np.errstate(invalid="ignore"):
                dist = np.abs(pts - pts[i]).max(axis=1)
            assert got[i] == np.count_nonzero(dist <= r[i]), (flags, i)


def test_labels_and_index_at_any_address():
    """int32 arrays that are not 4-byte aligned: never read where they are."""
    rng = np.random.default_rng(8)
    n = 24_001

    def unaligned(a):
        raw = np.zeros(a.nbytes + 4, dtype=np.uint8)
        raw[1:1 + a.nbytes] = a.view(np.uint8)
        return raw[1:1 + a.nbytes].view(np.int32)

    lab = rng.integers(0, 5, n).astype(np.int32)
    idx = np.sort(rng.choice(2 * n, n, replace=False)).astype(np.int32)
    x, u, v = rng.normal(size=n), rng.normal(size=2 * n), rng.normal(size=2 * n)
    for labels, index in ((lab, idx), (unaligned(lab), unaligned(idx))):
        assert labels.flags.aligned == (labels is lab)
        got = N.run_tasks([N.Task(N.SEMI, 3, [x], labels=labels, nclass=5, n=n),
                           N.Task(N.MI, 3, [u], [v], n=n, index=index)])
        if labels is lab:
            want = got
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n,k,data", [(270_000, 127, "normal"), (270_000, 127, "levels"), (270_000, 127, "huge"),
                                      (650_000, 52, "normal"), (4_300_000, 3, "normal")])
def test_strips_longer_than_a_block_orders(n, k, data):
    """Two-column grids whose strips exceed 4096 points are laid out by sorted
    strip keys: lists from n K = 3.3e7 on, walks from 4.2 million points."""
    rng = np.random.default_rng(k)
    pts = rng.normal(size=(n, 2))
    if data == "levels":
        pts = np.round(pts, 2) + 1e-10 * rng.normal(size=(n, 2))
    elif data == "huge":
        pts[:, 1] *= 1e300
    eps = N.knn_eps(pts, k)
    assert N.context(0).stats()["knn_tile_pairs"] < n * (n // 8) or data == "huge"
    far = np.argsort(np.abs(pts[:, 0]))[-3:]
    for i in [0, n - 1, *far, *rng.integers(0, n, 40 if n < 10 ** 6 else 10)]:
        assert eps[i] == np.partition(np.abs(pts - pts[i]).max(axis=1), k)[k], i


def _long_runs(n, lengths, rng):
    """Normal values, and runs of them 2^-40 apart: equal codes, out of order."""
    x = rng.normal(size=n)
    end = 0
    for m in lengths:
        x[end:end + m] = rng.choice([-1.3, 1.3]) + 0.2 * rng.random() + rng.permutation(m) * 2.0 ** -40
        end += m
    return rng.permutation(x)


@pytest.mark.parametrize("lengths", [[33], [33, 34, 63, 64, 65, 127, 128, 129], [255, 256, 257, 500, 1024],
                                     [2047, 2048], [2049], [2048, 2049, 33, 6000], [40] * 900])
def test_long_runs_of_equal_codes(lengths):
    """Runs at the edges of the forms that put them in order, and beyond the
    longest: what each task returns alone, without codes."""
    rng = np.random.default_rng(sum(lengths))
    sizes = [60_001, 500_000, 500_003]
    tasks = []
    for n in sizes:
        x = _long_runs(n, lengths, rng)
        tasks.append(N.Task(N.MI, 3, [x], [0.5 * x + rng.normal(size=n)]))
    ctx = N.context(0)
    both = N.run_tasks(tasks, flags=N.KEEP_INTERNALS)
    assert ctx.stats()["sort_passes"] == 4
    kept = [[N.fetch(t, w, n) for w in (0, 1, 2)] for t, n in enumerate(sizes)]
    for t, n in enumerate(sizes):
        assert N.run_tasks([tasks[t]], flags=N.KEEP_INTERNALS)[0] == both[t], n
        for w in (0, 1, 2):
            assert np.array_equal(N.fetch(0, w, n), kept[t][w]), (n, w)


def test_columns_with_repeated_values_are_sorted_once():
    """A tenth of a percent of each column rescaled from one value: its run of
    equal codes is put in order where it is.  The codes' sort alone is the measure;
    sorting the segments again by their digits takes 2.5 times as long."""
    n = 180_000
    rng = np.random.default_rng(3)
    ctx = N.context(0)

    def sort_ms(share):
        cols = []
        for _ in range(40):
            x = rng.normal(size=n)
            x[rng.random(n) < share] = 0.7
            cols.append(x + 1e-10 * rng.normal(size=n))
        tasks = [N.Task(N.MI, 3, [cols[i]], [cols[i + 1]], n=n) for i in range(0, 40, 2)]
        best = np.inf
        for _ in range(4):
            N.run_tasks(tasks, flags=N.TIMING)
            best = min(best, ctx.timings()["sort_radix"])
        assert ctx.stats()["sort_passes"] == 4
        return best

    assert sort_ms(0.001) < 2.0 * sort_ms(0.0)


def _small_points(data, n, d, rng):
    x = rng.normal(size=(n, d))
    if data == "duplicates":
        x = rng.integers(0, 4, size=(n, d)).astype(np.float64)
    elif data == "huge":
        x[:, 0] *= 1e300
    elif data == "offset":
        x += 1e9
    return x


@pytest.mark.parametrize("data", ["normal", "duplicates", "huge", "offset"])
@pytest.mark.parametrize("d", [2, 3, 4, 5])
def test_small_knn(oracle, d, data):
    """kNN of sets too small for a layout of their own: fewer points than
    neighbours, the warp's widths, both sides of the smallest grid."""
    rng = np.random.default_rng(40 + d)
    for n in [1, 2, 9, 31, 33, 65, 700, 1023, 1025, 4095]:
        pts = _small_points(data, n, d, rng)
        for k in [1, 3, 7, 8, 31] if n < 1000 else [3, 8]:
            assert np.array_equal(N.knn_eps(pts, k), oracle.knn_eps(pts, k)), (n, k)


@pytest.mark.parametrize("data", ["normal", "duplicates", "huge", "offset"])
@pytest.mark.parametrize("count, n", [(3, 2000), (26, 2000), (11, 4095), (100, 1024), (320, 40), (320, 900)])
def test_small_batches_take_the_form_that_fits(count, n, data):
    """Batches of small sets, from a few to those that get grids or fill the
    tile kernel, against brute force."""
    rng = np.random.default_rng(count)
    tasks = []
    for i in range(count):
        x = _small_points(data, n, 4, rng)
        y = 0.5 * x[:, 0] + rng.normal(size=n)
        tasks.append(N.Task(N.MI, 3, [x[:, 0].copy()], [y]) if i % 2 else
                     N.Task(N.CMI, 3, [x[:, 0].copy()], [y], [x[:, 1].copy(), x[:, 2].copy()][: 1 + i % 4 // 2]))
    flags = N.KEEP_INTERNALS | N.TIMING
    got = N.run_tasks(tasks, flags=flags)
    kept = [N.fetch(t, 0, n) for t in range(0, count, 7)]
    want = N.run_tasks(tasks, flags=flags | N.FORCE_BRUTE)
    assert np.array_equal(got, want, equal_nan=True)
    for t, e in zip(range(0, count, 7), kept):
        assert np.array_equal(N.fetch(t, 0, n), e, equal_nan=True), t


@pytest.mark.parametrize("nclass", [1, 2, 255, 256, 257, 900])
@pytest.mark.parametrize("n", [19_999, 20_000, 20_480, 70_001])
def test_class_order_on_the_device(n, nclass):
    """Class orders built on the device (the sizes about where it starts; one
    and two label bytes, empty classes) give what the host's order gives."""
    rng = np.random.default_rng(n + nclass)
    used = rng.permutation(nclass)[: max(1, nclass - nclass // 4)]
    tasks = []
    for kind in (N.SEMI, N.CSEMI, N.SEMI):
        lab = np.sort(rng.choice(used, n)) if len(tasks) == 2 else rng.choice(used, n)
        x = rng.normal(size=n) + 0.1 * lab / nclass
        tasks.append(N.Task(kind, 3, [x], [], [rng.normal(size=n)] if kind == N.CSEMI else [],
                            labels=lab.astype(np.int32), nclass=nclass, n=n))
    host = N.run_tasks(tasks, flags=N.KEEP_INTERNALS)
    for flags in (0, N.STAGE_HOST, N.TIMING):
        assert np.array_equal(N.run_tasks(tasks, flags=flags), host, equal_nan=True), flags
    bad = tasks[0].labels.copy()
    bad[-1] = nclass
    with pytest.raises(RuntimeError, match="label out of range"):
        N.run_tasks([N.Task(N.SEMI, 3, [x], [], [], labels=bad, nclass=nclass, n=n)])


@pytest.mark.parametrize("data", ["independent", "cubic", "square", "steps", "constant", "huge"])
@pytest.mark.parametrize("n", [4096, 4099, 20_001])
def test_strip_layouts(oracle, n, data):
    """Two-column grids built strip by strip: column-0 ranks spread over a
    strip's buckets, crowded into few of them (columns that are functions of
    each other), ties, and values that rule out the FP32 copy."""
    rng = np.random.default_rng(n)
    x = rng.normal(size=n)
    y = {"independent": rng.normal(size=n), "cubic": x ** 3, "square": x ** 2, "steps": np.round(x),
         "constant": np.full(n, 2.5), "huge": x * 1e300}[data]
    pts = np.column_stack((x, y))
    for k in (3, 20):
        assert np.array_equal(N.knn_eps(pts, k), oracle.knn_eps(pts, k)), k
    assert np.array_equal(N.knn_eps(pts[:, ::-1], 3), oracle.knn_eps(pts, 3))


def _small_tasks(rng, n, k, data):
    """Every estimator that the direct path serves, over n samples."""
    lab = rng.integers(0, 3, size=n).astype(np.int32)
    c = rng.normal(size=(n, 5))
    c[:, 1] += 0.6 * c[:, 0]
    if data == "rounded":
        c = np.round(c, 1)
    elif data == "duplicates":
        c = rng.integers(0, 3, size=(n, 5)).astype(np.float64)
    elif data == "huge":
        c[:, 0] *= 1e300
    elif data == "infinite":
        c[n // 2, 1] = np.inf
    col = [np.ascontiguousarray(v) for v in c.T]
    seen = np.unique(lab)
    lab = np.searchsorted(seen, lab).astype(np.int32)
    T, m = N.Task, len(seen)
    return [T(N.MI, k, col[:1], col[1:2], n=n), T(N.CMI, k, col[:1], col[1:2], col[2:3], n=n),
            T(N.CMI, k, col[:1], col[1:2], col[2:4], n=n), T(N.CMI, k, col[:1], col[1:2], col[2:], n=n),
            T(N.SEMI, k, col[:1], labels=lab, nclass=m, n=n), T(N.SEMI, k, col[:3], labels=lab, nclass=m, n=n),
            T(N.CSEMI, k, col[:1], (), col[1:2], labels=lab, nclass=m, n=n),
            T(N.CSEMI, k, col[:1], (), col[1:3], labels=lab, nclass=m, n=n),
            T(N.ENTROPY, k, col[:1], n=n), T(N.ENTROPY, k, col[:2], n=n), T(N.ENTROPY, k, col[:4], n=n)]


@pytest.mark.parametrize("data", ["normal", "rounded", "duplicates", "huge", "infinite"])
@pytest.mark.parametrize("n,k", [(1, 1), (2, 1), (5, 4), (31, 3), (32, 3), (33, 31), (64, 15), (65, 16),
                                 (257, 63), (300, 64), (1000, 3), (1024, 5), (1025, 3), (4095, 3), (4096, 3)])
def test_small_batches_equal_the_general_path(n, k, data):
    """The direct path's results -- values, distances and counts -- are those of
    the general path bit for bit: below, at and beyond its limits, with lists
    that near ties overflow and values that send the batch back."""
    tasks = _small_tasks(np.random.default_rng(n + k), n, k, data)
    slots = {N.MI: 2, N.CMI: 3, N.SEMI: 1, N.CSEMI: 3, N.ENTROPY: 0}

    def results(flags, batch):
        v = N.run_tasks(batch, flags=flags | N.KEEP_INTERNALS)
        return v, [[N.fetch(i, w, n) for w in range(1 + slots[t.kind])] for i, t in enumerate(batch)]

    want, inner = results(N.FORCE_BRUTE, tasks)
    got, kept = results(0, tasks)
    assert np.array_equal(got, want, equal_nan=True)
    for a, b in zip(kept, inner):
        for u, w in zip(a, b):
            assert np.array_equal(u.view(np.int64), w.view(np.int64))
    for i in (0, 2, 7):   # a task alone, and as device columns
        alone, k1 = results(0, tasks[i:i + 1])
        assert np.array_equal(alone, want[i:i + 1], equal_nan=True)
        for u, w in zip(k1[0], inner[i]):
            assert np.array_equal(u.view(np.int64), w.view(np.int64))


@pytest.mark.parametrize("data", ["outlier", "cauchy"])
@pytest.mark.parametrize("n,k", [(40, 3), (1000, 3), (1000, 20), (4095, 3)])
def test_small_batches_with_far_values(n, k, data):
    """A value far from all others, and heavy tails: the general path's results
    bit for bit, and few queries whose FP32 distances tie beyond the list."""
    rng = np.random.default_rng(n + k)
    c = rng.normal(size=(n, 4)) if data == "outlier" else rng.standard_cauchy(size=(n, 4))
    if data == "outlier":
        c[n // 2] = 1e6
    col = [np.ascontiguousarray(v) for v in c.T]
    lab = (np.arange(n) % 2).astype(np.int32)
    tasks = [N.Task(N.MI, k, col[:1], col[1:2], n=n), N.Task(N.CMI, k, col[:1], col[1:2], col[2:], n=n),
             N.Task(N.SEMI, k, col[:2], labels=lab, nclass=2, n=n), N.Task(N.ENTROPY, k, col[:3], n=n)]
    want = N.run_tasks(tasks, flags=N.FORCE_BRUTE | N.KEEP_INTERNALS)
    eps = [N.fetch(i, 0, n) for i in range(4)]
    got = N.run_tasks(tasks, flags=N.KEEP_INTERNALS)
    assert np.array_equal(got, want)
    for i in range(4):
        assert np.array_equal(N.fetch(i, 0, n), eps[i]), i
    # the outlier's own query, and the few about as far out as heavy tails go
    assert N.context(0).stats()["knn_deferred"] <= 4 * (1 if data == "outlier" else 0.01 * n)


@pytest.mark.parametrize("shift", [1e6, -1e6])
def test_two_far_clusters_are_centred_between(shift):
    """FP32 steps are 1/32 in either of two clusters 1e6 apart about the middle,
    and 1/16 in the far one about the other's median, whose queries then have four times
    the near ties: 6 % of all pairs are screened, not 11."""
    n = 100_000
    rng = np.random.default_rng(6)
    x = rng.normal(size=(n, 2))
    x[:, 1] = 0.6 * x[:, 0] + 0.8 * x[:, 1]
    pts = x + shift * rng.integers(0, 2, n)[:, None]
    eps = N.knn_eps(pts, 3)
    assert N.context(0).stats()["knn_tile_pairs"] < 0.085 * n * n
    rows = rng.integers(0, n, 50)
    for i in rows:
        assert eps[i] == np.partition(np.abs(pts - pts[i]).max(axis=1), 3)[3]


@pytest.mark.parametrize("n", [9, 129, 1000, 4095])
def test_small_batches_rescale_and_index(n):
    """Strided views, a shared sample index, class orders and conditions of one
    and two columns: the rescaled columns are the general path's bits."""
    from ennemi_gb300 import _driver
    rng = np.random.default_rng(n)
    raw = rng.normal(size=(n + 40, 4)) * [1.0, 3.0, 0.1, 2.0] + [0.0, 5.0, -1.0, 0.0]
    idx = np.sort(rng.choice(n + 30, size=n, replace=False)).astype(np.int32)
    lab = (np.arange(n) % 3).astype(np.int32)
    v = [raw[5:, c] for c in range(4)]
    k = min(3, n - 2)
    tasks = [N.Task(N.MI, k, [v[0]], [v[1]], n=n, index=idx), N.Task(N.MI, k, [v[1]], [v[2]], n=n),
             N.Task(N.CMI, k, [v[0]], [v[1]], [v[2]], n=n, index=idx),
             N.Task(N.CMI, k, [v[0]], [v[1]], [v[2], v[3]], n=n, index=idx),
             N.Task(N.SEMI, k, [v[0]], labels=lab, nclass=3, n=n, index=idx),
             N.Task(N.CSEMI, k, [v[0]], (), [v[1]], labels=lab, nclass=3, n=n)]
    noise = lambda m: _driver._noise.take(0, (m,))
    out = []
    for flags in (N.FORCE_BRUTE, 0):
        r = N.run_tasks(tasks, flags=flags | N.RESCALE | N.KEEP_INTERNALS, noise=noise)
        out.append((r, [N.fetch(t, 16 + c, n) for t, task in enumerate(tasks)
                        for c in range(len(task.x) + len(task.y) + len(task.z))]))
    assert np.array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


def test_device_input_matches_host_input():
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(7)
    x = rng.normal(size=30000)
    y = 0.5 * x + rng.normal(size=30000)
    host = N.run_tasks([E.mi_task(x, y, 3)])
    xd = torch.from_numpy(x).cuda()
    yd = torch.from_numpy(y).cuda()
    dev = N.run_tasks([N.Task(N.MI, 3, [xd], [yd], n=30000)], flags=N.INPUT_DEVICE)
    assert host[0] == dev[0]


def test_host_columns_read_in_place_match_staged_copies():
    """Contiguous host columns may be read by the gather kernel in place
    (devices that read pageable memory); strided, shared and class-permuted
    columns are staged.  Every route gives the same bits."""
    rng = np.random.default_rng(23)
    n = 40000
    a = rng.normal(size=n)
    b = 0.6 * a + rng.normal(size=n)
    m = rng.normal(size=(n, 3))                     # strided column views
    m[:, 1] += 0.5 * m[:, 0]
    lab = rng.integers(0, 4, size=n).astype(np.int32)
    s = a + 0.3 * lab
    tasks = [E.mi_task(a, b, 3),
             N.Task(N.MI, 3, [m[:, 0]], [m[:, 1]], n=n),
             N.Task(N.CMI, 3, [a], [m[:, 1]], [b], n=n),
             N.Task(N.CMI, 4, [m[:, 0], m[:, 2]], [b], [a], n=n),
             N.Task(N.SEMI, 3, [s], labels=lab, nclass=4, n=n),
             N.Task(N.ENTROPY, 3, [b, a], n=n)]
    for extra in (0, N.GRAPH):
        staged = N.run_tasks(tasks, flags=N.STAGE_HOST | extra)
        default = N.run_tasks(tasks, flags=extra)
        assert np.array_equal(staged, default), extra
    # odd lengths, and a column 8 bytes off a 16-byte boundary (read one
    # value per request instead of pairs)
    n2 = 40001
    buf = np.empty(n2 + 1)
    off = buf[1:]
    off[:] = rng.normal(size=n2)
    c = rng.normal(size=n2) + 0.4 * off
    assert c.ctypes.data % 16 == 0 and off.ctypes.data % 16 == 8
    odd = [E.mi_task(c, off, 3), E.cmi_task(off, c, c[::-1].copy(), 3), E.entropy_task(c, 3)]
    assert np.array_equal(N.run_tasks(odd, flags=N.STAGE_HOST), N.run_tasks(odd))
    pts = np.ascontiguousarray(m[:, :2])
    r = N.knn_eps(pts, 3)
    assert np.array_equal(r, N.knn_eps(pts, 3, flags=N.STAGE_HOST))
    assert np.array_equal(N.ball_count(pts, r - 1e-12),
                          N.ball_count(pts, r - 1e-12, flags=N.STAGE_HOST))


def test_public_estimators_on_gpu():
    rng = np.random.default_rng(0)
    cov = [[1, 0.6], [0.6, 1]]
    d = rng.multivariate_normal([0, 0], cov, size=4000)
    mi = E._estimate_single_mi(d[:, 0], d[:, 1], 3)
    assert abs(mi - (-0.5 * np.log(1 - 0.36))) < 0.03
    h = E._estimate_single_entropy(d[:, 0])
    assert abs(h - 0.5 * np.log(2 * np.pi * np.e)) < 0.05


def _tie_cases():
    """Columns whose sort keys tie in their high 48 bits (values within a
    relative 2^-36): the six-pass sort repairs short runs in place and sends
    a long run out of order to the full sort; long runs already in order
    (exact duplicates, or ascending input) need neither."""
    rng = np.random.default_rng(31)
    n = 6000
    v = rng.normal(size=n // 3)
    near = np.concatenate([v, np.nextafter(v, np.inf), np.nextafter(np.nextafter(v, -np.inf), -np.inf)])
    yield "short_runs", rng.permutation(near), 6
    yield "long_run_shuffled", 1.0 + rng.permutation(n) * 2.0 ** -52, 8
    yield "long_run_ascending", 1.0 + np.arange(n) * 2.0 ** -52, 6
    yield "duplicates", rng.integers(0, 7, size=n).astype(np.float64), 6
    mixed = rng.normal(size=n)
    mixed[: n // 2] = 3.0 + rng.permutation(n // 2) * 2.0 ** -51
    yield "half_long_run", rng.permutation(mixed), 8


TIES = list(_tie_cases())


@pytest.mark.parametrize("kind", ["mi", "ent", "cmi"])
@pytest.mark.parametrize("case", TIES, ids=[c[0] for c in TIES])
def test_sort_ties_in_high_bits(oracle, case, kind):
    name, x, passes = case
    rng = np.random.default_rng(5)
    n = len(x)
    y = rng.normal(size=n) + 0.5 * np.argsort(np.argsort(x)) / n
    inp = dict(x=x, y=y, z=rng.normal(size=(n, 1)) + x[:, None] * 0)
    if kind == "ent":
        inp = dict(x=x)
    ref_value, ref = _oracle_case(oracle, kind, 3, inp)
    task = make_task(kind, 3, inp)
    ctx = N.context(0)
    vals = N.run_tasks([task], flags=N.KEEP_INTERNALS)
    assert ctx.stats()["sort_passes"] == passes
    check_internals(0, kind, task.n, ref["eps"], ref)
    assert same_value(vals[0], ref_value), (vals[0], ref_value)


def test_graph_replay_matches_direct_launch():
    """The streaming pattern: capture once, then refill the same device
    buffers and replay without planning.  The expected values of both data
    sets are computed first, by direct launches on other buffers, so that no
    other batch runs on the context between the graph calls."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(21)
    n = 50000
    host_a = [rng.normal(size=n) for _ in range(3)]
    host_b = [host_a[0], 0.7 * host_a[0] + rng.normal(size=n), host_a[2]]

    def tasks_of(cols):
        return [N.Task(N.MI, 3, [cols[0]], [cols[1]], n=n),
                N.Task(N.CMI, 3, [cols[0]], [cols[1]], [cols[2]], n=n)]
    ctx = N.context(0)
    direct_a = N.run_tasks(tasks_of([torch.from_numpy(c).cuda() for c in host_a]), flags=N.INPUT_DEVICE)
    direct_b = N.run_tasks(tasks_of([torch.from_numpy(c).cuda() for c in host_b]), flags=N.INPUT_DEVICE)
    assert not np.array_equal(direct_a, direct_b)

    cols = [torch.from_numpy(c).cuda() for c in host_a]
    tasks = tasks_of(cols)
    first = N.run_tasks(tasks, flags=N.INPUT_DEVICE | N.GRAPH)   # plans and captures
    st = ctx.stats()
    assert st["planned"] == 1 and st["graph"] == 1
    again = N.run_tasks(tasks, flags=N.INPUT_DEVICE | N.GRAPH)   # replays, no planning
    st = ctx.stats()
    assert st["planned"] == 0 and st["graph"] == 1
    assert np.array_equal(direct_a, first) and np.array_equal(direct_a, again)
    # new data in the same buffers: the replay (still without planning) reads them
    cols[1].copy_(torch.from_numpy(host_b[1]))
    torch.cuda.synchronize()
    replay_b = N.run_tasks(tasks, flags=N.INPUT_DEVICE | N.GRAPH)
    st = ctx.stats()
    assert st["planned"] == 0 and st["graph"] == 1
    assert np.array_equal(direct_b, replay_b)


def test_tasks_sharing_columns_match_tasks_alone():
    """Tasks that read the same caller columns share their sort segments and
    rank-space matrices in one batch; every result equals the task run alone
    (eps bit for bit, counts exactly)."""
    rng = np.random.default_rng(31)
    n = 20000
    a, b, c = rng.normal(size=(3, n))
    b += 0.5 * a
    z = rng.normal(size=(n, 2))
    z1, z2 = np.ascontiguousarray(z[:, 0]), np.ascontiguousarray(z[:, 1])
    tasks = [N.Task(N.MI, 3, [a], [b], n=n), N.Task(N.MI, 3, [a], [c], n=n),
             N.Task(N.MI, 3, [b], [c], n=n), N.Task(N.MI, 3, [c], [a], n=n),
             N.Task(N.CMI, 3, [a], [b], [z1], n=n), N.Task(N.CMI, 3, [a], [c], [z1], n=n),
             N.Task(N.CMI, 3, [a], [b], [z1, z2], n=n), N.Task(N.CMI, 3, [b], [c], [z1, z2], n=n),
             N.Task(N.ENTROPY, 3, [a, z1], n=n)]
    slots = {N.MI: 2, N.CMI: 3, N.ENTROPY: 0}
    together = N.run_tasks(tasks, flags=N.KEEP_INTERNALS)
    kept = [[N.fetch(i, w, n) for w in range(1 + slots[t.kind])] for i, t in enumerate(tasks)]
    for i, t in enumerate(tasks):
        alone = N.run_tasks([t], flags=N.KEEP_INTERNALS)
        assert alone[0] == together[i], i
        for w in range(1 + slots[t.kind]):
            assert np.array_equal(N.fetch(0, w, n), kept[i][w]), (i, w)


@pytest.mark.parametrize("kind", ["dent", "dmi", "dcmi"])
def test_discrete_estimators_and_warnings(oracle, kind):
    """The device group-by against the oracle's counts on data with many
    levels, -0 / +0 and wide values; the reference's too-many-levels
    warnings, counted from the device's distinct-value figures."""
    import warnings
    rng = np.random.default_rng(61)
    n = 30000
    x = rng.integers(-500, 500, size=n).astype(np.float64) * 1e9
    x[::7] = -0.0
    x[3::7] = 0.0
    y = rng.integers(0, 3, size=n).astype(np.float64)
    z = rng.integers(0, 40, size=(n, 2)).astype(np.float64)
    if kind == "dent":
        task, (v_ref, arrs) = E.discrete_entropy_task(np.column_stack((x, y))), \
            oracle.discrete_entropy(np.column_stack((x, y)))
        slots, expect_warn = ["c"], 0
    elif kind == "dmi":
        task, (v_ref, arrs) = E.discrete_mi_task(x, y), oracle.discrete_mi(x, y)
        slots = ["cxy", "cx", "cy"]
        expect_warn = int(arrs["groups"][1] > n / 4) + int(arrs["groups"][2] > n / 4)
    else:
        task, (v_ref, arrs) = E.discrete_cmi_task(x, y, z), oracle.conditional_discrete_mi(x, y, z)
        slots = ["cxyz", "cxz", "cyz", "cz"]
        expect_warn = int(arrs["groups"][4] + arrs["groups"][5])
    groups = {}
    v = N.run_tasks([task], flags=N.KEEP_INTERNALS, groups_out=groups)[0]
    for s, name in enumerate(slots):
        assert np.array_equal(N.fetch(0, 1 + s, n), arrs[name]), name
    assert abs(v - v_ref) <= 1e-10, (v, v_ref)
    with warnings.catch_warnings(record=True) as w:
        warnings.simplefilter("always")
        E.discrete_warnings(task, groups[0])
    assert len(w) == expect_warn
    assert list(groups[0][:len(slots)]) == [int(g) for g in arrs["groups"][:len(slots)]]
