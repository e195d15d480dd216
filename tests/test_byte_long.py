"""Long pairs outside the DNA class (an N in every sequence2, or a substitution matrix) run on whole
blocks, teams of 4 warps and clusters of blocks: each of them, the lead list that the router hands to
the blocks, every end-gap rule, and their waits when they give up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
MODES = [dict(), dict(local=True), dict(last_row_free=True, last_column_free=True),
         dict(first_column_free=True, last_column_free=True), dict(first_row_free=True, last_row_free=True)]
SHAPES = [(1, 1), (9, 2), (31, 33), (64, 64), (100, 513), (513, 100), (200, 512), (700, 650), (1025, 1030), (400, 1500),
          (3, 2100), (2100, 3), (150, 4700)]
# thresholds: long from (cells), teams up to (rows), clusters from (cells, rows)
ROUTES = {"blocks": (1, 0, 1 << 60, 1), "teams": (1, 1 << 30, 1 << 60, 1), "clusters": (1, 0, 1, 1)}


@pytest.fixture(scope="module")
def pa(built_lib):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    return pa


def _batch(pa, seed, shapes):
    rng = np.random.default_rng(seed)
    s1, s2 = [], []
    for m, n in shapes:
        a = ACGT[rng.integers(0, 4, m)]
        b = np.where(rng.random(n) < 0.85, np.resize(a, n), ACGT[rng.integers(0, 4, n)])
        b[rng.integers(0, n)] = ord("N")
        s1.append(bytes(a))
        s2.append(bytes(b.astype(np.uint8)))
    return (*pa.pack(s1), *pa.pack(s2))


def _context(pa, route):
    cells, rows, huge, min_rows = ROUTES[route]
    ctx = pa.Context(0)
    ctx.set_cta_threshold(cells)
    ctx.set_team_threshold(rows)
    ctx.set_cluster_threshold(huge, min_rows)
    return ctx


def _conf(kw, matrix):
    local = bool(kw.get("local"))
    c = dict(local=local, match=2, mismatch=-3, gap_open=-5, gap_extension=-1, first_column_free=local,
             first_row_free=local, last_column_free=local, last_row_free=local)
    c.update(kw)
    if matrix:
        sc = np.full((5, 5), -3)
        np.fill_diagonal(sc, 2)
        c["matrix"] = (b"ACGTN", [int(x) for x in sc.ravel()])
    return c


def _check(oracle, c, batch, res):
    oc = oracle.make_cfg(2, -3, -5, -1, local=c["local"], matrix=c.get("matrix"),
                         **{k: c[k] for k in ("first_column_free", "first_row_free", "last_column_free", "last_row_free")})
    sc, e1, e2 = oracle.align_batch(oc, *batch)
    bad = np.flatnonzero((res["score"] != sc) | (res["end1"] != e1) | (res["end2"] != e2))
    assert len(bad) == 0, (len(bad), bad[:5], res[bad[:5]], list(zip(sc[bad[:5]], e1[bad[:5]], e2[bad[:5]])))


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("kw", MODES, ids=["global", "local", "free_end", "free_column", "free_row"])
@pytest.mark.parametrize("matrix", [False, True], ids=["bytes", "matrix"])
def test_routes_equal_oracle(pa, oracle, route, kw, matrix):
    batch = _batch(pa, 3, SHAPES * 3)
    c, ctx = _conf(kw, matrix), _context(pa, route)
    al = pa.Aligner(c, context=ctx)
    res = al.compute_arrays(*batch)
    _check(oracle, c, batch, res)
    assert al.last_stats["pairs_general"] == len(res)
    ctx.close()


@pytest.mark.parametrize("kw", MODES[:3], ids=["global", "local", "free_end"])
def test_lead_list_of_the_blocks(pa, oracle, kw):
    """More largest pairs than two waves of clusters (at most 152 SMs x 8 blocks / 4 = 304 clusters): the
    blocks take them first, then their own list."""
    batch = _batch(pa, 4, [(int(m), 300 + int(m) % 400) for m in range(20, 120)] * 7 + [(300, 40)] * 20)
    ctx = _context(pa, "clusters")
    ctx.set_cluster_threshold(1, 200)                  # 700 pairs of the largest class, 20 of the blocks' own
    c = _conf(kw, False)
    _check(oracle, c, batch, pa.Aligner(c, context=ctx).compute_arrays(*batch))
    ctx.close()


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("local", [False, True])
def test_waits_that_give_up_are_reported(pa, oracle, route, local):
    """No polls allowed, pairs of four passes: PA_ERR_TIMEOUT, then the context aligns the batch exactly."""
    batch = _batch(pa, 5, [(400, 1800 + k) for k in range(16)])
    c, ctx = _conf(dict(local=True) if local else {}, False), _context(pa, route)
    al = pa.Aligner(c, context=ctx)
    ctx.set_wait_limit(0)
    out = np.zeros(16, pa.RESULT_DTYPE)
    with pytest.raises(pa.PaError) as e:
        al.compute_arrays(*batch, out=out)
    assert e.value.status == 6
    flagged = (out["flags"] & 0x20) != 0
    assert flagged.any() and (out["score"][flagged] == np.iinfo(np.int32).min).all()
    ctx.set_wait_limit(1 << 24)
    _check(oracle, c, batch, al.compute_arrays(*batch))
    ctx.close()
