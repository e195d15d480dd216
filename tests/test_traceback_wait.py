"""Traceback when the waits between a pair's passes give up (no polls allowed): the call is computed
again without waits and returns the oracle's paths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("local", [False, True])
@pytest.mark.parametrize("kind", ["dna", "bytes", "matrix"])
def test_waits_that_give_up_cost_no_result(built_lib, oracle, local, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    rng = np.random.default_rng(5)
    alphabet = np.frombuffer(b"ACGT" if kind == "dna" else b"ACGTN", np.uint8)
    pairs = []
    for n in (1, 300, 513, 1024, 1500, 2300, 0, 700) * 3:        # one to five passes of 512 rows
        b = alphabet[rng.integers(0, len(alphabet), n)]
        a = np.where(rng.random(n) < 0.9, b, alphabet[rng.integers(0, len(alphabet), n)])
        pairs.append((bytes(np.delete(a, slice(n // 3, n // 3 + 7))), bytes(b)))
    c = dict(local=local, match=2, mismatch=-3, gap_open=-5, gap_extension=-1, first_column_free=local,
             first_row_free=local, last_column_free=local, last_row_free=local)
    if kind == "matrix":
        sc = np.full((5, 5), -3)
        np.fill_diagonal(sc, 2)
        c["matrix"] = (bytes(alphabet), [int(x) for x in sc.ravel()])
    oc = oracle.make_cfg(2, -3, -5, -1, local=local, matrix=c.get("matrix"))
    ctx = pa.Context(0)
    al = pa.Aligner(c, context=ctx)
    launches = []
    for limit in (0, 1 << 24):
        ctx.set_wait_limit(limit)
        for x, (a, b) in zip(al.compute_traceback(*zip(*pairs)), pairs):
            want = oracle.traceback(oc, a, b)
            assert (x.score(), *x.begin_position(), *x.end_position(), x.ops()) == want, (limit, len(a), len(b))
            assert not x.flags() & 0x20
        launches.append(al.last_stats["kernel_launches"])
    assert launches == [4, 3]                                    # the second kernel ran, then was not needed
    ctx.close()
