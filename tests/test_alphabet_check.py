"""The check of sequence2's alphabet that picks a pair's kernel: one byte outside A/C/G/T, at every
position of short sequences at every alignment, is found, and the same byte in a neighbour, in
front of the buffer or behind it is not.  A pair with such a byte is scored in 32-bit lanes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAD = [ord(x) for x in "NacgtU@B"] + [0x00, 0x80, 0xC1, 0xD4, 0xFF]


@pytest.mark.parametrize("base", [0, 1, 7, 15])
@pytest.mark.parametrize("n", [1, 3, 15, 16, 17, 33, 515])
def test_one_bad_byte(built_lib, oracle, base, n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    rng = np.random.default_rng(n)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    where = np.arange(n) if n < 64 else np.r_[0:20, 250:262, n - 20:n]
    s1, s2, plain = [], [], []
    for k, at in enumerate(where):
        # 0 to 2 symbols of clean pairs between the marked ones move the alignment along
        for length, bad in ((n, True), (1 + k % 3, False)):
            b = acgt[rng.integers(0, 4, length)]
            if bad:
                b[at] = BAD[k % len(BAD)]
            s1.append(bytes(acgt[rng.integers(0, 4, 9)]))
            s2.append(bytes(b))
            plain.append(not bad)
    (a, o1), (b, o2) = pa.pack(s1), pa.pack(s2)
    # on the device at an odd address, between bytes that are no bases
    dev = torch.full((base + b.size + 32,), ord("N"), dtype=torch.uint8, device="cuda:0")
    dev[base:base + b.size] = torch.from_numpy(b.copy()).cuda()
    t1, u1, u2 = (torch.from_numpy(x.view(np.int64) if x.dtype == np.uint64 else x.copy()).cuda() for x in (a, o1, o2))
    cfg = dict(local=True, match=4, mismatch=-5, gap_open=-10, gap_extension=-1, first_column_free=True,
               first_row_free=True, last_column_free=True, last_row_free=True)
    al = pa.Aligner(cfg, context=pa.Context(0))
    out = torch.empty(len(s1) * pa.RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda:0")
    al.compute_device(t1, u1, dev[base:base + b.size], u2, out, stats=True)
    res = out.cpu().numpy().view(pa.RESULT_DTYPE)
    oc = oracle.make_cfg(4, -5, -10, -1, local=True, first_column_free=True, first_row_free=True,
                         last_column_free=True, last_row_free=True)
    for got, want in zip((res["score"], res["end1"], res["end2"]), oracle.align_batch(oc, a, o1, b, o2)):
        assert np.array_equal(got, want)
    assert np.array_equal(res["width"] == 16, np.array(plain))
