"""The rank map of small alphabets (three distinguishing bits at any shift) and of alphabets just
past them, every byte value, aligned and unaligned, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALPHABETS = [b"A", b"ACGTN", b"acgtACGT", bytes(range(8)), bytes(range(8, 80, 8)[:8]), bytes(range(0, 256, 32)),
             b"\x00\xff", b"\x00\x01\x02\x03\x04\x05\x06\x87", b"AACCA", b"ACGTRYSW", b"ABCDEFGHI", b"01234567"]


@pytest.mark.parametrize("alphabet", ALPHABETS)
def test_rank_map_small_alphabets(built_lib, oracle, alphabet):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pairwise_aligner_gb300 as pa
    from pairwise_aligner_gb300 import seqio
    ctx = pa.Context(0)
    rng = np.random.default_rng(len(alphabet))
    data = np.concatenate([np.arange(256, dtype=np.uint8), rng.integers(0, 256, 70000, dtype=np.uint8)])
    want = oracle.rank_map(alphabet, data)
    dev = torch.from_numpy(data).cuda()
    for start, stop in ((0, len(data)), (1, len(data)), (16, 16 + 33), (0, 5)):
        out = torch.zeros(stop - start, dtype=torch.int8, device="cuda")
        bad = seqio.rank_map_device(ctx, alphabet, dev[start:stop], out, count_invalid=True)
        assert np.array_equal(out.cpu().numpy(), want[start:stop])
        assert bad == int((want[start:stop] < 0).sum())
    ctx.close()
