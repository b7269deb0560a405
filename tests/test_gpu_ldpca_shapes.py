"""GPU: the launch shapes dvc_ldpca_decode and dvc_LdpcaDecoder choose by the
number of codewords (speculative slots, clusters of 2, 4 and 8 blocks, one block
per ladder) against the batched form, which walks the same ladders from a work
queue and is pinned to the reference codeword by codeword.  Everything is
compared exactly: bits, rates, first and accepted codes, the BP iterations of
the sequential ladder and the entropy bound's bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(ctx, n, lr, acc, crc, start=None):
    count = len(crc)
    dec, res, ent, work, ms = ctx.ldpca_decode_batch(np.full(count, n, np.int32), lr.reshape(-1), acc.reshape(-1), crc,
                                                     start)
    return dec.reshape(count, n), res, ent


# the largest count of each shape and the smallest of the next: clusters of 4, 2
# and 1 (QCIF), 8, 4, 2 and 1 (CIF) on 148 SMs, and one block per ladder past 592
@pytest.mark.parametrize("n,count", [(1584, c) for c in (1, 2, 3, 4, 5, 592, 593)] +
                         [(6336, c) for c in (1, 4, 5, 9, 10, 18, 19)])
def test_shapes_match_the_batched_form(gpu_ctx, n, count):
    from dvc_b200 import ldpca_bench as lb
    lr, acc, crc, x = lb.make_codewords(n, count, 40 + count)
    for _ in range(2):  # the scratch is left ready for the next call
        dec, res, ent = gpu_ctx.ldpca_decode(lr, acc, crc)
        want_dec, want_res, want_ent = _batch(gpu_ctx, n, lr, acc, crc)
        assert np.array_equal(ent.view(np.uint32), want_ent.view(np.uint32))
        assert np.array_equal(res, want_res)
        assert np.array_equal(dec, want_dec)


@pytest.mark.parametrize("n,codes", [(1584, range(0, 65)), (6336, (0, 1, 2, 31, 62, 63, 64))])
def test_every_first_code(gpu_ctx, n, codes):
    """A ladder entered at each code (the groups of rows of every code, partial
    ones too, and the full-rate code itself)."""
    from dvc_b200 import ldpca_bench as lb
    rates = lb.code_rates(n)
    lr, acc, crc, x = lb.make_codewords(n, 65, 7)
    for c in codes:
        want_dec, want_res, _ = _batch(gpu_ctx, n, lr[c:c + 1], acc[c:c + 1], crc[c:c + 1], np.array([c], np.int32))
        dec, rate, llr = gpu_ctx.LdpcaDecoder(lr[c], np.unpackbits(acc[c]), int(crc[c]), float(rates[c]))
        assert rate == want_res[0, 0], c
        assert np.array_equal(dec, want_dec[0]), c


def test_shapes_match_the_oracle(gpu_ctx):
    from dvc_b200 import ldpca_bench as lb
    from oracle import pyoracle as po
    for n, count in ((1584, 5), (6336, 1)):
        lr, acc, crc, x = lb.make_codewords(n, count, 91 + n)
        dec, res, ent = gpu_ctx.ldpca_decode(lr, acc, crc)
        for i in range(count):
            odec, orate, ostart, oacc, _ = po.ldpca_decode(po.OracleLadder.get(n), lr[i], np.unpackbits(acc[i]),
                                                           int(crc[i]), float(ent[i]))
            assert (res[i, 0], res[i, 1], res[i, 2]) == (orate, ostart, oacc)
            assert np.array_equal(dec[i], odec)


@pytest.mark.parametrize("n,per_sm,more", [(1584, 2, -1), (1584, 2, 0), (1584, 4, 1), (6336, 2, -1), (6336, 2, 0)])
def test_queue_from_two_codewords_per_sm(gpu_ctx, n, per_sm, more):
    """Either side of the count from which a call goes through the work queue,
    against the same codewords in calls of a few (slots), with a full-rate and an
    all-zero-information codeword among them and without the optional outputs."""
    import torch
    from dvc_b200 import ldpca_bench as lb
    count = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    lr, acc, crc, x = lb.make_codewords(n, count, 1000 + count)
    lr[0] = 1.0              # no information: the bound asks for the full rate
    crc[count - 1] ^= 0x5A   # no code's bits match: the ladder's end
    dec, res, ent = gpu_ctx.ldpca_decode(lr, acc, crc)
    for i in sorted({0, count // 2, count - 1} | set(range(0, count, 37))):
        d, r, e = gpu_ctx.ldpca_decode(lr[i:i + 1], acc[i:i + 1], crc[i:i + 1])
        assert np.array_equal(res[i], r[0]) and np.array_equal(dec[i], d[0])
        assert ent[i:i + 1].view(np.uint32)[0] == e.view(np.uint32)[0]
