"""GPU: ladder files of other codeword lengths than the codec's two (shorter than a
block's threads, as long, with and without a partial round of columns) and of
more codes than the shipped ones against the oracle, in the forms a call may
take: speculative slots, one block per ladder (the call that owns its memory, and
one with two codewords per SM, whose queue holds the codec's lengths only).
Bits, rates, codes and the bound's bits are compared exactly."""
import os
import shutil

import numpy as np
import pytest

import ladder_files as lf

pytestmark = pytest.mark.gpu


@pytest.fixture
def context(gpu_ctx, tmp_path, monkeypatch):
    """context(ladders): a context on its own ladder file (gpu_ctx has swept the tables)."""
    from dvc_b200 import native
    made = []

    def make(ladders):
        shutil.copy(os.path.join(native.TABLE_DIR, "xlm_tables.bin"), tmp_path)
        monkeypatch.setattr(native, "DATA_DIR", lf.data_dir(tmp_path / "data", ladders))
        made.append(native.Context(0, table_dir=str(tmp_path)))
        return made[-1]

    yield make
    for c in made:
        c.close()


def noalloc(ctx, lr, acc, crc):
    import torch
    count, n = lr.shape
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (lr, acc, crc)]
    dec = torch.zeros((count, n), dtype=torch.uint8, device="cuda")
    res = torch.zeros((count, 4), dtype=torch.int32, device="cuda")
    ent = torch.zeros(count, dtype=torch.float32, device="cuda")
    s = torch.cuda.current_stream()
    assert ctx.ldpca_decode_noalloc(n, count, *[t.data_ptr() for t in dev], dec.data_ptr(), res.data_ptr(),
                                    ent.data_ptr(), 50, s.cuda_stream) == 0, ctx.last_error()
    s.synchronize()
    return dec.cpu().numpy(), res.cpu().numpy(), ent.cpu().numpy()


@pytest.mark.parametrize("n", [256, 1024, 1504, 3168, 6304])
def test_other_lengths_match_the_oracle(context, n):
    from oracle import pyoracle as po
    L = lf.circulant(n, 32, range(4, 33, 4))
    ctx, o = context([L]), lf.oracle(L)
    lr, acc, crc, x = lf.codewords(L, 4, n)
    many = [np.repeat(a, 80, axis=0) for a in (lr, acc, crc)]
    got = [ctx.ldpca_decode(lr, acc, crc), noalloc(ctx, lr, acc, crc), [a[::80] for a in ctx.ldpca_decode(*many)]]
    for dec, res, ent in got:
        for i in range(4):
            odec, orate, ostart, oacc, _ = po.ldpca_decode(o, lr[i], np.unpackbits(acc[i]), int(crc[i]),
                                                           po.compute_ce(lr[i]))
            assert np.float32(po.compute_ce(lr[i])).view(np.uint32) == ent[i:i + 1].view(np.uint32)[0]
            assert (res[i, 0], res[i, 1], res[i, 2]) == (orate, ostart, oacc)
            assert np.array_equal(dec[i], odec)
        assert np.array_equal(res, got[0][1])


@pytest.mark.parametrize("num", [65, 66, 129])
def test_many_codes_match_the_oracle(context, num):
    from oracle import pyoracle as po
    from dvc_b200 import ldpca_bench as lb
    ladders = lf.many_codes(num)
    L = lf.lad.ladder_for(ladders, 1584)
    ctx, o = context(ladders), lf.oracle(L)
    lr, acc, crc, x = lb.make_codewords(1584, 4, 70 + num)
    crc[3] ^= 0x5A  # no code's bits match: every code is tried, up to the full rate
    lr[3] = np.where(lr[3] > 1, np.float32(20), np.float32(0.05))  # ... from one of the first
    many = [np.repeat(a, 80, axis=0) for a in (lr, acc, crc)]
    got = [ctx.ldpca_decode(lr, acc, crc), noalloc(ctx, lr, acc, crc), [a[::80] for a in ctx.ldpca_decode(*many)]]
    for i in range(4):
        odec, orate, ostart, oacc, _ = po.ldpca_decode(o, lr[i], np.unpackbits(acc[i]), int(crc[i]),
                                                       po.compute_ce(lr[i]))
        assert i < 3 or (oacc == num - 1 and num - 1 - ostart > (64 if num > 66 else 0))
        for dec, res, ent in got:
            assert (res[i, 0], res[i, 1], res[i, 2]) == (orate, ostart, oacc)
            assert np.array_equal(dec[i], odec) and np.array_equal(res[i], got[0][1][i])
        dec, rate, llr = ctx.LdpcaDecoder(lr[i], np.unpackbits(acc[i]), int(crc[i]), float(got[0][2][i]))
        assert rate == orate and np.array_equal(dec, odec)


@pytest.mark.parametrize("n", [256, 1584, 6336])
def test_rows_of_most_edges_match_the_oracle(context, n):
    """Codes whose rows differ in degree by a thousand times (their groups of rows
    are cut where the degree halves), in every form, entered at each code."""
    from oracle import pyoracle as po
    ladders = [lf.merged(m) for m in sorted({n, 1584, 6336})]
    L = lf.lad.ladder_for(ladders, n)
    ctx, o = context(ladders), lf.oracle(L)
    lr, acc, crc, x = lf.codewords(L, 4, 7 * n)
    # nearly every bit is sure, the others lean to the wrong side
    doubt = np.random.default_rng(n).random(lr.shape) < [[0.0], [0.004], [0.02], [0.06]]
    for_0 = np.where(doubt, np.float32(1 / 1.5), np.float32(3000))
    lr = np.where(x == 0, for_0, 1 / for_0).astype(np.float32)
    crc[3] ^= 0x5A
    many = [np.repeat(a, 80, axis=0) for a in (lr, acc, crc)]
    got = [ctx.ldpca_decode(lr, acc, crc), noalloc(ctx, lr, acc, crc), [a[::80] for a in ctx.ldpca_decode(*many)]]
    accepted = set()
    for i in range(4):
        for start in range(5):
            bound = np.float32(L["bpp"][start]) / np.float32(n)
            odec, orate, ostart, oacc, _ = po.ldpca_decode(o, lr[i], np.unpackbits(acc[i]), int(crc[i]), float(bound))
            dec, rate, llr = ctx.LdpcaDecoder(lr[i], np.unpackbits(acc[i]), int(crc[i]), float(bound))
            assert rate == orate and np.array_equal(dec, odec), (i, start)
            accepted.add(oacc)
        odec, orate, ostart, oacc, _ = po.ldpca_decode(o, lr[i], np.unpackbits(acc[i]), int(crc[i]),
                                                       po.compute_ce(lr[i]))
        for dec, res, ent in got:
            assert (res[i, 0], res[i, 1], res[i, 2]) == (orate, ostart, oacc)
            assert np.array_equal(dec[i], odec) and np.array_equal(res[i], got[0][1][i])
    assert len(accepted) >= 3, accepted  # codes with such rows decode, too
