"""GPU: side-information refinement searches per 16x16 tile; tiles with one, a
few or no Wyner-Ziv blocks, at the frame's corners and edges, against the
oracle's decode of the same frame (exactly), for both thread counts of a tile."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(kind, hb, wb):
    """8x8 blocks that stay Wyner-Ziv coded."""
    wz = np.zeros((hb, wb), bool)
    if kind.startswith("block "):  # the motion learning's smallest launches, windows of 25 to 81 candidates
        for b in kind.split()[1:]:
            wz.reshape(-1)[int(b)] = True
    elif kind == "corners":
        wz[0, 0] = wz[0, -1] = wz[-1, 0] = wz[-1, -1] = True
    elif kind == "one per tile":
        wz[::2, 1::2] = True
    elif kind == "scattered":
        wz = np.random.default_rng(4).random((hb, wb)) < 0.15
    return wz


@pytest.mark.parametrize("threads", ["256", "512"])
@pytest.mark.parametrize("kind", ["corners", "one per tile", "scattered"])
def test_sparse_tiles_match_the_oracle(kind, threads, monkeypatch):
    _compare(kind, threads, monkeypatch)


@pytest.mark.parametrize("kind", ["block 0", "block 395", "block 21 22 200"])
def test_a_few_blocks_match_the_oracle(kind, monkeypatch):
    _compare(kind, "256", monkeypatch)


def _compare(kind, threads, monkeypatch):
    from dvc_b200 import bitstream as bs, decoder, encoder, native, synth
    from oracle import pyoracle as po
    monkeypatch.setenv("DVC_SI_THREADS", threads)
    ori, key = synth.make_sequence("qcif", 3, 21)
    st = bs.parse_wz(encoder.encode_sequence(ori, 2, 2))
    fr = st.frames[1]
    h, w = ori[1].shape
    other = ~_map(kind, h // 8, w // 8)
    fr.ac_range, fr.crc, fr.acc_synd = encoder.encode_wz_frame(ori[1], 2, other88=other)
    fr.mode = np.where(other, bs.INTRA_B, bs.WZ_B).astype(np.uint8).reshape(-1)
    fr.intra_mode = 1
    start = np.array(key, np.uint8)
    start[1] = ori[1]  # intra pixels
    ctx = native.Context(0)
    try:
        out = ctx.debug_wz_frame(decoder.frame_item(st, fr, start))
    finally:
        ctx.close()
    ref = po.decode_frame(st, fr, key[0], key[2], recon_init=start[1], want=("si",))
    assert np.array_equal(out["recon"], ref["recon"])
    assert np.array_equal(out["planes"][:, 2], ref["accepted"])
    assert np.array_equal(out["si_final"].reshape(-1), np.asarray(ref["si_final"]).reshape(-1))
