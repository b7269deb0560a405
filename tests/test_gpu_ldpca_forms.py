"""GPU: the forms of the LDPCA kernel against one another on the same codewords
(bits, rates, codes, BP iterations and the bound's bits, all exactly)."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _batched(ctx, n, lr, acc, crc):
    dec, res, ent, _, _ = ctx.ldpca_decode_batch(np.full(len(crc), n, np.int32), lr.reshape(-1), acc.reshape(-1), crc)
    return dec.reshape(len(crc), n), res, ent


def _same(got, want):
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert np.array_equal(got[2].view(np.uint32), want[2].view(np.uint32))


@pytest.mark.parametrize("n", [1584, 6336])
@pytest.mark.parametrize("less", [1, 40])
def test_most_codewords_that_take_slots(gpu_ctx, n, less):
    """The largest counts below two codewords per SM, from which on calls go
    through the queue that the expected values come from."""
    import torch
    from dvc_b200 import ldpca_bench as lb
    count = 2 * torch.cuda.get_device_properties(0).multi_processor_count - less
    lr, acc, crc, x = lb.make_codewords(n, count, 300 + n + less)
    crc[::29] ^= 0x5A  # ladders that run to the full rate among them
    _same(gpu_ctx.ldpca_decode(lr, acc, crc), _batched(gpu_ctx, n, lr, acc, crc))


@pytest.mark.parametrize("threads", ["1024", "512", "256"])
@pytest.mark.parametrize("n,count", [(1584, 1), (1584, 149), (1584, 700), (6336, 1), (6336, 310)])
def test_block_per_ladder(gpu_ctx, n, count, threads, monkeypatch):
    """The form without scratch, which only the call on the caller's device memory
    takes whatever the count, in every launch shape (one, a full wave and more)."""
    import torch
    from dvc_b200 import ldpca_bench as lb, native
    lr, acc, crc, x = lb.make_codewords(n, count, 500 + n + count)
    crc[::29] ^= 0x5A
    want = _batched(gpu_ctx, n, lr, acc, crc)
    monkeypatch.setenv("DVC_LDPCA_THREADS", threads)
    monkeypatch.setenv("DVC_LDPCA_THREADS_QCIF", threads)
    ctx = native.Context(0)  # reads them
    try:
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (lr, acc, crc)]
        out = [torch.zeros((count, n), dtype=torch.uint8, device="cuda"),
               torch.zeros((count, 4), dtype=torch.int32, device="cuda"), torch.zeros(count, device="cuda")]
        s = torch.cuda.current_stream()
        assert ctx.ldpca_decode_noalloc(n, count, *[t.data_ptr() for t in dev + out], 50, s.cuda_stream) == 0
        s.synchronize()
        _same([t.cpu().numpy() for t in out], want)
    finally:
        ctx.close()
        monkeypatch.undo()
        native.Context(0).close()  # the default shapes again, for the process


@pytest.mark.parametrize("n,count", [(1584, 64), (6336, 24)])
def test_block_per_ladder_with_a_given_bound(gpu_ctx, n, count, tmp_path):
    """The bound given instead of summed: the ladder starts with no barrier but its
    own between the staged syndrome and the first code (tests/given_bound.cpp)."""
    from dvc_b200 import build, ldpca_bench as lb, native
    exe = str(tmp_path / "given_bound")
    cmd = ["g++", "-O1", "-std=c++17", "-w", "-I", "/usr/local/cuda/include", "-I", os.path.dirname(HERE) + "/include",
           "-I", build.CSRC, "-o", exe, os.path.join(HERE, "given_bound.cpp"), build.LIB,
           "-Wl,-rpath," + os.path.dirname(build.LIB), "-L/usr/local/cuda/lib64", "-lcudart_static", "-lpthread", "-ldl",
           "-lrt"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    lr, acc, crc, x = lb.make_codewords(n, count, 17 + n)
    crc[-1] ^= 0x5A  # no code's bits match: the ladder ends at the full rate
    for name, a in (("lr", lr), ("acc", acc), ("crc", crc)):
        np.ascontiguousarray(a).tofile(tmp_path / name)
    r = subprocess.run([exe, native.DATA_DIR, native.TABLE_DIR, str(n), str(count)] +
                       [str(tmp_path / f) for f in ("lr", "acc", "crc")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-1000:])
