"""The library's host code on the CPU, linked with a CUDA runtime that runs no
kernel (tests/host_routes.cpp): which launches a call makes, what it does when
memory is refused, what it holds and gives back."""
import os
import shutil
import subprocess

import pytest

from ladder_files import circulant, data_dir, lad, many_codes, merged

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda"


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    """run(mode, *args) -> the lines the driver prints; its tables are cached for the module."""
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers not available")
    from dvc_b200 import build
    build.build()
    tmp = tmp_path_factory.mktemp("routes")
    objs = [os.path.join(build.OBJDIR, os.path.basename(s) + ".o") for s in build.sources()]
    objs = [o for o in objs if "libm_tables" not in o]  # the driver's own, which sweep nothing
    out = str(tmp / "host_routes")
    r = subprocess.run([gxx, "-O1", "-std=c++17", "-w", "-I", os.path.join(CUDA, "include"), "-I",
                        os.path.join(ROOT, "include"), "-I", build.CSRC, "-o", out,
                        os.path.join(ROOT, "tests", "host_routes.cpp")] + objs + ["-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]

    def run(mode, data, *args, env=None):
        r = subprocess.run([out, mode, str(data), str(tmp)] + [str(a) for a in args], capture_output=True, text=True,
                           timeout=300, env=dict(os.environ, **(env or {})))
        assert r.returncode == 0, (r.returncode, r.stdout[-1000:], r.stderr[-1000:])
        return r.stdout.splitlines()

    run.tmp = tmp
    return run


def launches(lines):
    return [x.split() for x in lines if x.startswith("launch ")]


def test_a_ladder_file_after_one_that_needs_less_memory(routes):
    """Codes of the same length take more or less shared memory by the degrees of
    their rows: a second context's launches must not be held to the first's."""
    shipped = lad.read_compact(os.path.join(ROOT, "dvc_b200", "ladders", "ldpca_ladders.bin"))
    few = [dict(L, bpp=L["bpp"][-2:], idx=L["idx"][-2:]) for L in shipped]  # the highest codes: rows of equal degree
    lines = routes("files", data_dir(routes.tmp / "few", few), data_dir(routes.tmp / "all", shipped))
    smem = [int(x[9]) for x in launches(lines) if "ladder_kernel" in x[1] or "ldpca_batch_kernel" in x[1]]
    assert len(smem) == 12 and any(b > a for a, b in zip(smem[:6], smem[6:])), lines
    assert [x for x in lines if x.startswith("rc")] == ["rc 0"] * 12, lines


@pytest.mark.parametrize("n,count", [(256, 1), (256, 3), (1024, 40)])
def test_other_codeword_lengths_reach_the_ladder(routes, n, count):
    """A ladder file may hold other lengths than the two of the codec's sizes:
    the cluster shapes, cut for those two, are not for them."""
    d = data_dir(routes.tmp / ("n%d" % n), [circulant(n, 32, range(4, 33, 4))])
    lines = routes("decode", d, n, count)
    assert "rc 0" in lines, lines
    ladder = [x for x in launches(lines) if "ldpca_ladder_kernel" in x[1]]
    assert len(ladder) == 1 and ladder[0][7] == "1", lines


@pytest.mark.parametrize("num,own_block", [(65, False), (66, True), (129, True)])
@pytest.mark.parametrize("count", [1, 40, 600])
def test_ladders_of_many_codes_take_a_block_each(routes, num, own_block, count):
    """The slots' iteration counts and the queue's masks hold 64 codes a codeword:
    a file with more keeps the form without either."""
    d = data_dir(routes.tmp / ("codes%d" % num), many_codes(num))
    lines = routes("decode", d, 1584, count)
    assert "rc 0" in lines, lines
    ladder = [x for x in launches(lines) if "ldpca_ladder_kernel" in x[1]]
    queue = [x for x in launches(lines) if "ldpca_batch_kernel" in x[1]]
    alone = [(int(x[3]), int(x[7])) for x in ladder] == [(count, 1)] and not queue
    assert alone == own_block and len(ladder) + len(queue) == 1, lines


@pytest.mark.parametrize("n,accepted", [(96, True), (100, False), (260, False)])
def test_lengths_that_are_no_whole_bytes_are_refused(routes, n, accepted):
    """Syndromes are stored eight bits to a byte, n / 8 bytes a codeword: with
    another length the last bits of one would be read past its end."""
    lines = routes("decode", data_dir(routes.tmp / ("n%d" % n), [circulant(n, 4, range(1, 5))]), n, 1)
    if accepted:
        assert "rc 0" in lines, lines
    else:
        assert lines[0] == "create -4 ladder edge count not a multiple of 8 or above 65535", lines


SHIPPED = os.path.join(ROOT, "dvc_b200", "ladders")


@pytest.mark.parametrize("n,count,size,after", [
    (1584, 1, 1 << 20, 0), (6336, 7, 1 << 20, 0), (6336, 295, 7500000, 0),  # no room for the slots
    (1584, 0, 1 << 20, 0), (6336, 0, 6336 * 4, 1)])                          # count 0: dvc_LdpcaDecoder
def test_calls_without_memory_for_slots_decode_a_block_each(routes, n, count, size, after):
    lines = routes("scarce", SHIPPED, n, count, size, after)
    assert [x for x in lines if x.startswith("rc")] == ["rc 0 last 0"] * 2, lines
    poor, rich = [(int(x[3]), int(x[7])) for x in launches(lines) if "ldpca_ladder_kernel" in x[1]]
    assert poor == (max(count, 1), 1) and rich[0] > poor[0], lines


@pytest.mark.parametrize("n,count", [(1584, 2**31 - 1), (6336, 2**22 + 1)])
def test_a_count_that_no_device_holds_is_refused(routes, n, count):
    """... with a status, and without host memory for so many codewords."""
    assert "rc -3" in routes("huge", SHIPPED, n, count)


@pytest.mark.parametrize("sequences,levels,max_batch,streams,own,side", [
    (64, 1, 4, 2, 2, 6), (40, 1, 8, 4, 4, 28), (9, 1, 16, 1, 1, 4), (33, 1, 16, 4, 3, 14), (66, 1, 33, 2, 2, 0),
    (6, 3, 16, 8, 4, 14),  # levels of 6, 12 and 16 + 8 frames: the first three batches follow one another
    (6, 3, 16, 2, 2, 14), (6, 3, 4, 16, 11, 3 * 6), (1, 3, 16, 8, 3, 3)])
def test_a_sessions_batches_share_their_streams(routes, sequences, levels, max_batch, streams, own, side):
    """A session makes no stream that no batch is on, and a batch's groups (up to
    eight) decode on the streams of one that it runs after where there is one."""
    lines = routes("session", SHIPPED, sequences, levels, max_batch, streams)
    assert [x for x in lines if x.startswith("rc")] == ["rc 0"] * 3, lines
    assert "streams %d" % (own + side) in lines, lines
    assert lines[-1] == "left bytes 0 streams 0 events 0"


@pytest.mark.parametrize("w,h", [(176, 144), (352, 288)])
@pytest.mark.parametrize("q", [1, 4, 8])
@pytest.mark.parametrize("range_,count", [(1, 1), (200, 1), (2000, 1), (200, 16)])
def test_the_server_charges_what_a_request_holds(routes, w, h, q, range_, count):
    """The budget is one on device memory: a request counts at least for the bytes
    that are allocated for it, and beyond them for no more than the widest
    speculation (32 slots of a codeword's bits), every step's job and 64 KB."""
    lines = routes("server", SHIPPED, w, h, q, range_, count)
    got = [x.split() for x in lines if x.startswith("in flight")][0]
    flight, charged, held = int(got[2]), int(got[4]), int(got[6])
    assert flight == count
    more = 32 * (w * h // 16 + 4) + 63 * 112 + 65536 + 1024
    assert held <= charged <= held + count * more, (charged, held)


def test_every_value_of_a_tuned_parameter_is_another_launch_shape(routes):
    """The autotuner times each value of a thread count once: two that launch the
    same kernels would be chosen between by noise, and the default setting is the
    one a process without the variables runs."""
    from dvc_b200 import autotune as at
    unset = dict.fromkeys(at.ENV_ALL, "")

    def shape(**env):
        return tuple(x for x in routes("shapes", SHIPPED, env=dict(unset, **env)) if x.startswith("launch"))

    plain = tuple(x for x in routes("shapes", SHIPPED) if x.startswith("launch"))
    for name, values in at.KNOBS:
        if name != at.ENV_FLOOR:
            got = [shape(**{name: v}) for v in values]
            assert len(set(got)) == len(values), name
            assert got[0] == plain, name


@pytest.mark.parametrize("which", ["shipped", "129 codes", "a row of most edges"])
def test_layout_of_every_code(routes, which):
    """... of rows of any degrees: a code keeps within twice its edges' positions
    (the shipped ones within a hundredth more than the edges), and a launch of any
    form holds it."""
    d = {"shipped": lambda: SHIPPED, "129 codes": lambda: data_dir(routes.tmp / "c129", many_codes(129)),
         "a row of most edges": lambda: data_dir(routes.tmp / "merged", [merged(n) for n in (256, 1600, 6336)])}[which]()
    seen = [x.split() for x in routes("layout", d) if x.startswith("length")]
    assert seen and all(x[-1] == "0" for x in seen), seen
    for x in seen:
        n, positions = int(x[1]), int(x[5])
        assert positions <= (2 if which[0] == "a" else 1.12) * 3 * n
        for count in (1, 100, 700):
            lines = routes("decode", d, n, count)
            assert "rc 0" in lines and not any("refused" in t for t in lines), lines
