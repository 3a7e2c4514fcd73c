"""Host side of the launches without a GPU: the C ABI (csrc/c_api.cpp) and the
uneven-size launch (csrc/geneig_uneven_launch.cpp) over a fake CUDA runtime and fake launchers (tests/host/fake_cuda.cpp), which log every
record, wait and launch and can fail any of them."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]
CSRC = REPO / "sunny_gen_eigensolver_b200" / "csrc"
CUDA = Path("/usr/local/cuda/include")
U = ctypes.c_size_t


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or not (CUDA / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    out = tmp_path_factory.mktemp("host") / "libhost.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", f"-I{REPO / 'include'}", f"-I{CSRC}",
                    f"-I{CUDA}", str(CSRC / "c_api.cpp"),
                    str(CSRC / "geneig_uneven_launch.cpp"), str(REPO / "tests" / "host" / "fake_cuda.cpp"), "-ldl", "-o", str(out)],
                   check=True)
    L = ctypes.CDLL(str(out))
    for name in ("sunny_geneig_create_config", "sunny_geneig_uneven_create"):
        getattr(L, name).restype = ctypes.c_void_p
    L.sunny_geneig_create_config.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_char_p, ctypes.c_int]
    L.sunny_geneig_launch.argtypes = [ctypes.c_void_p, U, U, U, U, U, ctypes.c_int, U]
    L.sunny_geneig_destroy.argtypes = [ctypes.c_void_p]
    A = ctypes.POINTER(U)
    L.sunny_geneig_uneven_create.argtypes = [ctypes.c_int] + [ctypes.POINTER(ctypes.c_int)] * 3 + [ctypes.c_int]
    L.sunny_geneig_uneven_launch.argtypes = [ctypes.c_void_p, A, A, A, A, A, ctypes.POINTER(ctypes.c_int), U]
    L.sunny_geneig_uneven_destroy.argtypes = [ctypes.c_void_p]
    L.fake_reset.argtypes = [ctypes.c_char_p, U]
    L.fake_capture.argtypes = [U, ctypes.c_int]
    L.fake_log.restype = L.fake_dependencies.restype = ctypes.c_char_p
    L.fake_dependencies.argtypes = [U]
    return L


def reset(L, fail="", memory=1 << 40):
    L.fake_reset(fail.encode(), memory)


def log(L):
    return L.fake_log().decode().splitlines()


def launch(L, s, stream):
    return L.sunny_geneig_launch(s, 4096, 8192, 12288, 16384, 20480, 3, stream)


@pytest.mark.parametrize("n,mode,ordered", [(54, 0, False), (61, 0, True), (72, 0, True), (110, 0, True), (216, 0, True),
                                            (54, 2, True)])
def test_launches_of_an_l2_slot_handle_are_ordered_across_streams(lib, n, mode, ordered):
    s = lib.sunny_geneig_create_config(n, 0, mode, b"", 0)
    reset(lib)
    for stream in (11, 11, 12, 11):
        assert launch(lib, s, stream) == 0
    lines = log(lib)
    if not ordered:
        assert lines == [f"launch {n} on {x}" for x in (11, 11, 12, 11)]
    else:
        ev = lines[1].split()[1]
        assert lines == [f"launch {n} on 11", f"record {ev} on 11", f"launch {n} on 11", f"record {ev} on 11",
                         f"wait {ev} on 12", f"launch {n} on 12", f"record {ev} on 12",
                         f"wait {ev} on 11", f"launch {n} on 11", f"record {ev} on 11"]
        reset(lib)
        lib.fake_capture(12, 1)                      # replays are the caller's to order
        assert launch(lib, s, 12) == 0
        lib.fake_capture(12, 0)
        assert log(lib) == [f"launch {n} on 12"]
        reset(lib)
        lib.sunny_geneig_destroy(s)
        assert log(lib) == [f"sync_event {ev}"]
        return
    lib.sunny_geneig_destroy(s)


def test_launch_that_failed_is_still_waited_for(lib):
    """The mixed form's launch is two kernels: when the second fails the first is
    already using the handle's slots."""
    s = lib.sunny_geneig_create_config(54, 0, 2, b"", 0)
    reset(lib, fail="launch:0")
    assert launch(lib, s, 11) != 0
    assert launch(lib, s, 12) == 0
    lines = log(lib)
    ev = lines[1].split()[1]
    assert lines == ["launch 54 on 11 FAILS", f"record {ev} on 11", f"wait {ev} on 12", "launch 54 on 12", f"record {ev} on 12"]
    lib.sunny_geneig_destroy(s)


SIZES = [12, 54, 72, 108, 162, 216]


def uneven_create(L, sizes=SIZES):
    return L.sunny_geneig_uneven_create(len(sizes), (ctypes.c_int * len(sizes))(*sizes), None, None, 0)


def uneven_launch(L, h, stream, sizes=SIZES, counts=None):
    k = len(sizes)
    p = (U * k)(*[4096] * k)
    return L.sunny_geneig_uneven_launch(h, p, p, p, p, p, (ctypes.c_int * k)(*(counts or [5] * k)), stream)


def unjoined(lines, stream):
    """Work that `stream` does not wait for at the end of the log: kernels on other streams after the last
    record of an event that `stream` waits for later."""
    kernels = [(i, x.split(" on ")[1].split()[0]) for i, x in enumerate(lines)
               if x.split()[0] in ("cta", "tiled", "persistent") and not x.endswith("FAILS")]
    bad = []
    for i, st in kernels:
        if st == str(stream):
            continue
        joins = [j for j, x in enumerate(lines) if j > i and x.startswith("record") and x.endswith(f" on {st}")]
        waited = any(x == f"wait {lines[j].split()[1]} on {stream}" for j in joins for x in lines[j:])
        if not waited and not any(x == f"sync_stream {st}" for x in lines[i:]):
            bad.append(lines[i])
    return bad


FAILURES = [f"{c}:{k}" for c, n in (("cta", 2), ("tiled", 2), ("persistent", 1), ("wait", 9), ("record", 6)) for k in range(n)]


@pytest.mark.parametrize("fail", [""] + FAILURES)
def test_uneven_launch_joins_its_streams_whatever_fails(lib, fail):
    h = uneven_create(lib)
    reset(lib, fail=fail)
    st = uneven_launch(lib, h, 11)
    lines = log(lib)
    assert (st == 0) == (not any(x.endswith("FAILS") for x in lines))
    assert unjoined(lines, 11) == []
    if not fail:
        assert sum(x.startswith(("cta", "tiled", "persistent")) for x in lines) == 5
    if not fail.startswith("record") and any(x.split()[0] in ("cta", "tiled", "persistent") for x in lines):
        # the next call on another stream waits for this one
        reset(lib)
        assert uneven_launch(lib, h, 12) == 0
        assert log(lib)[0].startswith("wait") and log(lib)[0].endswith("on 12")
    lib.sunny_geneig_uneven_destroy(h)


def test_captured_uneven_launch_keeps_to_the_callers_stream(lib):
    """Each size is a branch of the graph from the point of the call, and what follows comes after all of them; the
    handle's streams and events stay out of the capture, so that its launches go on elsewhere while it lasts."""
    h = uneven_create(lib)
    reset(lib)
    lib.fake_capture(11, 1)
    root = lib.fake_dependencies(11).decode().split()
    assert uneven_launch(lib, h, 11) == 0
    kernels = [x.split() for x in log(lib) if x.split()[0] in ("cta", "tiled", "persistent")]
    assert len(kernels) == 5 and not any(x.startswith(("record", "wait")) for x in log(lib))
    # largest first, each from the point of the call and when the one before it has begun
    assert [k[1] for k in kernels] == ["216", "162", "108", "72", "on"]
    nodes = [k[k.index("node") + 1] for k in kernels]
    for i, k in enumerate(kernels):
        assert k[k.index("on") + 1] == "11" and k[k.index("after") + 1:] == root + [f"{x}-begun" for x in nodes[max(i - 1, 0):i]]
    nodes.sort()
    assert sorted(lib.fake_dependencies(11).decode().split()) == nodes
    assert uneven_launch(lib, h, 12) == 0                 # not captured
    lib.fake_capture(13, 1)                                # a second capture
    assert uneven_launch(lib, h, 13) == 0 and uneven_launch(lib, h, 12) == 0
    assert uneven_launch(lib, h, 11) == 0                 # the first one goes on
    again = [x.split() for x in log(lib) if " on 11 " in x and "node" in x][5:]
    assert len(again) == 5
    for k in again:
        assert sorted(x for x in k[k.index("after") + 1:] if not x.endswith("begun")) == nodes
    lib.fake_capture(11, 0)
    lib.fake_capture(13, 0)
    lib.sunny_geneig_uneven_destroy(h)


@pytest.mark.parametrize("fail", [f"{c}:{k}" for c, n in (("cta", 2), ("tiled", 2), ("persistent", 1), ("capture_info", 5),
                                                        ("set_dependencies", 4)) for k in range(n)])
def test_captured_uneven_launch_joins_its_branches_whatever_fails(lib, fail):
    h = uneven_create(lib)
    reset(lib, fail=fail)
    lib.fake_capture(11, 1)
    assert uneven_launch(lib, h, 11) != 0
    nodes = [x.split() for x in log(lib) if "node" in x and not x.endswith("FAILS")]
    left = lib.fake_dependencies(11).decode().split()
    assert all(k[k.index("node") + 1] in left for k in nodes)
    lib.fake_capture(11, 0)
    lib.sunny_geneig_uneven_destroy(h)


def test_branches_start_largest_first_without_priorities(lib):
    """Each side stream waits for the launch completion of the size before it, and no stream is put above the
    caller's (priority 0 is the lowest)."""
    reset(lib)
    h = uneven_create(lib)
    assert [x for x in log(lib) if x.startswith("stream")] and all(x.endswith("priority 0") for x in log(lib))
    reset(lib)
    assert uneven_launch(lib, h, 11) == 0
    lines = log(lib)
    fork = lines[0].split()[1]
    assert lines[0] == f"record {fork} on 11"
    before, i = fork, 1
    for n in (216, 162, 108, 72):
        st = lines[i].split()[3]
        assert lines[i] == f"wait {before} on {st}" and st != "11"
        before = lines[i + 1].split()[1]
        assert lines[i + 1] == f"starts {before} with {st}" and lines[i + 2].split()[:4] == [
            "cta" if n <= 110 else "tiled", str(n), "on", st]
        i += 3
    assert lines[i] == f"wait {before} on 11" and lines[i + 1] == "persistent on 11"
    lib.sunny_geneig_uneven_destroy(h)


def _slots(n):
    mat = n * (n | 1)
    return 148 * (1 if n > 200 else 2) * 16 * (3 * mat + max((mat + 1) // 2, 16 * n))


def test_uneven_handle_falls_back_to_one_slot_array(lib):
    """Each size above 110 has slots of its own where they fit; where they do not, the largest size's are enough and
    everything runs on the caller's stream."""
    lib.fake_memory_used.restype = U
    sizes = [442, 452, 462, 472, 482, 492, 502, 512]
    all_, one = sum(map(_slots, sizes)), max(map(_slots, sizes))
    reset(lib, memory=all_ + 4096)
    h = uneven_create(lib, sizes)
    assert h and lib.fake_memory_used() == all_ + 8
    lib.sunny_geneig_uneven_destroy(h)
    assert lib.fake_memory_used() == 0
    reset(lib, memory=one + 4096)
    h = uneven_create(lib, sizes)
    assert h and lib.fake_memory_used() == one + 8
    assert not any(x.startswith("stream") for x in log(lib))
    reset(lib)
    assert uneven_launch(lib, h, 11, sizes) == 0
    lines = log(lib)
    slots = lines[0].split()[-1]
    assert lines[:-1] == [f"tiled {n} on 11 slots {slots}" for n in reversed(sizes)] and lines[-1].startswith("record")
    reset(lib)
    lib.fake_capture(11, 1)
    assert uneven_launch(lib, h, 11, sizes) == 0
    kernels = [x.split() for x in log(lib)]
    for before, k in zip(kernels, kernels[1:]):          # a chain
        assert k[k.index("after") + 1:] == [before[before.index("node") + 1]]
    lib.fake_capture(11, 0)
    lib.sunny_geneig_uneven_destroy(h)
    assert lib.fake_memory_used() == 0
    reset(lib, memory=one - 1)
    assert not uneven_create(lib, sizes) and lib.fake_memory_used() == 0
