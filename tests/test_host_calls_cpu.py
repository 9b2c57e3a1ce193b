"""What the engine's host code asks of the CUDA runtime, seen by a runtime without
a device (fake_cudart/fake_cudart.cc, preloaded into a child process)."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def calls(td, tmp_path_factory):
    """Runs Python code in a child with the fake runtime; returns the log's lines."""
    from td16_b200 import build
    work = tmp_path_factory.mktemp("fake")
    fake = str(work / "libfake_cudart.so")
    include = os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc") or build.nvcc())), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", include, "-o", fake,
                    os.path.join(HERE, "fake_cudart", "fake_cudart.cc")], check=True)

    def run(code):
        log = str(work / "log")
        if os.path.exists(log):
            os.remove(log)
        env = dict(os.environ, LD_PRELOAD=fake, FAKE_CUDART_LOG=log, PYTHONPATH=ROOT)
        subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=120)
        with open(log) as f:
            return f.read().splitlines()

    return run


INIT = "import td16_b200 as td; td.init_slots(1, [0], 64 << 20)\n"
NOALLOC = """
import ctypes as C
from td16_b200 import _lib
err = C.create_string_buffer(256)
buf = (C.c_uint8 * 64)()
rc = _lib.lib().td_search_batch_noalloc(C.c_int(1), buf, buf, C.c_uint(0), C.c_uint64(0), None, err, C.c_size_t(256))
assert rc == 0, err.value
"""


@pytest.mark.parametrize("code", [INIT, NOALLOC, INIT + NOALLOC, NOALLOC + INIT])
def test_tables_are_on_the_device_before_a_kernel_reads_them(calls, code):
    """The build of the endgame table reads the triple and pair tables on a stream
    that waits for no other: they are uploaded on that stream, or their upload has
    been waited for.  (An upload from pageable memory on the default stream may
    return before it has arrived.)"""
    arrived, pending, builds = set(), {}, 0
    for line in calls(code):
        what, *rest = line.split()
        if what == "upload":
            pending[rest[0]] = rest[2]
            arrived.discard(rest[0])
        elif what == "synchronize":
            arrived |= {t for t, st in pending.items() if st == rest[1]}
            pending = {t: st for t, st in pending.items() if st != rest[1]}
        elif what == "launch" and "td_" in rest[0]:
            builds += "td_eg_build" in rest[0]
            for table in ("td_tri_table", "td_pair_table"):
                assert table in arrived or pending.get(table) == rest[2], (line, table)
    assert builds == 5  # one pass per number of missing moves, once per device


def test_pairs_pin_host_memory_once(calls):
    """Groups of pairs that grow from call to call: one pinned block of bounded
    size per slot, pinned by the first call."""
    lines = calls(INIT + """
import numpy as np
for slot_calls in range(2):
    for count in (1, 10, 11, 1000, 70000, 200003):
        pair = np.tile(np.arange(17, dtype=np.uint8), (count, 1))
        td._lib.search_pairs(0, pair, pair, 17, 1, 0.0, 9, 1)
td.init_slots(2, [0], 64 << 20)
td._lib.search_pairs(1, pair, pair, 17, 1, 0.0, 9, 1)
""")
    prepared = [i for i, line in enumerate(lines) if "td_pairs_prepare" in line]
    assert len(prepared) == 13
    pinned = [int(line.split()[1]) for line in lines[: prepared[11]] if line.startswith("hostalloc")]
    assert sum(pinned) <= 5 << 20
    assert not [line for line in lines[prepared[0]: prepared[11]] if line.startswith("host")]


def test_pairs_do_not_sleep_on_a_blocking_event(calls):
    """The outputs come back through pinned memory, so their copy does not end the
    wait by itself; a thread that sleeps until then wakes late."""
    lines = calls(INIT + """
import numpy as np
pair = np.tile(np.arange(17, dtype=np.uint8), (16, 1))
td._lib.search_pairs(0, pair, pair, 17, 1, 0.0, 9, 1)
""")
    lines = lines[[i for i, line in enumerate(lines) if "td_pairs_prepare" in line][0]:]
    lines = lines[[i for i, line in enumerate(lines) if "td_pairs_unpack" in line][0]:]
    assert "wait event blocking" not in lines
    assert lines[1].startswith(("synchronize stream", "wait event spinning"))


@pytest.mark.parametrize("flags", [0, 1])
def test_captured_launches_keep_their_buffers(calls, flags):
    """Batches that outgrow what a captured launch was given: its buffers are freed
    with the slot and not before, and what is kept for it is bounded by what the
    slot holds anyway."""
    lines = calls(INIT + f"""
import ctypes as C
buf = (C.c_uint8 * (1 << 20))()
at = C.addressof(buf)
g = td._lib.BatchGraph(0, 10, at, at, {flags})
for count in range(20, 2000, 20):
    td._lib.search_batch_device(0, count, at, at, {flags})
    td._lib.configure_split(64, (1 << 20) + count)
    td._lib.configure_table(6 + count % 7)
g.launch()
g.close()
import os
open(os.environ["FAKE_CUDART_LOG"], "a").write("destroy\\n")
td.destroy()
""")
    start, end = lines.index("capture"), lines.index("destroy")
    live, freed_early = {}, []
    for i, line in enumerate(lines):
        what, *rest = line.split()
        if what == "mallocasync":
            live[rest[0]] = int(rest[1])
        elif what == "free" and rest[0] in live:
            if start < i < end:
                freed_early.append(rest[0])
            del live[rest[0]]
        if i == end:
            held = sum(live.values())
    assert not freed_early
    assert not live  # the slot gives everything back
    assert held <= (420 << 20)
