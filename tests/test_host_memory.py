"""Device memory as the library's host side holds it: mms_api.cu on a CUDA
runtime in host memory (tests/host_runtime), which counts the memory held,
refuses what does not fit and notes every use of memory already given back."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "mumatscale_b200" / "csrc"

PRELUDE = """
import ctypes as C
import numpy as np
import mumatscale_b200 as M
lib = M.load_library()
lib.host_runtime_held.restype = C.c_size_t
lib.host_runtime_limit.argtypes = lib.host_runtime_total.argtypes = [C.c_size_t]
lib.host_runtime_stale.restype = lib.host_runtime_graph_launches.restype = C.c_longlong
held, limit, stale = lib.host_runtime_held, lib.host_runtime_limit, lib.host_runtime_stale
ALL = 1 << 40
p = M.read_deck(DECK)
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    """Runs a script on the library built with that runtime."""
    lib = tmp_path_factory.mktemp("host_runtime") / "libmms_host.so"
    sources = [CSRC / f for f in ("mms_api.cu", "host_setup.cpp", "deck.cpp", "output.cpp")]
    sources.append(ROOT / "tests" / "host_runtime" / "host_runtime.cpp")
    subprocess.run(["g++", "-x", "c++", "-std=c++17", "-O1", "-fPIC", "-shared", "-w", "-I/usr/local/cuda/include",
                    f"-I{CSRC}", "-o", str(lib), *map(str, sources), "-lz", "-ldl", "-lpthread", "-Wl,--no-undefined"],
                   check=True)
    deck = ROOT / "tests" / "golden" / "decks" / "small4.in"

    def go(script: str) -> str:
        r = subprocess.run([sys.executable, "-c", f"from pathlib import Path\nDECK = Path({str(deck)!r})" + PRELUDE + script],
                           cwd=ROOT, env=dict(os.environ, MMS_LIBRARY=str(lib)), capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return go


@pytest.mark.parametrize("spare", [0, 1, 2, 3])
def test_batch_after_a_rebuild_without_memory(run, spare):
    """A tile whose buffers do not fit: the batch steps no more until they do,
    and never with those it gave back (spare: the buffers that still fit)."""
    run(f"""
with M.Batch([p, p]) as b:
    b.step(3)
    before = held()
    # what a rebuild gives back: measured by one that fails at once
    limit(0)
    try:
        b.set_stencil_tile(2, 1)
        raise SystemExit("no failure")
    except M.MmsError as e:
        assert e.status == 11, e
    freed = before - held()
    assert freed > 0
    limit(held() + {spare} * freed // 4)
    try:
        b.step(2)
        done = 2
    except M.MmsError as e:
        assert e.status == 11, e
        done = 0
    assert [d.timestep for d in b.domains] == [3 + done] * 2
    limit(ALL)
    b.step(4)
    assert [d.timestep for d in b.domains] == [7 + done] * 2
    assert b.stencil_tile()[:2] == (2, 1)
assert stale() == 0, stale()
""")


RECORD = """
d = M.Domain(p)
d.step(4)
target = d.download("ce")
def record(steps, every):
    d.adjoint_record(steps, every)
    return held()
def tight(fn, *args):
    try:
        fn(*args)
    except M.MmsError as e:
        assert e.status == 11, e
        return True
"""


def test_a_second_domain_fits_after_a_gradient(run):
    """What fitted beside a record before its gradient fits after it."""
    run(RECORD + """
before = record(20, 10)
g = d.adjoint_gradient(target)
kept = held() - before
assert kept > 0
for make in (lambda: M.Domain(p), lambda: M.Batch([p])):
    with make():  # its own size, measured with room to spare
        size = held() - before - kept
    d.adjoint_gradient(target)
    assert held() == before + kept
    limit(before + size)
    with make():
        pass
    limit(ALL)
    assert held() == before  # the buffers went
    assert d.adjoint_gradient(target) == g
    assert d.adjoint_replay_loss(target) == g["loss"]
    assert held() == before + kept
d.adjoint_release()
d.close()
assert held() == 0 and stale() == 0
""")


def test_large_work_buffers_go_with_the_call(run):
    run(RECORD + """
state = 3 * 8 * d.num_cells()
before = record(3, (5 << 30) // state)  # states of 5 GiB
d.adjoint_gradient(target)
assert held() == before
d.adjoint_replay_loss(target)  # two states
assert 0 < held() - before < 1 << 30
assert stale() == 0
""")


def test_a_gradient_without_memory(run):
    """It fails with the status it always had, holds nothing, and both the
    record and the domain go on."""
    run(RECORD + """
before = record(20, 10)
limit(before + 1000)
assert tight(d.adjoint_gradient, target)
assert tight(d.adjoint_replay_loss, target)
assert held() == before
d.step(3)
limit(ALL)
assert d.adjoint_gradient(target)["steps"] == 20
d.adjoint_record(5, 5)
assert d.adjoint_gradient(target)["steps"] == 5
assert stale() == 0
""")


def test_buffers_are_given_back_between_threads(run):
    """One thread differentiates while another makes domains that fit only
    beside idle buffers that are given back."""
    run(RECORD + """
import threading
before = record(20, 10)
d.adjoint_gradient(target)
kept = held() - before
with M.Domain(p):
    size = held() - before - kept
limit(before + kept // 2 + size)
stop, made = threading.Event(), 0
def differentiate():
    while not stop.is_set():
        tight(d.adjoint_gradient, target)
t = threading.Thread(target=differentiate)
t.start()
for _ in range(40):
    if not tight(lambda: M.Domain(p).close()):
        made += 1
stop.set()
t.join()
limit(ALL)
assert d.adjoint_gradient(target)["steps"] == 20
d.close()
assert stale() == 0 and held() == 0
""")


def test_the_grid_a_batch_reports(run):
    """The CTAs of the stencil's launch: one per tile of every domain."""
    run("""
with M.Batch([p, p]) as b, M.Domain(p) as d:
    for tile in ((1, 0), (2, 3), (1, 1)):
        b.set_stencil_tile(*tile)
        nx, ny, nz = p.grid
        planes = tile[1] or 4  # (the stand-in's own choice)
        tiles = -(-nx // (32 * tile[0])) * -(-ny // 8) * -(-nz // planes)
        assert b.stencil_tile() == (*tile, 2 * tiles), (b.stencil_tile(), tiles)
""")
