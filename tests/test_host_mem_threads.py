"""Host pages brought in: the helper threads are shared by all callers, none stays, and a process that cannot make
threads still gets its pages.  Each case in a process of its own, whose threads are counted."""
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

HEAD = """
import ctypes as C, mmap, os, resource, sys, threading, time
sys.path.insert(0, %r)
from miniisosurface_gb300 import _lib
lib = C.CDLL(%r)
def threads():
    return len(os.listdir("/proc/self/task"))
def settled(n):  # a joined thread's entry may outlive the join by a moment
    end = time.time() + 5
    while threads() > n and time.time() < end: time.sleep(0.01)
    return threads() <= n
def fresh(mb):  # an anonymous mapping without pages
    m = mmap.mmap(-1, mb << 20, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    return m, C.addressof(C.c_char.from_buffer(m))
def resident():
    return int(open("/proc/self/statm").read().split()[1]) * mmap.PAGESIZE
def populate(at, mb):
    return lib.iso_populate_host(C.c_int64(1), (C.c_void_p * 1)(at), (C.c_int64 * 1)(mb << 20))
"""


def run(built, body):
    code = HEAD % (str(ROOT), str(built)) + body
    res = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout + res.stderr


def test_no_thread_stays(built):
    run(built, """
m, at = fresh(64)
before, rss = threads(), resident()
assert populate(at, 64) == 0
assert settled(before), (before, threads())
assert resident() - rss >= 60 << 20
""")


def test_callers_share_the_helpers(built):
    """8 callers at once: their own threads, and together three helpers at most (as many again may be on their way
    out)."""
    callers = 8
    run(built, """
callers = %d
maps = [fresh(128) for _ in range(callers)]
before, most, bad = threads(), 0, []
def call(at):
    if populate(at, 128) != 0: bad.append(at)
ts = [threading.Thread(target=call, args=(at,)) for _, at in maps]
for t in ts: t.start()
while any(t.is_alive() for t in ts): most = max(most, threads())
for t in ts: t.join()
assert not bad
assert most <= before + callers + 2 * 3, (before, most)
assert settled(before), (before, threads())
""" % callers)


def test_no_threads_to_be_had(built):
    """No address space for another thread's stack: the caller does it alone."""
    run(built, """
m, at = fresh(64)
rss = resident()
now = int(open("/proc/self/statm").read().split()[0]) * mmap.PAGESIZE
resource.setrlimit(resource.RLIMIT_AS, (now + (2 << 20), resource.RLIM_INFINITY))
assert populate(at, 64) == 0
assert resident() - rss >= 60 << 20
""")


def test_present_pages_cost_no_thread(built):
    """Memory that has its pages already (an array from memory the allocator kept): no helper is made.  Thread ids
    count up, so that helpers between two threads' ids show; other processes may take some now and then."""
    run(built, """
def id_now():
    t = threading.Thread(target=lambda: None)
    t.start(); t.join()
    return t.native_id
def between(at):
    a = id_now()
    assert populate(at, 64) == 0
    return id_now() - a
m, at = fresh(64)
assert between(at) > 1  # without pages: helpers
assert min(between(at) for _ in range(20)) == 1
""")
