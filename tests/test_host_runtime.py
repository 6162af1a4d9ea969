"""The library's host side - memory, streams, the order of its copies and launches - on a CUDA runtime
that only keeps a log (fake_cudart.cpp, preloaded into a child process).  No GPU."""
import os
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = "/usr/local/cuda/include"

PRELUDE = """
import ctypes as C, importlib, sys
import numpy as np
sys.path.insert(0, %r)
fake = C.CDLL(None)
fake.fake_log.restype = C.c_char_p
fake.fake_live.restype = C.c_long
fake.fake_set.argtypes = [C.c_char_p, C.c_long]
def log():
    return [line.split() for line in fake.fake_log().decode().splitlines()]
aero = importlib.import_module("3d_aero_lab_b200")
cfd = importlib.import_module("3d_aero_lab_b200.cfd")
L = importlib.import_module("3d_aero_lab_b200._lib")
lib = L.lib()
def box(NX, NY, NZ, device=0):
    "A solver over a box of fluid."
    N = NX * NY * NZ
    geo = cfd.Geom(N)
    geo.t[:], geo.phi[:] = 0, 1
    for d in range(4):
        geo.ap[d][:] = d < 3
    f = lambda n: np.arange(n + 1, dtype=np.float64)
    return aero.CfdGPU(cfd.Grid(f(NX), f(NY), f(NZ)), geo, device=device)
""" % ROOT


@pytest.fixture(scope="session")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", CUDA_INCLUDE, "-o", so,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp")], check=True)

    def run(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(code)], capture_output=True, text=True,
                           env=dict(os.environ, LD_PRELOAD=so, MALLOC_PERTURB_="165"), timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


@pytest.mark.parametrize("make", ["box(20, 6, 9)", "aero.Case(cells=3000).solver",
                                  "cfd.cfd_geom(aero.shape_of(aero.build_aircraft('fighter')), "
                                  "cfd.cfd_grid(aero.shape_of(aero.build_aircraft('fighter')), 3000), 0.0)"])
def test_uploads_go_down_the_stream_that_reads_them(fake, make):
    """A copy from pageable memory may return before it has reached the device, so it must be queued on
    the stream of the kernels that read it; on the default stream nothing orders it before them."""
    fake(f'''
    fake.fake_clear()
    x = {make}
    L = log()
    assert ["cudaMemcpy", "1"] not in L                      # no host-to-device copy on the default stream
    readers = {{l[1] for l in L if l[0] == "launch"}}
    up = [l for l in L if l[0] == "cudaMemcpyAsync" and l[2] == "1"]
    assert up and len(readers) == 1 and {{l[1] for l in up}} == readers
    ''')


@pytest.mark.parametrize("kernel", [2, 4])
def test_z_chunks_wait_for_every_chunk_that_they_read(fake, kernel):
    """Whatever the planes, the z run and the chunks asked for: every earlier stage's launch over a plane
    within two of a launch's own is ordered before it, by its stream or by the events it waits for."""
    fake(f"""
    for NZ in range(1, 14):
        s = box(6, 4, NZ)
        for kz in (0, 1, 2, 3):
            s.set_kernel({kernel}, kz)
            run = s.kernel()[1]
            for chunks in (2, 3, 4):
                s.set_chunks(chunks)
                K = s.chunks()
                assert 1 <= K <= chunks
                assert K == min(2, -(-NZ // run)) or K > 2 or run == 1, (NZ, run, chunks, K)
                fake.fake_clear()
                s.step(3)
                if K == 1:
                    continue
                done, events, stages = {{}}, {{}}, []      # launches that a stream, an event comes after
                for line in log():
                    if line[0] == "record":
                        events[line[1]] = set(done.setdefault(line[2], set()))
                    elif line[0] == "wait":
                        done.setdefault(line[1], set()).update(events[line[2]])
                    elif line[0] == "launch":
                        if not stages or len(stages[-1]) == K:
                            stages.append([])
                        first = stages[-1][-1][2] if stages[-1] else 0
                        me = (len(stages), first, min(NZ, first + int(line[2]) * run))
                        before = done.setdefault(line[1], set())
                        for earlier in stages[:-1]:
                            for e in earlier:
                                if e[1] < me[2] + 2 and e[2] > me[1] - 2:
                                    assert e in before, (NZ, run, K, me, e)
                        stages[-1].append(me)
                        before.add(me)
                assert len(stages) == 6 and all(x[-1][2] == NZ for x in stages)
    """)


def test_destruction_waits_for_its_own_streams_and_spoils_no_capture(fake):
    """A device-wide synchronisation is refused while another thread captures a stream of the device, and
    spoils that capture: destroying a solver, choosing its planes and tuning a batch make none.  The
    solver's streams are waited for before its memory goes back."""
    fake("""
    fake.fake_set(b"capturing", 1)
    a, b = box(6, 4, 9), box(6, 4, 9)
    a.set_kernel(4, 2)
    a.set_chunks(3)
    a.step(2)
    a.set_owned(1, 8)
    a.set_owned(0, 9)
    t = aero.Batch([a, b])
    t.tune(2)
    t.dispose()
    assert not [l for l in log() if l[0] == "cudaDeviceSynchronize"]
    fake.fake_clear()
    own = str(a.stream)
    a.dispose()
    L = log()
    freed = [i for i, l in enumerate(L) if l[0] in ("cudaFree", "cudaFreeAsync")]
    waited = {l[1] for l in L[:freed[0]] if l[0] == "cudaStreamSynchronize"}
    assert waited == {own}                                           # which comes after the chunks'
    assert not [l for l in L if l[0] == "cudaMalloc"]                # nobody else had its address
    c = box(6, 4, 9)
    c.set_kernel(4, 2)
    c.set_chunks(3)
    c.step(1)
    fake.fake_fail(b"launch", 1, 5)                                  # a step that fails half-way
    assert lib.a3d_solver_step(c._h, 1) != 0
    own = str(c.stream)
    fake.fake_clear()
    c.dispose()
    L = log()
    freed = [i for i, l in enumerate(L) if l[0] in ("cudaFree", "cudaFreeAsync")]
    waited = {l[1] for l in L[:freed[0]] if l[0] == "cudaStreamSynchronize"}
    assert own in waited and len(waited) == 4                        # the chunks' own too
    b.plane_ptr(0, 0, 0)                                             # b's address is out: the device is waited for
    fake.fake_clear()
    b.dispose()
    order = [l[0] for l in log()]
    assert order.index("cudaMalloc") < order.index("cudaFree") < order.index("cudaFreeAsync")
    assert not [l for l in log() if l[0] == "cudaDeviceSynchronize"]
    """)


def test_a_solver_can_be_dropped_when_memory_has_run_out(fake):
    """Whose address a caller holds: there is no byte left to wait for the device with."""
    fake("""
    s = box(6, 4, 9)
    s.plane_ptr(0, 0, 0)
    fake.fake_set(b"limit", 0)
    assert lib.a3d_solver_destroy(s._h) == 0
    s._h = C.c_void_p()
    assert fake.fake_live() == 0
    assert [l for l in log() if l[0] == "cudaDeviceSynchronize"]
    """)


def test_memory_of_a_solver_that_could_not_be_waited_for_is_not_recycled(fake):
    fake("""
    s = box(6, 4, 9)
    mine, live = str(s.stream), fake.fake_live()
    fake.fake_fail(b"cudaStreamSynchronize", 900, 1)
    fake.fake_clear()
    assert lib.a3d_solver_destroy(s._h) != 0 and b"wait" in lib.a3d_last_error()
    assert fake.fake_live() == live
    o = box(6, 4, 9)
    assert str(o.stream) != mine
    assert lib.a3d_solver_destroy(s._h) == 0                         # later it can be
    s._h = C.c_void_p()
    """)


def test_a_block_waits_for_no_other_solver(fake):
    """The pool does not hand out memory that another stream has yet to give back, and a thread that frees
    a large case, which waits for the device, holds up no other thread's case."""
    fake("""
    import threading, time
    big = box(600, 200, 40)                                          # 288 MB of state: of cudaMalloc
    a = [l for l in log() if l[0] == "cudaMemPoolSetAttribute"]
    REUSE_ALLOW_INTERNAL_DEPENDENCIES = 3
    assert [l[3] for l in a if int(l[2]) == REUSE_ALLOW_INTERNAL_DEPENDENCIES] == ["0"]
    fake.fake_set(b"free_us", 2000000)
    t = threading.Thread(target=big.dispose)
    t.start()
    time.sleep(0.3)
    t0 = time.time()
    small = box(6, 4, 9)
    assert time.time() - t0 < 1 and t.is_alive()
    t.join()
    fake.fake_set(b"free_us", 0)
    """)


def test_a_force_list_that_found_no_memory_is_empty(fake):
    """Choosing other planes makes a new list; if there is no memory for it the call says so, and no
    list is left whose length speaks of cells that it does not have."""
    fake("""
    fake.fake_set(b"entries", 40)
    s = box(6, 4, 9)
    n = C.c_int64()
    L.check(lib.a3d_solver_force_list(s._h, C.byref(n), 0, None, None, None, None, None))
    assert n.value == 40
    fake.fake_fail(b"cudaMallocFromPoolAsync", 2, 2)                 # the offsets' block, then the list's
    assert lib.a3d_solver_set_owned(s._h, 1, 8) == 3
    L.check(lib.a3d_solver_force_list(s._h, C.byref(n), 0, None, None, None, None, None))
    assert n.value == 0
    """)


def test_planes_can_be_reached_from_peer_devices(fake):
    """cudaDeviceEnablePeerAccess covers memory of cudaMalloc but not of a pool: where a state's address
    goes out, or another device's slab stores into it, the pool is opened to the peers, once."""
    fake("""
    grants = lambda: [l[1:] for l in log() if l[0] == "cudaMemPoolSetAccess"]
    READ_WRITE = "3"
    a, b = box(6, 4, 9), box(6, 4, 9)
    assert grants() == []
    for s in (a, a, b):
        s.plane_ptr(0, 0, 0)
    assert grants() == [["1", "1", READ_WRITE]]                      # device 0's pool to device 1
    c = box(6, 4, 9, device=1)
    for _ in range(5):
        c.copy_planes_from(a, 0, 4, 2, 0)
    assert sorted(grants()) == [["1", "1", READ_WRITE], ["2", "0", READ_WRITE]]
    """)


@pytest.mark.parametrize("size", ["6, 4, 9", "600, 200, 40"])  # state in the pool, from cudaMalloc
def test_a_solver_may_be_destroyed_while_the_process_exits(fake, size):
    """By an exit handler, a global object of the program or a thread that still runs: the pools are
    there to the end.  (Freed memory is overwritten in these tests, so that its use shows.)"""
    fake(f"""
    s = box({size})
    fake.fake_at_exit(lib.a3d_solver_destroy, s._h)
    s._h = C.c_void_p()
    """)


@pytest.mark.parametrize("kernel,NZ,chunks", [(2, 79, 1), (2, 80, 4), (2, 94, 4), (2, 280, 4),
                                              (4, 80, 1), (4, 94, 1), (4, 95, 3), (4, 269, 3), (4, 270, 4)])
def test_automatic_chunks_of_each_tile(fake, kernel, NZ, chunks):
    """Planes of 10,000 cells: the paired tile's dependent launches hold longer than the single-cell
    tile's plain ones."""
    fake(f"""
    s = box(100, 100, {NZ})
    s.set_kernel({kernel})
    assert s.chunks() == {chunks}
    """)


@pytest.mark.parametrize("cases,run", [(1, 1), (2, 1), (3, 2), (5, 2), (6, 4), (11, 4), (12, 8), (36, 8), (37, 16)])
def test_z_run_of_a_batch(fake, cases, run):
    """Cases of 16 columns by 16 planes on 296 resident thread blocks, one wave of single planes each
    alone: single planes up to 1.8 waves, then two; 4, 8 and 16 planes as soon as their rules hold.  A case
    with a run of its own keeps it."""
    fake(f"""
    ss = [box(128, 64, 16) for _ in range({cases})]
    assert all(s.kernel() == (4, 1) for s in ss)
    def runs():
        b = aero.Batch(ss)
        fake.fake_clear()
        b.step(2)
        got = [16 // int(l[2]) for l in log() if l[0] == "launch"]
        assert len(got) == 4 * len(ss) and all(s.kernel()[0] == 4 for s in ss)
        return got
    assert set(runs()) == {{{run}}}
    assert all(s.kernel() == (4, 1) for s in ss)
    ss[0].set_kernel(4, 8)
    assert set(runs()[:4]) == {{8}}
    """)


@pytest.mark.parametrize("size", ["60, 40, 50", "600, 200, 40"])  # the state in the pool, from cudaMalloc
@pytest.mark.parametrize("make", ["box({})", "aero.CfdGPU(box_grid({}), shape=shape)"])
def test_a_case_without_memory_fails_alone(fake, size, make):
    """The call that found no memory says so and leaves nothing behind: neither blocks, nor a CUDA
    error that another solver's next launch would report."""
    fake(f"""
    shape = aero.shape_of(aero.build_aircraft("fighter"))
    def box_grid(*n):
        return cfd.Grid(*[np.arange(k + 1, dtype=np.float64) for k in n])
    s = box(6, 4, 9)
    live = fake.fake_live()
    for limit in (10**4, 10**6, 3 * 10**6, 5 * 10**6, 12 * 10**6, 10**8, 3 * 10**8):
        fake.fake_set(b"limit", limit)
        try:
            x = {make.format(size)}
        except aero.AeroError as e:
            assert e.status == 3, e
        else:
            x.dispose()
            del x
        s.step(2)
        s.mach_max()
        assert fake.fake_live() == live
    fake.fake_set(b"limit", 1 << 50)
    """)
