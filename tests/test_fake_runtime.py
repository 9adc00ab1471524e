"""The host side of the library on a CUDA runtime that only records
(tests/abi_c/fake_cudart.c): what is launched, on which device, with which
workspaces, and what happens when the runtime refuses.  Runs on the CPU; no
kernel runs."""
import ctypes
import os
import shutil
import subprocess

import pytest

import ernn_gb300 as E
from conftest import ROOT

TAPE, SCRATCH, DATA = 1 << 40, 1 << 41, 1 << 42  # addresses that are never dereferenced


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gcc = shutil.which("gcc")
    include = "/usr/local/cuda/include"
    E.load_library()  # builds the objects where they are missing
    out_dir = os.path.dirname(E._lib.library_path())
    objs = [os.path.join(out_dir, os.path.basename(f)[:-3] + ".o") for f in E._lib._build.sources()]
    if gcc is None or not os.path.exists(os.path.join(include, "cuda_runtime_api.h")) or not all(map(os.path.exists, objs)):
        pytest.skip("gcc, the CUDA headers or the library's objects absent")
    out = str(tmp_path_factory.mktemp("fake") / "libernn_fake.so")
    subprocess.run([gcc, "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", include,
                    os.path.join(ROOT, "tests", "abi_c", "fake_cudart.c"), *objs, "-lstdc++", "-o", out], check=True)
    lib = ctypes.CDLL(out)
    for name, (res, args) in E._lib.SIGNATURES.items():
        f = getattr(lib, name)
        f.restype, f.argtypes = res, args
    lib.fake_launch.restype = ctypes.c_char_p
    lib.fake_memset.restype = ctypes.c_void_p
    return lib


def setup(lib, device=0, sms=152, refuse_cooperative=0, clusters=1):
    lib.fake_set(device, sms, refuse_cooperative, clusters)
    lib.fake_reset()


def problem(**kw):
    base = dict(nshots=1, nx=64, ny=48, nt=20, stride=1, mode=0, record=1, nrec=8, src_comp=1, src_bx=9, src_by=9,
                ckpt_k=20, path=0, flags=0, h=1e-4, dt=5e-9)
    base.update(kw)
    return E._lib.ErnnProblem(*[base[f] for f, _ in E._lib.ErnnProblem._fields_])


def call(lib, p, tape=TAPE, scratch=SCRATCH):
    """ernn_forward and ernn_adjoint; their return codes."""
    ptr = ctypes.c_void_p
    ins = E._lib.ErnnInputs(*[ptr(DATA + (k << 36)) for k in range(7)])
    nt, ns = lib.ernn_tape_bytes(ctypes.byref(p), 1), lib.ernn_adjoint_scratch_bytes(ctypes.byref(p))
    a, b, c, d = (ptr(DATA + (k << 36)) for k in (8, 9, 10, 11))
    return (lib.ernn_forward(ctypes.byref(p), ctypes.byref(ins), a, b, ptr(tape), nt, 1, None),
            lib.ernn_adjoint(ctypes.byref(p), ctypes.byref(ins), a, b, ptr(tape), nt, ptr(scratch), ns, c, d, None))


def launches(lib):
    """(kernel, device, cooperative, grid, first bytes of the first argument) of every launch since setup."""
    out = []
    for i in range(lib.fake_launches()):
        v, smem, arg = (ctypes.c_int * 5)(), ctypes.c_size_t(), (ctypes.c_ubyte * 96)()
        name = lib.fake_launch(i, v, ctypes.byref(smem), arg).decode()
        out.append((name, v[0], v[1], v[2], bytes(arg)))
    return out


@pytest.mark.parametrize("kw", [
    dict(nx=61, ny=43), dict(nx=200, ny=243, nshots=4), dict(nx=300, ny=301, nshots=9), dict(path=3), dict(mode=1, ny=47),
    dict(mode=1, path=3), dict(mode=2, ny=47), dict(nx=128, ny=128), dict(mode=2, nx=200, ny=243, nshots=4),
])
def test_every_device_of_a_process_gets_its_own_limits(lib, kw):
    for device in (0, 1, 0, 2):
        setup(lib, device)
        assert call(lib, problem(**kw)) == (0, 0), device
        assert lib.fake_launches() > 0 and all(l[1] == device for l in launches(lib))


def test_grids_follow_the_device_they_run_on(lib):
    p = problem(nx=300, ny=301, nshots=16)  # more tiles than either device has slots for
    grid = {}
    for device, sms in ((0, 152), (3, 40)):
        setup(lib, device, sms)
        assert call(lib, p) == (0, 0)
        grid[device] = max(l[3] for l in launches(lib) if "blk_adj_kernel" in l[0])
    assert grid == {0: 304, 3: 80}


@pytest.mark.parametrize("sms", [152, 132, 40])
@pytest.mark.parametrize("kw", [
    dict(mode=1, nx=960, ny=1216),             # 570 tiles of 64 x 32: the tiles of four steps
    dict(mode=1, nx=1024, ny=1216),            # 608: the tiled per-step kernels
    dict(mode=1, nx=1024, ny=1216, path=3), dict(mode=1, nx=961, ny=1215), dict(nx=960, ny=1216), dict(nx=960, ny=1215),
])
def test_work_areas_are_cleared_inside_the_buffers(lib, kw, sms):
    """Also with a tape that is on no 16-byte boundary, which changes the
    kernels but not the sizes that were asked for."""
    p = problem(ckpt_k=7, **kw)
    nt, ns = lib.ernn_tape_bytes(ctypes.byref(p), 1), lib.ernn_adjoint_scratch_bytes(ctypes.byref(p))
    for tape, scratch in ((TAPE, SCRATCH), (TAPE + 8, SCRATCH + 8)):
        setup(lib, 0, sms)
        assert call(lib, p, tape, scratch) == (0, 0)
        for i in range(lib.fake_memsets()):
            n = ctypes.c_size_t()
            a = lib.fake_memset(i, ctypes.byref(n))
            inside = [lo <= a and a + n.value <= lo + size for lo, size in ((tape, nt), (scratch, ns))]
            assert any(inside) or a >= DATA, (hex(a), n.value)


@pytest.mark.parametrize("mode,S,nx,ny,tiles", [
    # grids measured on either side of the line between plain and time-blocked kernels
    (2, 1, 301, 301, True), (2, 20, 130, 130, True), (2, 16, 250, 250, True), (2, 1, 3000, 240, True),
    (2, 1, 4000, 42, True), (2, 40, 130, 130, True), (2, 100, 9, 1000, True), (2, 1, 1000, 1000, True),
    (2, 300, 50, 50, False), (2, 120, 64, 64, False), (2, 1, 8000, 61, False), (2, 1, 20000, 48, False),
    (1, 1, 301, 301, True), (1, 7, 301, 301, True), (1, 1, 700, 701, True), (1, 30, 130, 130, True),
    (1, 40, 17, 1001, True), (1, 8, 98, 560, True), (1, 300, 40, 41, True), (1, 2, 512, 512, True),
    (1, 8, 500, 121, False), (1, 1, 8000, 61, False), (1, 6, 2000, 123, False), (1, 300, 24, 121, False),
    (1, 10, 200, 201, False), (1, 7, 563, 51, False),
])
def test_per_cell_modes_take_the_kernels_measured_faster(lib, mode, S, nx, ny, tiles):
    setup(lib)
    assert call(lib, problem(mode=mode, nshots=S, nx=nx, ny=ny)) == (0, 0)
    assert lib.ernn_last_path() == (E.PATH_TILED if tiles else E.PATH_STEP)



@pytest.mark.parametrize("S,nx,ny,kept,ckpt,alone", [
    # constant planes: every state kept, checkpoints every 13 steps, forward alone (True: tiles)
    (8, 301, 301, True, True, True), (1, 1000, 1000, True, True, True), (1, 301, 301, True, True, True),
    (16, 250, 250, True, False, False), (20, 130, 130, True, False, False), (3, 2245, 136, False, False, False),
    (2, 3000, 44, True, False, False), (300, 50, 50, False, False, False),
])
def test_constant_planes_ask_for_what_a_call_runs(lib, S, nx, ny, kept, ckpt, alone):
    names = {True: E.PATH_TILED, False: E.PATH_STEP}
    setup(lib)
    for k, want in ((26, kept), (13, ckpt)):
        assert call(lib, problem(mode=2, nshots=S, nx=nx, ny=ny, nt=26, ckpt_k=k)) == (0, 0)
        assert lib.ernn_last_path() == names[want], k
    p = problem(mode=2, nshots=S, nx=nx, ny=ny, nt=26, ckpt_k=26)
    ptr = ctypes.c_void_p
    ins = E._lib.ErnnInputs(*[ptr(DATA + (k << 36)) for k in range(7)])
    n = lib.ernn_tape_bytes(ctypes.byref(p), 0)
    assert lib.ernn_forward(ctypes.byref(p), ctypes.byref(ins), ptr(DATA + (8 << 36)), ptr(DATA + (9 << 36)), ptr(TAPE), n, 0,
                            None) == 0
    assert lib.ernn_last_path() == names[alone]


class Pass(ctypes.Structure):
    """The first fields of BlkFwd and BlkAdj (out: of BlkAdj the last two levels)."""
    _fields_ = [(n, ctypes.c_int32) for n in ("geo", "plain_order", "nx", "ny", "pitch", "S", "nt", "step", "T")] + [
        ("cur", ctypes.c_uint64), ("prev", ctypes.c_uint64), ("out", ctypes.c_uint64 * 2)]


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("nt,ckpt_k", [(30, 30), (205, 205), (205, 103), (97, 9)])
def test_refused_cooperative_launches_become_a_launch_per_pass(lib, mode, nt, ckpt_k):
    """The passes of a refused run, in order, with the states they read and
    write: those of a call that never tries runs."""
    p = problem(nx=61, ny=243, mode=mode, nt=nt, ckpt_k=ckpt_k)

    def passes(**kw):
        setup(lib, **kw)
        assert call(lib, p) == (0, 0)
        out = []
        for name, _, coop, _, arg in launches(lib):
            assert not coop
            if "blk_" in name:
                a = Pass.from_buffer_copy(arg)
                out.append((name, a.step, a.T, a.cur, a.prev, a.out[0], a.out[1]))
        return out
    refused = passes(refuse_cooperative=1)
    lib.ernn_set_launch_overlap(0)
    try:
        apart = passes()
    finally:
        lib.ernn_set_launch_overlap(1)
    assert refused == apart and len(apart) >= 2 * (nt // 4)
    setup(lib)
    assert call(lib, p) == (0, 0)
    assert any(coop for _, _, coop, _, _ in launches(lib))  # (they are runs where the runtime takes them)


@pytest.mark.parametrize("kw,mode", [
    (dict(nx=61, ny=43, nt=200), "scalar"), (dict(nx=300, ny=301, nshots=9, nt=20), "scalar"),
    (dict(nx=61, ny=43, mode=2, nt=200), "fields"), (dict(nx=200, ny=243, nshots=4, mode=2), "fields"),
    (dict(nx=61, ny=43, mode=1), "damage"), (dict(nx=1024, ny=1216, mode=1), "damage"),
    (dict(nx=128, ny=128), "scalar"), (dict(nx=61, ny=33), "scalar"), (dict(nx=61, ny=33, mode=1), "damage"),
])
def test_bench_names_the_kernels_that_run(lib, kw, mode):
    import bench
    setup(lib)
    p = problem(**{**kw, "ckpt_k": kw.get("nt", 20)})
    assert call(lib, p) == (0, 0)
    loop = [l[0] for l in launches(lib) if any(k in l[0] for k in ("blk_", "run_", "tma_", "step_kernel", "resident"))]
    adjoint = [l for l in loop if "adj" in l]
    names = bench.kernel_names(lib.ernn_last_path(), mode, p.nt / max(len(adjoint), 1))
    assert any(names["forward"] in l for l in loop) and any(names["adjoint"] in l for l in loop), (names, set(loop))
