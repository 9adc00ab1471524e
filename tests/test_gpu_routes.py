"""Calls at the edges of the rules that choose the kernels give on every route
what the plain per-step kernels give.  GPU only."""
import ctypes

import numpy as np
import pytest
import torch

import ernn_gb300 as E
from cases import DT, H, RHO, random_case, rel
from oracle import oracle as O
from test_gpu_block import run
from test_gpu_instances import _canvas, _instances, _run_canvas, _run_single, _weights
from test_gpu_parity import DEV, FWD_TOL, GRAD_TOL, run_oracle, to_geometry, weights

pytestmark = pytest.mark.gpu


def forward_into_poison(case, path):
    """ernn_forward through the C ABI, whose receiver indices are device data
    that no host check sees, into outputs full of NaN."""
    geom = to_geometry(case, path=path)
    lib = E.load_library()
    prob = geom.problem(case.mode)
    C = torch.tensor(case.C, dtype=torch.float32, device=DEV)
    D = None if case.D is None else torch.tensor(case.D, dtype=torch.float32, device=DEV)
    rho = torch.tensor([case.rho], dtype=torch.float32, device=DEV)
    out = torch.full((2,) + geom.out_shape(), float("nan"), device=DEV)
    ptr = lambda t: ctypes.c_void_p(None if t is None else t.data_ptr())
    ins = E._lib.ErnnInputs(ptr(C), ptr(D), ptr(rho), ptr(geom.src_signal), ptr(geom.src_map), ptr(geom.src_origin),
                            ptr(geom.rec_idx))
    n = lib.ernn_tape_bytes(ctypes.byref(prob), 1)
    tape = torch.empty(n, dtype=torch.uint8, device=DEV)
    rc = lib.ernn_forward(ctypes.byref(prob), ctypes.byref(ins), ptr(out[0]), ptr(out[1]), ptr(tape),
                          ctypes.c_size_t(n), 1, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    return out.cpu().numpy(), lib.ernn_last_path()


@pytest.mark.parametrize("kw,path", [
    (dict(nx=61, ny=243), E.PATH_TILED),                              # passes of one launch
    (dict(nx=313, ny=389, S=3), E.PATH_TILED),                        # a launch per pass
    (dict(nx=61, ny=243, mode=O.MODE_DFIELD), E.PATH_TILED),
    (dict(nx=61, ny=243, mode=O.MODE_FIELDS), E.PATH_TILED),
    (dict(nx=64, ny=64, S=2), E.PATH_RESIDENT),
    (dict(nx=61, ny=33), E.PATH_STEP),
])
def test_receivers_outside_the_grid_record_zeros(kw, path):
    case = random_case(nt=23, stride=2, record=O.RECORD_RECEIVERS, nrec=12, **kw)
    inside = case.rec_idx.copy()
    case.rec_idx[:, [0, 5, 11]] = [-1, case.nx * case.ny, -2 ** 31]
    case.rec_idx[0, 7] = 2 ** 31 - 1
    got, used = forward_into_poison(case, E.PATH_AUTO)
    assert used == path
    want, _ = forward_into_poison(case, E.PATH_STEP)
    out = case.rec_idx != inside  # (S, nrec)
    shot, rec = np.nonzero(out)
    assert np.all(got[:, shot, :, rec] == 0) and np.all(want[:, shot, :, rec] == 0)
    assert np.all(np.isfinite(got)) and rel(got, want) <= 1e-5


@pytest.mark.parametrize("kw", [
    dict(nx=64, ny=64, S=2, nrec=1025),    # more receivers than a CTA of a cluster may own
    dict(nx=128, ny=132, nrec=1500),
    dict(nx=20, ny=1600, nrec=9),          # no cluster size whose CTAs all own rows and hold them
])
def test_problems_that_no_cluster_takes_run_on_tiles(kw):
    case = random_case(nt=50, record=O.RECORD_RECEIVERS, **kw)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, 12)
    assert used == E.PATH_TILED
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, 12)
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


# Grids whose rows one tile holds: 88 rows of at most 64 columns, 40 of at most
# 128; grids lower than a tile's 24 rows.
ROWS64 = [(88, 41, 153), (89, 63, 120), (97, 61, 120), (177, 43, 95), (180, 57, 62)]
ROWS128 = [(40, 121, 153), (41, 127, 153), (180, 125, 31), (121, 123, 40)]
LOW = [(1, 1601, 22), (4, 1501, 25), (8, 241, 70), (23, 365, 50)]


@pytest.mark.parametrize("nx,ny,S", ROWS64 + ROWS128 + LOW)
@pytest.mark.parametrize("record,nrec", [(O.RECORD_FIELDS, 0), (O.RECORD_RECEIVERS, 200)])
@pytest.mark.parametrize("nt,ckpt_k", [(22, None), (27, 6)])
def test_narrow_and_low_odd_grids(nx, ny, S, record, nrec, nt, ckpt_k):
    """The plain kernels' rounding order: bit for bit."""
    case = random_case(nx=nx, ny=ny, nt=nt, S=S, record=record, nrec=nrec, stride=1 + nt % 2, src_comp=nx % 2)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, ckpt_k)
    assert used == E.PATH_TILED
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, ckpt_k)
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


@pytest.mark.parametrize("nx,ny,S,path", [
    (5000, 32, 4, E.PATH_AUTO), (4000, 36, 5, E.PATH_AUTO),      # rows below 40 cells, 608 tiles of 64 x 32
    (20000, 4, 1, E.PATH_TILED), (4500, 64, 5, E.PATH_AUTO),
    (300, 8, 40, E.PATH_TILED), (177, 60, 95, E.PATH_TILED), (89, 64, 120, E.PATH_TILED),
    (180, 124, 31, E.PATH_TILED), (41, 128, 160, E.PATH_TILED),
])
@pytest.mark.parametrize("per_shot", [False, True])
def test_narrow_grids_of_whole_quads(nx, ny, S, path, per_shot):
    """The tiled rounding order: equal to the plain kernels' to FP32 rounding
    over 30 steps (2^-24 a step and term, as between the two orders before)."""
    case = random_case(nx=nx, ny=ny, nt=30, S=S, record=O.RECORD_RECEIVERS, nrec=150, stride=2)
    case.rec_idx[:, 0] = case.src_origin[:, 0].clip(0, nx - 1) * ny + case.src_origin[:, 1].clip(0, ny - 1)
    wx, wy = weights(case)
    got = []
    for pth in (path, E.PATH_STEP):
        geom = to_geometry(case, 7, pth)
        C = torch.tensor(case.C, dtype=torch.float32, device=DEV)
        rho = torch.tensor(case.rho, dtype=torch.float32, device=DEV)
        if per_shot:
            C = C[None] * (1 + 0.05 * torch.arange(S, device=DEV)[:, None] / S)
            rho = rho.reshape(1).repeat(S)
        C.requires_grad_(True)
        ux, uy = E.propagate(C, rho, geom)
        assert E.load_library().ernn_last_path() == (E.PATH_TILED if pth == path else E.PATH_STEP)
        ((ux.double() * torch.as_tensor(wx, device=DEV)).sum() + (uy.double() * torch.as_tensor(wy, device=DEV)).sum()).backward()
        got.append((ux.detach().cpu().numpy(), uy.detach().cpu().numpy(), C.grad.double().cpu().numpy()))
    for a, b in zip(*got):
        assert np.any(b != 0) and rel(a, b) <= 1e-5, rel(a, b)


@pytest.mark.parametrize("ckpt_k", [None, 6])
def test_canvas_of_narrow_instances(ckpt_k):
    """Instances whose rows one tile holds (two waves of 40-row tiles, one of
    whole-row tiles): each one's traces as if run alone, bit for bit, its
    gradient against the 64-bit oracle (alone it has other tiles, and with
    them other FP32 partial sums)."""
    rng = np.random.default_rng(2)
    specs = [(int(rng.integers(180, 330)), 4 * int(rng.integers(2, 17)), int(rng.integers(9, 30))) for _ in range(70)]
    specs[:4] = [(176, 64, 30), (177, 60, 29), (88, 8, 9), (8, 64, 17)]
    insts = _instances(specs)
    geom = _canvas(insts, ckpt_k)
    wx, wy = _weights(insts, geom.nt)
    cx, cy, cg = _run_canvas(insts, geom, wx, wy)
    for k, d in enumerate(insts):
        nt = d["nt"]
        sx, sy, sg = _run_single(d, wx[k:k + 1, :nt], wy[k:k + 1, :nt], ckpt_k)
        assert np.array_equal(cx[k, :nt], sx) and np.array_equal(cy[k, :nt], sy), k
        assert not np.any(cx[k, nt:]) and not np.any(cy[k, nt:])
        case = O.Case(d["nx"], d["ny"], nt, H, DT, RHO, d["C"], d["sig"][None].astype(np.float64),
                      d["smap"][None].astype(np.float64), np.array([d["org"]], np.int32), record=O.RECORD_RECEIVERS,
                      rec_idx=d["rec"][None])
        gC, _ = O.adjoint(case, O.forward(case, "f64", keep_states=True)[2], wx[k:k + 1, :nt], wy[k:k + 1, :nt], "f64")
        assert rel(cg[k], gC) <= GRAD_TOL and rel(sg, gC) <= GRAD_TOL, (k, rel(cg[k], gC), rel(sg, gC))


@pytest.mark.parametrize("nx,ny,S", [(61, 127, 1), (200, 243, 3)])  # passes of one launch; a launch per pass
@pytest.mark.parametrize("nrec", [1, 40, 511, 513, 1100])
def test_constant_planes_with_receivers_crowded_on_a_tile(nx, ny, S, nrec):
    """Around the 512 threads of a tile's CTA, on both sides of tile edges
    (rows 8 k, column 120), two receivers on one cell among them."""
    case = random_case(nx=nx, ny=ny, nt=20, S=S, mode=O.MODE_FIELDS, record=O.RECORD_RECEIVERS, nrec=nrec)
    cells = np.array([i * ny + j for j in range(60, 127) for i in range(5, 27)])
    case.rec_idx[:] = np.random.default_rng(nrec).permutation(cells)[:nrec]
    case.rec_idx[:, -1] = case.rec_idx[:, 0]
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, 6)
    assert used == E.PATH_TILED
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, 6)
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


# Grids on the 40-row tiles, around multiples of 40 rows and 120 columns.
@pytest.mark.parametrize("mode,nx,ny,S", [
    (O.MODE_SCALAR, 80, 129, 51), (O.MODE_SCALAR, 161, 131, 26), (O.MODE_SCALAR, 79, 241, 34),
    (O.MODE_DFIELD, 81, 361, 24), (O.MODE_DFIELD, 121, 243, 24), (O.MODE_DFIELD, 241, 361, 9),
])
@pytest.mark.parametrize("record,nrec", [(O.RECORD_FIELDS, 0), (O.RECORD_RECEIVERS, 150)])
@pytest.mark.parametrize("nt,ckpt_k", [(17, None), (23, 6)])
def test_forty_row_tiles(mode, nx, ny, S, record, nrec, nt, ckpt_k):
    case = random_case(nx=nx, ny=ny, nt=nt, S=S, mode=mode, record=record, nrec=nrec, stride=1 + nt % 2, src_comp=nx % 2)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, ckpt_k)
    assert used == E.PATH_TILED
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, ckpt_k)
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


@pytest.mark.parametrize("mode", [O.MODE_DFIELD, O.MODE_FIELDS])
@pytest.mark.parametrize("nx,ny", [(8, 120), (25, 121), (41, 243), (40, 119)])
@pytest.mark.parametrize("record,nrec", [(O.RECORD_FIELDS, 0), (O.RECORD_RECEIVERS, 60)])
def test_per_cell_modes_vs_fp64_oracle_at_tile_edges(mode, nx, ny, record, nrec):
    case = random_case(nx=nx, ny=ny, nt=45, S=2, mode=mode, record=record, nrec=nrec)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, 11)
    assert used == E.PATH_TILED
    ox, oy, og = run_oracle(case, wx, wy)
    assert rel(ax, ox) <= FWD_TOL and rel(ay, oy) <= FWD_TOL
    assert rel(ag, og) <= GRAD_TOL, rel(ag, og)


@pytest.mark.parametrize("mode", [O.MODE_SCALAR, O.MODE_FIELDS])
def test_the_profiler_times_the_launches_of_an_unprofiled_call(mode):
    """Passes that share a launch share it under the profiler too."""
    case = random_case(nx=61, ny=243, nt=120, mode=mode, record=O.RECORD_RECEIVERS, nrec=12)
    wx, wy = weights(case)
    lib = E.load_library()

    def launches():
        n = lib.ernn_launch_count()
        run(case, wx, wy, E.PATH_AUTO, None)
        return lib.ernn_launch_count() - n
    plain = launches()
    E._lib.profile(True)
    try:
        profiled = launches()
        torch.cuda.synchronize()
        prof = E._lib.profile_read()
    finally:
        E._lib.profile(False)
    assert profiled == plain
    # 120 steps are 30 passes of four: two launches each way
    assert prof["forward"][1] == 2 and prof["adjoint"][1] == 2
