"""Time-blocked tile kernels (up to four steps per launch) against the plain
per-step kernels at the sizes where a tile ends: stored rows of a tile (24 and
40), its 120 columns, halo columns, quads cut by the grid's last column, step
counts that leave launches of one to three steps, checkpoints on and off them.

Both evaluate the same sequence of rounded operations per cell, so the
recorded fields are equal bit for bit; the gradient's sums group their FP32
partial sums differently (relative 2^-24 sqrt(terms of a partial sum), below
1e-5).  GPU only."""
import numpy as np
import pytest
import torch

import ernn_gb300 as E
from cases import random_case, rel
from oracle import oracle as O
from test_gpu_parity import DEV, GRAD_TOL, run_oracle, to_geometry, weights

pytestmark = pytest.mark.gpu


def run(case, wx, wy, path, ckpt_k):
    geom = to_geometry(case, path=path, ckpt_k=ckpt_k)
    C = torch.tensor(case.C, dtype=torch.float32, device=DEV, requires_grad=case.D is None)
    D = None if case.D is None else torch.tensor(case.D, dtype=torch.float32, device=DEV, requires_grad=True)
    ux, uy = E.propagate(C, torch.tensor(case.rho, dtype=torch.float32, device=DEV), geom, D=D)
    used = E.load_library().ernn_last_path()
    ((ux.double() * torch.as_tensor(wx, device=DEV)).sum() + (uy.double() * torch.as_tensor(wy, device=DEV)).sum()).backward()
    return ux.detach().cpu().numpy(), uy.detach().cpu().numpy(), (C if D is None else D).grad.double().cpu().numpy(), used


SIZES = [(8, 41), (17, 40 + 3), (24, 41), (25, 119), (23, 121), (40, 122), (41, 127), (48, 129), (3, 243), (97, 250), (130, 361)]


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("record", [O.RECORD_FIELDS, O.RECORD_RECEIVERS])
@pytest.mark.parametrize("nt,ckpt_k", [(41, None), (42, 7), (30, 1), (33, 6)])
def test_same_fields_as_the_plain_kernels(nx, ny, record, nt, ckpt_k):
    case = random_case(nx=nx, ny=ny, nt=nt, S=2, stride=1 + nt % 2, record=record, nrec=min(40, nx * ny),
                       src_comp=nx % 2)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, ckpt_k)
    assert used == E.PATH_TILED  # ny % 4 != 0: not the resident path's
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, ckpt_k)
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


@pytest.mark.parametrize("mode", [O.MODE_DFIELD, O.MODE_FIELDS])
@pytest.mark.parametrize("nx,ny", [(8, 41), (25, 119), (23, 124), (61, 76), (97, 250)])
@pytest.mark.parametrize("record", [O.RECORD_FIELDS, O.RECORD_RECEIVERS])
@pytest.mark.parametrize("nt,ckpt_k", [(37, None), (30, 1), (33, 6)])
def test_per_cell_modes_same_fields_as_the_plain_kernels(mode, nx, ny, record, nt, ckpt_k):
    case = random_case(nx=nx, ny=ny, nt=nt, S=2, stride=1 + nt % 2, mode=mode, record=record, nrec=40, src_comp=nx % 2)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, ckpt_k)
    assert used == E.PATH_TILED
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, ckpt_k)
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


@pytest.mark.parametrize("mode", [O.MODE_SCALAR, O.MODE_DFIELD, O.MODE_FIELDS])
def test_every_cell_a_receiver(mode):
    case = random_case(nx=50, ny=126, nt=20, S=2, mode=mode, record=O.RECORD_RECEIVERS, nrec=50 * 126, stride=2)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, 6)
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, 6)
    assert used == E.PATH_TILED
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


@pytest.mark.parametrize("kw,ckpt_k", [
    (dict(nx=170, ny=133, nt=300, S=3, record=O.RECORD_RECEIVERS, nrec=40), 9),
    (dict(nx=130, ny=361, nt=250, stride=3, record=O.RECORD_RECEIVERS, nrec=1500), None),
    (dict(nx=145, ny=79, nt=400, stride=2), None),
    (dict(nx=330, ny=437, nt=120, S=9, record=O.RECORD_RECEIVERS, nrec=60), 20),  # several tiles per CTA
])
def test_gradient_of_each_constant_follows_the_plain_kernels(kw, ckpt_k):
    """The adjoint states are the plain kernels' bit for bit, so only the order
    of the imaging sums differs: FP32 over a thread's cells of one step (24 at
    most: 2^-24 sqrt(24) = 3e-7 of the terms, averaged over the steps)."""
    case = random_case(**kw)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, ckpt_k)
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, ckpt_k)
    assert used == E.PATH_TILED
    assert np.all(np.abs(ag - bg) <= 1e-6 * np.abs(bg) + 1e-7 * np.abs(bg).max()), (ag, bg)


@pytest.mark.parametrize("mode,S,nx,ny,path", [
    (O.MODE_SCALAR, 16, 941, 41, E.PATH_TILED), (O.MODE_DFIELD, 8, 98, 559, E.PATH_TILED),
    (O.MODE_DFIELD, 7, 563, 51, E.PATH_STEP), (O.MODE_DFIELD, 1, 563, 51, E.PATH_TILED),
])
def test_narrow_grids_on_either_side_of_the_cost_rule(mode, S, nx, ny, path):
    case = random_case(nx=nx, ny=ny, nt=9, S=S, mode=mode, record=O.RECORD_RECEIVERS, nrec=12)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, 4)
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, 4)
    assert used == path
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


@pytest.mark.parametrize("mode,S,nx,ny", [
    (O.MODE_SCALAR, 1, 41, 242), (O.MODE_FIELDS, 2, 41, 122),    # 8-row tiles, one per SM
    (O.MODE_SCALAR, 5, 121, 361), (O.MODE_SCALAR, 9, 49, 241),   # 24-row tiles
    (O.MODE_SCALAR, 3, 313, 389), (O.MODE_SCALAR, 13, 105, 243), # more tiles than SMs: a launch per pass
])
@pytest.mark.parametrize("record,nrec", [(O.RECORD_FIELDS, 0), (O.RECORD_RECEIVERS, 70)])
@pytest.mark.parametrize("nt,ckpt_k,stride", [(102, None, 1), (205, 103, 3), (61, 17, 1)])
def test_runs_of_passes(mode, S, nx, ny, record, nrec, nt, ckpt_k, stride):
    """Several passes per launch, tiles kept in registers between them: step
    counts over one launch (24 passes of four steps), odd last passes, segments
    that are no multiple of four."""
    case = random_case(nx=nx, ny=ny, nt=nt, S=S, stride=stride, mode=mode, record=record, nrec=nrec, src_comp=nx % 2)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, ckpt_k)
    assert used == E.PATH_TILED
    bx, by, bg, _ = run(case, wx, wy, E.PATH_STEP, ckpt_k)
    assert np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert rel(ag, bg) <= 1e-5, rel(ag, bg)


def test_run_in_a_captured_graph_and_on_two_streams():
    """A run replayed from a graph, and two at once on two streams (together
    more tiles than SMs), give the results of a plain call."""
    cases = [random_case(nx=nx, ny=241, nt=130, S=1, record=O.RECORD_RECEIVERS, nrec=30) for nx in (301, 290)]
    want, calls = [], []
    for c in cases:
        geom = to_geometry(c, path=E.PATH_AUTO)
        C = torch.tensor(c.C, dtype=torch.float32, device=DEV)
        r = torch.tensor(c.rho, dtype=torch.float32, device=DEV)
        calls.append(lambda C=C, r=r, geom=geom: E.propagate(C, r, geom))
        with torch.no_grad():
            want.append([v.clone() for v in calls[-1]()])
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    with torch.no_grad():
        for _ in range(3):
            got = []
            for st, call in zip(streams, calls):
                with torch.cuda.stream(st):
                    got.append(call())
            torch.cuda.synchronize()
            for g, w in zip(got, want):
                assert torch.equal(g[0], w[0]) and torch.equal(g[1], w[1])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = calls[0]()
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], want[0][0]) and torch.equal(out[1], want[0][1])


def test_autotune_measures_the_kernels_that_no_path_names():
    from ernn_gb300 import autotune
    case = random_case(nx=90, ny=243, nt=120, S=1, record=O.RECORD_RECEIVERS, nrec=8)
    geom = to_geometry(case, None, E.PATH_AUTO)
    C = torch.tensor(case.C, dtype=torch.float32, device=DEV)
    rho = torch.tensor(case.rho, dtype=torch.float32, device=DEV)
    path, k, rows = autotune.tune(geom, C, rho, probe_steps=96)  # ny % 4 != 0: neither RESIDENT nor TILED
    assert path in (E.PATH_AUTO, E.PATH_STEP) and 1 <= k <= case.nt and rows == 16


def test_large_odd_grid_vs_fp64_oracle():
    case = random_case(nx=330, ny=437, nt=60, S=5, record=O.RECORD_RECEIVERS, nrec=60)
    wx, wy = weights(case)
    ax, ay, ag, used = run(case, wx, wy, E.PATH_AUTO, 9)
    assert used == E.PATH_TILED
    ox, oy, og = run_oracle(case, wx, wy)
    assert rel(ax, ox) <= 1e-5 and rel(ay, oy) <= 1e-5
    assert rel(ag, og) <= GRAD_TOL, rel(ag, og)
