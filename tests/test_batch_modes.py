"""A batch of several models takes the same kernels as a graph and as eager calls: shots
per CTA from the whole batch's work, by the library's rule; a batch of one takes what a
call of its own takes."""
import ctypes
import random

import numpy as np
import pytest
import torch

from conftest import rel_l2
from helpers import small_problem


def test_shots_per_cta_is_the_librarys_rule():
    from neuralmech_gb300 import _lib
    from neuralmech_gb300.batch import _auto_spc
    rule = _lib.load()["_ZN3wfd8auto_spcEiid"]  # wfd::auto_spc(int, int, double)
    rule.argtypes, rule.restype = [ctypes.c_int, ctypes.c_int, ctypes.c_double], ctypes.c_int
    rng = random.Random(3)
    for _ in range(2000):
        args = rng.randint(1, 2000), int(2 ** rng.uniform(0, 12)), 2 ** rng.uniform(0, 5)
        assert _auto_spc(*args) == rule(*args), args


def test_only_batches_without_a_tiling_are_given_one():
    from neuralmech_gb300 import Grid
    from neuralmech_gb300.batch import _batch_grids
    g = Grid((400, 700), (10.0, 10.0), 1e-3, 50)
    tiled = Grid((400, 700), (10.0, 10.0), 1e-3, 50, tile_rows=16)
    deep = Grid((40, 40, 70), (10.0,) * 3, 1e-3, 50)
    assert _batch_grids([g], [5]) == [g]
    out = _batch_grids([g, tiled, deep, g], [5, 5, 5, 20])
    assert out[1:3] == [tiled, deep] and 1 < out[0].shots_per_cta <= 5 and 1 < out[3].shots_per_cta <= 20


def _models(cuda, specs):
    out = []
    for k, sp in enumerate(specs):
        grid, v, wav, src, rec = small_problem(seed=k, **sp)
        obs = 1e-3 * np.random.default_rng(k).standard_normal((src.shape[0], grid.nt, rec.shape[1]))
        out.append(dict(vel=torch.from_numpy(v).to(cuda), wavelet=torch.from_numpy(wav).to(cuda), src=src, rec=rec,
                        observed=torch.from_numpy(obs.astype(np.float32)).to(cuda), grid=grid))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("specs", [
    [dict(shape=(64, 200), nshot=3, nt=60), dict(shape=(48, 140), nshot=7, nt=45, order=4, step_block=2),
     dict(shape=(90, 260), nshot=4, nt=50)],
    [dict(shape=(75, 210), nshot=3, nt=60)],  # one model: the resident kernel, in a graph too
], ids=["three", "one"])
def test_graph_and_eager(cuda, specs):
    from neuralmech_gb300 import _lib, misfit_gradient
    from neuralmech_gb300.batch import BatchFWI
    models = _models(cuda, specs)
    graph, eager = BatchFWI(models, autotune=False), BatchFWI(models, autotune=False, graph=False)
    assert graph.configs == eager.configs
    assert all((c[1] > 0) == (len(models) > 1) for c in graph.configs)
    n0 = int(_lib.load().wfd_kernel_launches())
    runs = [graph.run(), eager.run()]
    torch.cuda.synchronize()
    n = int(_lib.load().wfd_kernel_launches()) - n0
    assert n == 2 * graph.graph_kernels  # the same launches
    assert (graph.graph_kernels < models[0]["grid"].nt) == (len(models) == 1)  # resident or streaming
    for _ in range(2):
        runs.append(graph.run())  # (its outputs are the batch's own: replays write them again)
    for J, grads in runs:
        for i, m in enumerate(models):
            ref = misfit_gradient(m["vel"], m["wavelet"], m["src"], m["rec"], m["observed"], graph.models[i].call.grid)
            assert abs(J[i].item() / ref[0].item() - 1) <= 1e-9
            assert rel_l2(grads[i].cpu().numpy(), ref[1].cpu().numpy()) < 1e-6
