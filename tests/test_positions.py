"""Positions in every form that torch.as_tensor takes, through the one copy that host
positions travel in: each gives the same cells (whole numbers: equal)."""
import numpy as np
import pytest
import torch

CELLS = [[20, 31], [9, 44], [12, 12]]


def _forms():
    a = np.array(CELLS)
    return {
        "list": CELLS,
        "tuples": tuple(map(tuple, CELLS)),
        "int64": a,
        "uint8": a.astype(np.uint8),
        "strided": np.asfortranarray(a)[:, :],
        "float": a + 0.75,
        "tensor": torch.tensor(CELLS),
        "bf16 tensor": torch.tensor(CELLS, dtype=torch.bfloat16),
        "tensor with grad": torch.tensor(CELLS, dtype=torch.float64, requires_grad=True),
        "scalars": [[torch.tensor(v) for v in c] for c in CELLS],
        "arrays": list(a),
    }


@pytest.mark.parametrize("form", _forms())
def test_host_positions(form):
    from neuralmech_gb300.wavefd import _as_positions, _host_positions, _positions, _to_device
    pos = _as_positions(_forms()[form])
    none = np.zeros((0, 2), np.int32)
    host = [_host_positions(pos, 2, 2), _host_positions(none, 2, 2), None, np.ones(5, np.float32)]
    got, empty, nothing, ones = _to_device(host, "cpu")
    assert torch.equal(got, _positions(torch.tensor(CELLS), 2, 2, "cpu"))
    assert got.dtype == torch.int32 and got.is_contiguous()
    assert empty.shape == (2, 0, 3) and nothing is None and torch.equal(ones, torch.ones(5))


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["device scalars", "device tensor", "device array"])
def test_device_positions(cuda, form):
    from neuralmech_gb300.wavefd import Grid, _prepare

    class Foreign:  # a device array of another library
        def __init__(self, t):
            self.t, self.__cuda_array_interface__ = t, t.__cuda_array_interface__

    t = torch.tensor(CELLS, device=cuda)
    pos = {"device scalars": [[torch.tensor(v, device=cuda) for v in c] for c in CELLS], "device tensor": t,
           "device array": Foreign(t)}[form]
    grid = Grid((40, 60), (10.0, 10.0), 1e-3, 10)
    c = _prepare(torch.full((40, 60), 1500.0, device=cuda), np.zeros(10), pos, CELLS, grid)
    assert c.src.device == c.rec.device == c.vel.device
    assert torch.equal(c.src, c.rec) and c.src[0, :, 0].tolist() == [20, 9, 12] and c.src[0, :, 2].tolist() == [31, 44, 12]


@pytest.mark.parametrize("sponge", [0, 3])
def test_no_points_at_all(sponge):
    """Neither sources nor receivers, with and without a sponge: the one copy may hold nothing."""
    from neuralmech_gb300.wavefd import Grid, _host_positions, _to_device, sponge_profiles
    none = _host_positions(np.zeros((2, 0, 2), np.int32), 2, 2)
    profiles = sponge_profiles(Grid((40, 60), (10.0, 10.0), 1e-3, 10, sponge=sponge))
    src, rec, gz, gy, gx = _to_device([none, none, *profiles], "cpu")
    assert src.shape == rec.shape == (2, 0, 3) and src.dtype == torch.int32 and gy is None
    assert (gz is None and gx is None) if sponge == 0 else (gz.shape == (40,) and gx.shape == (60,))


@pytest.mark.gpu
def test_no_points_in_a_call(cuda):
    from neuralmech_gb300.wavefd import Grid, misfit_gradient, wave_forward
    grid = Grid((40, 60), (10.0, 10.0), 1e-3, 10, sponge=0)
    vel = torch.full((40, 60), 1500.0, device=cuda)
    none, wav = np.zeros((2, 0, 2), np.int32), torch.zeros((2, 10, 0), device=cuda)
    assert wave_forward(vel, wav, none, none, grid).shape == (2, 10, 0)
    J, g = misfit_gradient(vel, wav, none, none, torch.zeros((2, 10, 0), device=cuda), grid)
    assert float(J) == 0 and not bool(g.any())
