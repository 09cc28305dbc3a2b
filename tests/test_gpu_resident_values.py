"""The small grids' brick kernel against the tiles, bit for bit, where a value or a
buffer is out of the ordinary: infinities, NaN, -0, denormals and huge numbers;
occupancy at any address."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (32, 20, 17)


def tiles(marl, field, occ, p, substeps):
    """The same substeps one call each, which the brick kernel does not take."""
    import torch

    f, o = torch.from_numpy(field.copy()).cuda(), torch.from_numpy(occ).cuda()
    s = torch.empty_like(f)
    for _ in range(substeps):
        marl.diffuse_device(f.data_ptr(), s.data_ptr(), o.data_ptr(), DIMS, p, 1)
    return f.cpu().numpy()


@pytest.mark.parametrize("kind", ["nan", "inf", "-inf", "minus_zero", "denormal", "huge", "negative"])
def test_values(marl, kind):
    import torch

    rng = np.random.default_rng(4)
    field = rng.random((*DIMS[::-1], 12), dtype=np.float32) * np.float32(2)
    some = rng.random(field.shape) < 0.002
    if kind in ("nan", "inf", "-inf"):
        field[some] = np.float32(kind)
    elif kind == "minus_zero":
        field[rng.random(field.shape) < 0.6] = np.float32(-0.0)
    elif kind == "denormal":
        field *= np.float32(1e-39)
    elif kind == "huge":
        field[some] = np.float32(3e38)
    else:
        field -= np.float32(1)
    occ = (rng.random(DIMS[::-1]) < 0.15).astype(np.uint8)
    p = marl.default_params()
    want = tiles(marl, field, occ, p, 10)
    f, o = torch.from_numpy(field.copy()).cuda(), torch.from_numpy(occ).cuda()
    s = torch.empty_like(f)
    marl.diffuse_device(f.data_ptr(), s.data_ptr(), o.data_ptr(), DIMS, p, 10)
    np.testing.assert_array_equal(f.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("substeps", [3, 10])  # tiles; bricks
@pytest.mark.parametrize("offset", [0, 1, 8, 16])
def test_occupancy_at_any_address(marl, oracle_mod, substeps, offset):
    import torch

    rng = np.random.default_rng(6)
    field = rng.random((*DIMS[::-1], 12), dtype=np.float32)
    occ = (rng.random(DIMS[::-1]) < 0.2).astype(np.uint8)
    p = marl.default_params()
    cpu = field.copy()
    oracle_mod.diffuse(cpu, occ, DIMS, p, substeps)
    store = torch.full((occ.size + 64,), 1, dtype=torch.uint8, device="cuda")
    o = store[offset:offset + occ.size]
    o.copy_(torch.from_numpy(occ).reshape(-1))
    f = torch.from_numpy(field).cuda()
    s = torch.empty_like(f)
    marl.diffuse_device(f.data_ptr(), s.data_ptr(), o.data_ptr(), DIMS, p, substeps)
    np.testing.assert_array_equal(f.cpu().numpy(), cpu)
