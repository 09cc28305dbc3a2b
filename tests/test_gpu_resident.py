"""Small grids of the device-pointer diffusion calls, where all substeps are one
kernel of bricks that exchange their surfaces: bit-identical to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def call(marl, entry, field, occ, dims, p, substeps):
    import torch

    f, o = torch.from_numpy(field.copy()).cuda(), torch.from_numpy(occ).cuda()
    if entry == "noalloc":
        marl.diffuse_device_noalloc(f.data_ptr(), o.data_ptr(), dims, p, substeps)
    else:
        s = torch.full_like(f, float("nan"))
        marl.diffuse_device(f.data_ptr(), s.data_ptr(), o.data_ptr(), dims, p, substeps)
    return f.cpu().numpy()


# One voxel; a line; a plane; grids of one brick and of many, with ragged last
# bricks; either side of the size limit.
@pytest.mark.parametrize("entry", ["device", "noalloc"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (300, 1, 1), (1, 1, 149), (23, 1, 40), (3, 5, 2), (37, 21, 13), (16, 16, 3),
                                  (130, 7, 40), (40, 40, 25), (41, 40, 25)])
def test_small_grids(marl, oracle_mod, entry, dims):
    rng = np.random.default_rng(sum(dims))
    shape = dims[::-1]
    field = rng.random((*shape, 12), dtype=np.float32) * np.float32(2)
    occ = (rng.random(shape) < 0.15).astype(np.uint8) * np.uint8(255)  # any non-zero byte is occupied
    p = marl.default_params()
    for substeps in (4, 5, 6, 10):  # from five on in one kernel
        cpu = field.copy()
        oracle_mod.diffuse(cpu, (occ != 0).astype(np.uint8), dims, p, substeps)
        np.testing.assert_array_equal(call(marl, entry, field, occ, dims, p, substeps), cpu, err_msg=str(substeps))


@pytest.mark.parametrize("pattern", ["full", "slabs", "checker"])
def test_occupied_faces(marl, oracle_mod, pattern):
    """Bricks whose shared faces are occupied wholly, or at every other voxel."""
    dims = (36, 24, 20)
    z, y, x = np.meshgrid(*(np.arange(n) for n in dims[::-1]), indexing="ij")
    occ = {"full": np.ones_like(x), "slabs": (x % 3 == 0) | (z % 5 == 4), "checker": (x + y + z) % 2}[pattern]
    occ = occ.astype(np.uint8)
    field = np.random.default_rng(7).random((*dims[::-1], 12), dtype=np.float32)
    p = marl.default_params()
    cpu = field.copy()
    oracle_mod.diffuse(cpu, occ, dims, p, 7)
    for _ in range(20):  # the bricks meet in another order each time
        np.testing.assert_array_equal(call(marl, "device", field, occ, dims, p, 7), cpu)
