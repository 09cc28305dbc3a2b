"""The device-pointer diffusion on a stream that has only some of the SMs (a green
context's): it cannot hold the small grids' cooperative launch, so the tiles run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (37, 21, 13)


def ok(r):
    assert int(r[0]) == 0, r
    return r[1] if len(r) == 2 else r[1:]


@pytest.fixture
def partial():
    """(context, stream) with 16 SMs, and the context that was current before."""
    cu = pytest.importorskip("cuda.bindings.driver")
    import torch

    torch.zeros(1, device="cuda")
    before = ok(cu.cuCtxGetCurrent())
    dev = ok(cu.cuDeviceGet(0))
    sms = ok(cu.cuDeviceGetDevResource(dev, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(cu.cuDevSmResourceSplitByCount(1, sms, 0, 16))
    assert 8 <= groups[0].sm.smCount <= 32
    green = ok(cu.cuGreenCtxCreate(ok(cu.cuDevResourceGenerateDesc(groups, 1)), dev,
                                   int(cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM)))
    stream = ok(cu.cuGreenCtxStreamCreate(green, int(cu.CUstream_flags.CU_STREAM_NON_BLOCKING), 0))
    yield cu, before, ok(cu.cuCtxFromGreenCtx(green)), int(stream)
    ok(cu.cuCtxSetCurrent(before))
    cu.cuStreamDestroy(stream)
    cu.cuGreenCtxDestroy(green)


@pytest.mark.parametrize("entry", ["device", "noalloc"])
def test_falls_back_to_tiles(marl, oracle_mod, partial, entry):
    import torch

    cu, before, green, stream = partial
    rng = np.random.default_rng(2)
    field = rng.random((*DIMS[::-1], 12), dtype=np.float32)
    occ = (rng.random(DIMS[::-1]) < 0.15).astype(np.uint8)
    p = marl.default_params()
    cpu = field.copy()
    oracle_mod.diffuse(cpu, occ, DIMS, p, 10)
    o = torch.from_numpy(occ).cuda()
    # The small stream and the whole device in turn, the stream's own context current or not.
    for context, s in ((before, 0), (before, stream), (green, stream), (before, 0), (green, stream), (before, 0)):
        f = torch.from_numpy(field.copy()).cuda()
        scratch = torch.empty_like(f)
        torch.cuda.synchronize()
        ok(cu.cuCtxSetCurrent(context))
        try:
            if entry == "noalloc":
                marl.diffuse_device_noalloc(f.data_ptr(), o.data_ptr(), DIMS, p, 10, s)
            else:
                marl.diffuse_device(f.data_ptr(), scratch.data_ptr(), o.data_ptr(), DIMS, p, 10, s)
        finally:
            ok(cu.cuCtxSetCurrent(before))
        np.testing.assert_array_equal(f.cpu().numpy(), cpu)
