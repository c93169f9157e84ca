"""Updates and snapshots of user tensors that start anywhere in their storage, at sizes around the kernels' tiles."""
import pytest
import torch

from sharedtensor_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 4095, 4096, 4097, 4099, 3 * 4096 + 1, 1_300_007])
def test_slices(n, offset):
    cu = _native.cuda()
    s = torch.cuda.current_stream().cuda_stream
    torch.manual_seed(n + offset)
    rep = cu.GpuReplica(0, n, cu.GpuConfig())
    expect = torch.randn(n, device="cuda")
    rep.load_values(expect.data_ptr(), s)

    def piece(dtype=torch.float32, at=offset):
        return torch.randn(n + at, device="cuda").to(dtype)[at:]

    d, new, old, g = piece(), piece(), piece(at=(offset + 1) % 4), piece(torch.bfloat16)
    rep.add(d.data_ptr(), s)
    rep.sub_add(new.data_ptr(), old.data_ptr(), s)
    rep.add_scaled_bf16(g.data_ptr(), -0.5, s)
    expect = ((expect + d) + (new - old)) + (-0.5) * g.float()
    for dtype, snap in ((torch.float32, rep.snapshot), (torch.bfloat16, rep.snapshot_bf16)):
        store = torch.full((n + offset + 4,), 7.0, device="cuda", dtype=dtype)
        snap(store[offset:].data_ptr(), s)
        torch.cuda.synchronize()
        assert torch.equal(store[offset:offset + n], expect.to(dtype))
        assert (store[:offset] == 7).all() and (store[offset + n:] == 7).all()
    assert rep.check_guards() == 0
