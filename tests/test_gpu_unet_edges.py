"""The tensor-core kernels of the denoiser at the edges of their tiles:
columns of 16 (y) x 8 (x) voxels cut by the volume, rings shorter and longer
than a segment, channel groups of 16 and 32, against FP64 references."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def U():
    from chatcarlo_b200 import _unet_native
    return _unet_native


def _taps(x):
    """(tap, x shifted by it with zero padding) of x [B, D, H, W, C]."""
    d, h, w = x.shape[1:4]
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    for t in range(27):
        z, y, c = t // 9, t // 3 % 3, t % 3
        yield t, p[:, z:z + d, y:y + h, c:c + w]


@pytest.mark.parametrize("ca,cout,dims,slices", [
    (16, 16, (1, 1, 1, 1), 1),              # one voxel: 26 taps see only padding
    (16, 16, (2, 3, 17, 9), 1),             # one row and one column beyond a tile
    (16, 32, (1, 5, 16, 8), 64),            # exactly one column, more splits than planes
    (32, 16, (1, 2, 33, 7), 3),             # three y tiles, x narrower than a tile
    (32, 64, (3, 4, 15, 23), 5),            # two output groups
    (48, 32, (1, 19, 10, 12), 2),           # three groups of 16 input channels, ring wraps inside a segment
    (128, 128, (1, 2, 8, 9), 1),            # 4 x 4 channel-group pairs
])
def test_weight_gradient_halo_planes(U, ca, cout, dims, slices):
    """Every product is exact in FP32 and every one of the at most n additions
    into an accumulator or into dw errs by at most 2^-23 of the running sum,
    so |dw - exact| <= n 2^-23 sum |dz x|."""
    g = torch.Generator(device="cuda").manual_seed(ca + cout + dims[2])
    n = dims[0] * dims[1] * dims[2] * dims[3]
    x = torch.randn(*dims, ca, generator=g, device="cuda").relu().to(torch.bfloat16)
    dz = torch.randn(*dims, cout, generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.zeros(27, cout, ca, device="cuda")
    U.check(U.lib().ccu_conv3d_wgrad(x.data_ptr(), ca, None, 0, *dims, dz.data_ptr(), cout, dw.data_ptr(), slices,
                                     torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert U.status() == 0
    z = dz.double().reshape(n, cout)
    for t, v in _taps(x.double()):
        v = v.reshape(n, ca)
        bound = (n + 1) * 2.0 ** -23 * (z.abs().T @ v.abs())
        assert bool(((dw[t].double() - z.T @ v).abs() <= bound).all()), t
