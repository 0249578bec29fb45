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


@pytest.mark.parametrize("cin,cout,split,dims", [
    (16, 48, 16, (1, 3, 17, 9)),            # slices of 32 and 16, the output split inside the first
    (32, 96, 32, (2, 2, 16, 8)),            # three slices of 32
    (64, 192, 64, (1, 5, 7, 11)),           # six slices of 32
    (64, 128, 128, (1, 1, 1, 1)),           # four slices, one voxel
    (128, 128, 128, (2, 4, 9, 17)),         # eight slices of 16, a ring of two planes
    (128, 96, 40, (1, 3, 16, 16)),          # six slices of 16, split inside a slice
])
@pytest.mark.parametrize("masked", [False, True])
def test_convolution_output_slices(U, cin, cout, split, dims, masked):
    """Sums of 27 cin products, exact in FP32, err by at most 2^-23 of the sum
    of their magnitudes per addition; the BF16 store rounds once (2^-8)."""
    g = torch.Generator(device="cuda").manual_seed(cin + cout + dims[2])
    n = dims[0] * dims[1] * dims[2] * dims[3]
    x = torch.randn(*dims, cin, generator=g, device="cuda").to(torch.bfloat16)
    w32 = torch.randn(27, cout, cin, generator=g, device="cuda") * 0.05
    w = torch.empty(U.lib().ccu_packed_weight_elems(cout, cin), dtype=torch.bfloat16, device="cuda")
    bias = torch.randn(cout, generator=g, device="cuda")
    mask = torch.randn(n, split, generator=g, device="cuda").to(torch.bfloat16)
    out0 = torch.empty(n, split, dtype=torch.bfloat16, device="cuda")
    out1 = torch.empty(n, max(cout - split, 8), dtype=torch.bfloat16, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    U.check(U.lib().ccu_pack_weights(w32.data_ptr(), cout, cin, w.data_ptr(), None, st))
    U.check(U.lib().ccu_conv3d(x.data_ptr(), cin, None, 0, *dims, w.data_ptr(), bias.data_ptr(), cout, 0,
                               out0.data_ptr(), split, mask.data_ptr() if masked else None,
                               out1.data_ptr() if split < cout else None, st))
    torch.cuda.synchronize()
    assert U.status() == 0
    wd = w32.to(torch.bfloat16).double()
    ref = bias.double().expand(n, cout).clone()
    mag = ref.abs()
    for t, v in _taps(x.double()):
        v = v.reshape(n, cin)
        ref += v @ wd[t].T
        mag += v.abs() @ wd[t].abs().T
    if masked:
        ref[:, :split] *= mask > 0
    got = torch.cat([out0, out1], 1)[:, :cout].double() if split < cout else out0.double()
    assert bool(((got - ref).abs() <= 2.0 ** -8 * ref.abs() + (27 * cin + 4) * 2.0 ** -23 * mag).all())


@pytest.mark.parametrize("c,n,offset", [(1, 1000, 0), (4, 77, 0), (8, 1, 0), (16, 4097, 0), (64, 333, 0), (256, 50, 0),
                                        (16, 4097, 1)])           # offset 1: dz is not 16-byte aligned
def test_bias_gradient_widths(U, c, n, offset):
    """Every one of at most n additions errs by at most 2^-24 of the running sum of magnitudes."""
    g = torch.Generator(device="cuda").manual_seed(c + n)
    buf = torch.randn(n * c + offset, generator=g, device="cuda").to(torch.bfloat16)
    dz = buf[offset:].view(n, c)
    db = torch.ones(c, device="cuda")
    U.check(U.lib().ccu_bias_grad(dz.data_ptr(), n, c, db.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    ref, mag = 1.0 + dz.double().sum(0), 1.0 + dz.double().abs().sum(0)
    assert bool(((db.double() - ref).abs() <= (n + 1) * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("ca,cb,dims", [
    (32, 0, (1, 1, 1, 16)), (32, 0, (2, 90, 37, 94)), (32, 0, (1, 3000, 1, 16)), (48, 0, (2, 62, 37, 94)),
    (48, 0, (1, 380, 33, 30)), (16, 32, (2, 62, 38, 94)), (32, 16, (1, 380, 34, 32)), (48, 0, (1, 600, 33, 24)),
])
def test_sixteen_channels_on_pairs_of_voxels(U, ca, cb, dims):
    """The kernel on pairs sums the same products in the same order as the one
    without (an issue group set by hand keeps it off), so the values are equal."""
    g = torch.Generator(device="cuda").manual_seed(ca + cb + dims[3])
    n = dims[0] * dims[1] * dims[2] * dims[3]
    a = torch.randn(n, ca, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(n // 8, cb, generator=g, device="cuda").to(torch.bfloat16) if cb else None
    w32 = torch.randn(27, 16, ca + cb, generator=g, device="cuda") * 0.1
    w = torch.empty(U.lib().ccu_packed_weight_elems(16, ca + cb), dtype=torch.bfloat16, device="cuda")
    bias = torch.randn(16, generator=g, device="cuda")
    mask = torch.randn(n, 16, generator=g, device="cuda").to(torch.bfloat16)
    head, x = torch.randn(17, generator=g, device="cuda"), torch.randn(n, generator=g, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    U.check(U.lib().ccu_pack_weights(w32.data_ptr(), 16, ca + cb, w.data_ptr(), None, st))
    got = []
    try:
        for group in (0, 1):
            U.check(U.lib().ccu_set_conv_group(group))
            outs = []
            for m, relu in ((None, 1), (mask.data_ptr(), 0)):
                o = torch.empty(n, 16, dtype=torch.bfloat16, device="cuda")
                U.check(U.lib().ccu_conv3d(a.data_ptr(), ca, b.data_ptr() if cb else None, cb, *dims, w.data_ptr(),
                                           bias.data_ptr(), 16, relu, o.data_ptr(), 16, m, None, st))
                outs.append(o)
            if cb == 0:
                h = torch.empty(n, device="cuda")
                U.check(U.lib().ccu_conv3d_head(a.data_ptr(), ca, *dims, w.data_ptr(), bias.data_ptr(), head.data_ptr(),
                                                x.data_ptr(), h.data_ptr(), None, 0, st))
                outs.append(h)
            got.append(outs)
    finally:
        U.check(U.lib().ccu_set_conv_group(0))
    torch.cuda.synchronize()
    assert U.status() == 0
    for p, q in zip(*got):
        assert torch.equal(p, q)


@pytest.mark.parametrize("ca,cb,cout,dims,slices,path", [
    (16, 0, 16, (1, 1, 1, 1), 1, 0),            # one voxel
    (16, 0, 16, (2, 3, 17, 9), 1, 0),           # one row and one column beyond a tile
    (32, 0, 128, (1, 5, 16, 8), 64, 0),         # four output groups, more splits than planes
    (64, 0, 32, (3, 19, 33, 7), 2, 0),          # two input groups: the first alone sums; the ring wraps
    (32, 64, 16, (1, 4, 18, 16), 3, 0),         # concatenated: the first part's launch alone sums
    (16, 32, 64, (1, 2, 6, 10), 2, 0),          # concatenated, gathering kernel
    (16, 0, 32, (2, 4, 9, 11), 4, 1),           # gathering kernel by choice
])
def test_bias_gradient_beside_the_weight_gradient(U, ca, cb, cout, dims, slices, path):
    """At most n additions of exactly converted values in FP32, each erring by
    at most 2^-24 of the sum of the magnitudes."""
    g = torch.Generator(device="cuda").manual_seed(ca + cout + dims[2])
    n = dims[0] * dims[1] * dims[2] * dims[3]
    a = torch.randn(n, ca, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(max(1, n // 8), max(1, cb), generator=g, device="cuda").to(torch.bfloat16)
    dz = torch.randn(n, cout, generator=g, device="cuda").to(torch.bfloat16)
    dw, db = torch.zeros(27, cout, ca + cb, device="cuda"), torch.ones(cout, device="cuda")
    try:
        U.check(U.lib().ccu_set_wgrad_path(path))
        U.check(U.lib().ccu_conv3d_wgrad_bias(a.data_ptr(), ca, b.data_ptr() if cb else None, cb, *dims, dz.data_ptr(), cout,
                                              dw.data_ptr(), db.data_ptr(), slices, torch.cuda.current_stream().cuda_stream))
    finally:
        U.check(U.lib().ccu_set_wgrad_path(0))
    torch.cuda.synchronize()
    assert U.status() == 0
    ref, mag = 1.0 + dz.double().sum(0), 1.0 + dz.double().abs().sum(0)
    assert bool(((db.double() - ref).abs() <= (n + 1) * 2.0 ** -24 * mag).all())
    assert bool((dw.abs().sum((0, 2)) > 0).all())


@pytest.mark.parametrize("cin,cout,split,dims", [
    (80, 16, 16, (2, 300, 17, 9)),          # 16 planes per CTA: the ring turns several times
    (80, 48, 16, (1, 310, 18, 21)),
    (112, 128, 128, (1, 150, 33, 7)),
    (144, 16, 16, (1, 300, 20, 10)),        # two passes of 80 and 64 input channels
    (112, 48, 40, (1, 3, 5, 6)),
])
@pytest.mark.parametrize("masked", [False, True])
def test_convolution_on_rings_that_five_planes_would_fit(U, cin, cout, split, dims, masked):
    """Passes of 80 and 112 input channels, whose deepest ring (5 or 3 planes)
    two issuing warps may not use."""
    test_convolution_output_slices(U, cin, cout, split, dims, masked)


@pytest.mark.parametrize("ca,cb,cout,dims", [
    (16, 0, 16, (2, 5, 17, 9)),             # a row and a column of a tile's padding beside real voxels
    (32, 0, 64, (1, 33, 16, 8)),            # whole tiles: only the planes -1 and D are padding
    (16, 0, 32, (1, 1, 3, 5)),
    (32, 64, 16, (1, 4, 18, 16)),           # concatenated
    (16, 0, 16, (1, 2, 160, 237)),          # 300 columns: whole ones per CTA, and some left over
])
@pytest.mark.parametrize("where", ["x", "dz", "both"])
def test_weight_gradient_of_infinities_and_nan(U, ca, cb, cout, dims, where):
    """An infinity reaches the taps and channels whose sums contain it, and no
    others; what stays finite is within the bound of the finite test."""
    g = torch.Generator(device="cuda").manual_seed(ca + cout + dims[1])
    n = dims[0] * dims[1] * dims[2] * dims[3]
    coarse = (dims[0], *(s // 2 for s in dims[1:]))
    x = torch.rand(*dims, ca, generator=g, device="cuda").add(0.5).to(torch.bfloat16)
    b = torch.rand(*(coarse if cb else (1, 1, 1, 1)), max(cb, 1), generator=g, device="cuda").add(0.5).to(torch.bfloat16)
    dz = torch.rand(*dims, cout, generator=g, device="cuda").add(0.5).to(torch.bfloat16)      # no zeros: 0 x inf is a NaN
    if where != "dz":
        x[0, 0, 0, 0, 3], x[-1, -1, -1, -1, 5] = float("inf"), -float("inf")
        x[0, dims[1] // 2, -1, 0, 7] = float("nan")
        b[0, 0, 0, 0, 0] = float("inf")
    if where != "x":
        dz[0, 0, 0, 0, 1], dz[-1, -1, -1, -1, 2] = float("inf"), float("inf")
    dw, db = torch.zeros(27, cout, ca + cb, device="cuda"), torch.zeros(cout, device="cuda")
    U.check(U.lib().ccu_conv3d_wgrad_bias(x.data_ptr(), ca, b.data_ptr() if cb else None, cb, *dims, dz.data_ptr(), cout,
                                          dw.data_ptr(), db.data_ptr(), 2, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert U.status() == 0
    full = x.double()
    if cb:
        up = b.double().repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)
        full = torch.cat([full, up], -1)
    z = dz.double().reshape(n, cout)
    finite = lambda t: torch.nan_to_num(t, nan=0.0, posinf=0.0, neginf=0.0)  # noqa: E731
    for t, v in _taps(full):
        v = v.reshape(n, ca + cb)
        ref = torch.stack([(z[:, c, None] * v).sum(0) for c in range(cout)])
        assert torch.equal(torch.isnan(dw[t]), torch.isnan(ref)), t
        inf = torch.isinf(ref)
        assert torch.equal(torch.isinf(dw[t]), inf) and torch.equal(dw[t][inf].sign().double(), ref[inf].sign()), t
        keep = torch.isfinite(ref)
        bound = (n + 1) * 2.0 ** -23 * (finite(z).abs().T @ finite(v).abs())
        assert bool(((dw[t].double() - ref).abs() <= bound)[keep].all()), t
    assert torch.equal(torch.isinf(db), torch.isinf(z.sum(0)))


@pytest.mark.parametrize("ca,cout,planes", [
    (16, 32, 74), (16, 32, 75),             # 2 groups of 16 output channels x planes: 148 SMs, and beyond
    (32, 128, 18), (32, 128, 19),           # 8 groups
    (64, 64, 18), (64, 64, 300),            # 2 groups of input channels x 4
])
def test_weight_gradient_on_both_sides_of_the_group_rule(U, ca, cout, planes):
    """Groups of 16 and of 32 output channels, at the line between them."""
    test_weight_gradient_halo_planes(U, ca, cout, (1, planes, 13, 7), 1)
    test_bias_gradient_beside_the_weight_gradient(U, ca, 0, cout, (1, planes, 13, 7), 1, 0)
    test_weight_gradient_of_infinities_and_nan(U, ca, 0, cout, (1, planes, 13, 7), "both")


def _on_pairs(cin, dims):
    """Whether a slice of 16 output channels runs on pairs of voxels: an even
    width, 32 or 48 input channels, little padding and enough planes per SM."""
    b, d, h, w = dims
    planes = b * d * -(-h // 16) * -(-w // 16)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return w % 2 == 0 and cin in (32, 48) and -(-w // 16) * 16 * 5 <= -(-w // 8) * 8 * 6 and planes >= sms * (10 if cin == 48 else 20)


@pytest.mark.parametrize("cin,cout,split,dims,pairs", [
    (32, 16, 16, (2, 250, 33, 30), True),   # ragged in y and x
    (48, 16, 8, (1, 380, 31, 32), True),    # the split between the two halves of a voxel
    (32, 48, 16, (2, 250, 33, 30), True),   # the last 16 of 48 channels, all of them in the second output
    (48, 48, 40, (1, 380, 31, 32), True),   # the split inside that slice
    (48, 48, 16, (1, 600, 33, 24), False),  # 24 voxels would pad to 32
    (32, 48, 40, (2, 250, 33, 31), False),  # an odd width
    (32, 16, 16, (1, 900, 17, 16), False),  # 1800 planes: too few
])
@pytest.mark.parametrize("masked", [False, True])
def test_pairs_of_voxels_against_fp64(U, cin, cout, split, dims, pairs, masked):
    """The slices on pairs of voxels, and their neighbours that run without,
    against the sums in FP64."""
    assert _on_pairs(cin, dims) == pairs
    test_convolution_output_slices(U, cin, cout, split, dims, masked)
