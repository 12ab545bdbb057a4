"""GPU kernels of the warm-start surrogate against CPU references.

Each tcgen05 convolution (forward, input gradient through the packed
flipped weights, weight gradient), the pooling / upsampling kernels and their
backward, the head and loss, and Adam are checked against torch's CPU
operators on the same bf16-rounded inputs; then the whole U-Net's output,
loss and every parameter gradient against oracle/unet_ref.py, which rounds to
bf16 at the same points as the GPU path.

Tolerances: a bf16 output differs from the fp32 reference by its rounding
(relative 2^-8) plus fp32 summation order, so bf16 outputs are held to
1e-2 of the tensor's largest magnitude elementwise; fp32 outputs (weight and
bias gradients, head) to 1e-4 relative L2.  Whole-network gradients go
through ten bf16 roundings of activations and gradients: bf16 alone moves
them 1-9 % (relative L2 per tensor) from the exact fp64 gradient; the
emulating reference reproduces most of that, and the GPU's distance to it
must stay below 0.75 of that bf16 effect per tensor, with a cosine
similarity of the whole gradient of at least 0.999.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from master_b200 import capi
from master_b200 import surrogate as sgm

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def lib():
    return capi.load()


def P(t):
    return C.c_void_p(t.data_ptr()) if t is not None else C.c_void_p(0)


def stream():
    return C.c_void_p(torch.cuda.current_stream(DEV).cuda_stream)


def rnd_bf16(shape, gen, scale=1.0):
    return (torch.randn(shape, generator=gen, dtype=torch.float32) * scale).to(torch.bfloat16)


def to_ncdhw(x):
    """(B, S, S, S, C) -> (B, C, S, S, S) fp64 on the CPU."""
    return x.detach().cpu().to(torch.float64).permute(0, 4, 1, 2, 3)


def torch_weights(w):
    """(cout, 27, cin) -> conv3d weight (cout, cin, 3, 3, 3)."""
    cout, _, cin = w.shape
    return w.reshape(cout, 3, 3, 3, cin).permute(0, 4, 1, 2, 3)


def ref_conv(x, w, bias=None):
    y = F.conv3d(F.pad(x, (1, 1, 1, 1, 1, 1), mode="circular"), torch_weights(w))
    if bias is not None:
        y = y + bias.view(1, -1, 1, 1, 1)
    return y


def close_bf16(gpu, ref, tol=1e-2):
    g = gpu.detach().cpu().to(torch.float64)
    scale = max(ref.abs().max().item(), 1e-30)
    err = (g - ref).abs().max().item() / scale
    assert err <= tol, f"max error {err:.3e} of scale {scale:.3e}"


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


def sync_ok():
    torch.cuda.synchronize(DEV)
    f = C.c_uint()
    capi.check(lib().dsmc_sg_status(C.byref(f), 1))
    assert f.value == 0, f"surrogate kernel error flags {f.value:#x}"


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (48, 16),
                                      (32, 96), (16, 48)])
def test_conv_forward_matches_torch(cin, cout):
    g = torch.Generator().manual_seed(cin * 100 + cout)
    B, S = 2, 16
    # input as a view into a wider buffer (channel offset 8 of cin + 16)
    buf = rnd_bf16((B, S, S, S, cin + 16), g)
    w = rnd_bf16((cout, 27, cin), g, scale=(2.0 / (27 * cin)) ** 0.5)
    bias = torch.randn(cout, generator=g) * 0.1
    out = torch.zeros((B, S, S, S, cout + 8), dtype=torch.bfloat16)
    d_buf, d_w, d_b, d_out = buf.to(DEV), w.to(DEV), bias.to(DEV), out.to(DEV)
    capi.check(lib().dsmc_sg_conv3(stream(), B, S, P(d_buf), cin + 16, 8, cin, P(d_w), P(d_b), cout, P(d_out),
                                   cout + 8, 8, 1, None, 0, 0))
    sync_ok()
    x = to_ncdhw(buf[..., 8:8 + cin])
    ref = torch.relu(ref_conv(x, w.to(torch.float64), bias.to(torch.float64)))
    close_bf16(to_ncdhw(d_out[..., 8:8 + cout]), ref)
    assert (d_out[..., :8].float() == 0).all()  # channels outside the view untouched


def test_conv_mask_and_no_bias():
    g = torch.Generator().manual_seed(7)
    B, S, cin, cout = 1, 32, 32, 16
    x = rnd_bf16((B, S, S, S, cin), g)
    w = rnd_bf16((cout, 27, cin), g, scale=0.05)
    mask = rnd_bf16((B, S, S, S, cout), g)
    out = torch.zeros((B, S, S, S, cout), dtype=torch.bfloat16, device=DEV)
    dx, dw, dm = x.to(DEV), w.to(DEV), mask.to(DEV)
    capi.check(lib().dsmc_sg_conv3(stream(), B, S, P(dx), cin, 0, cin, P(dw), None, cout, P(out), cout, 0, 0, P(dm),
                                   cout, 0))
    sync_ok()
    ref = ref_conv(to_ncdhw(x), w.to(torch.float64)) * (to_ncdhw(mask) > 0)
    close_bf16(to_ncdhw(out), ref)


@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 64), (96, 32), (48, 16)])
def test_conv_input_gradient_through_packed_weights(cin, cout):
    """dX = conv(dY, w_dgrad): the forward kernel on the weights that
    dsmc_sg_pack_weights flips and transposes, against torch's autograd."""
    g = torch.Generator().manual_seed(cin + cout)
    B, S = 2, 16
    w32 = torch.randn((cout, 27, cin), generator=g) * 0.05
    dy = rnd_bf16((B, S, S, S, cout), g)
    wf = torch.empty(cout * 27 * cin, dtype=torch.int16, device=DEV)
    wd = torch.empty_like(wf)
    capi.check(lib().dsmc_sg_pack_weights(stream(), P(w32.to(DEV)), cout, cin, P(wf), P(wd)))
    dx = torch.zeros((B, S, S, S, cin), dtype=torch.bfloat16, device=DEV)
    capi.check(lib().dsmc_sg_conv3(stream(), B, S, P(dy.to(DEV)), cout, 0, cout, P(wd), None, cin, P(dx), cin, 0, 0,
                                   None, 0, 0))
    sync_ok()
    wb = w32.to(torch.bfloat16).to(torch.float64)
    assert torch.equal(wf.view(torch.bfloat16).cpu().to(torch.float64).reshape(cout, 27, cin), wb)
    x = torch.zeros((B, cin, S, S, S), dtype=torch.float64, requires_grad=True)
    y = ref_conv(x, wb)
    y.backward(to_ncdhw(dy))
    close_bf16(to_ncdhw(dx), x.grad)


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 64), (64, 64), (96, 32), (48, 16)])
def test_conv_weight_gradient_matches_torch(cin, cout):
    g = torch.Generator().manual_seed(3 * cin + cout)
    B, S = 2, 16
    x = rnd_bf16((B, S, S, S, cin), g)
    dy = rnd_bf16((B, S, S, S, cout), g)
    dw = torch.zeros(cout * 27 * cin, dtype=torch.float32, device=DEV)
    db = torch.zeros(cout, dtype=torch.float32, device=DEV)
    dxd, dyd = x.to(DEV), dy.to(DEV)
    capi.check(lib().dsmc_sg_conv3_wgrad(stream(), B, S, P(dyd), cout, 0, cout, P(dxd), cin, 0, cin, P(dw)))
    capi.check(lib().dsmc_sg_bias_grad(stream(), B, S, P(dyd), cout, 0, cout, P(db)))
    sync_ok()
    W = torch.zeros((cout, cin, 3, 3, 3), dtype=torch.float64, requires_grad=True)
    b = torch.zeros(cout, dtype=torch.float64, requires_grad=True)
    y = F.conv3d(F.pad(to_ncdhw(x), (1, 1, 1, 1, 1, 1), mode="circular"), W) + b.view(1, -1, 1, 1, 1)
    y.backward(to_ncdhw(dy))
    ref = W.grad.permute(0, 2, 3, 4, 1).reshape(cout, 27, cin).numpy()
    assert rel_l2(dw.cpu().numpy().reshape(cout, 27, cin), ref) <= 1e-4
    assert rel_l2(db.cpu().numpy(), b.grad.numpy()) <= 1e-4


@pytest.mark.parametrize("B,S,cin,cout", [(1, 16, 16, 16), (3, 16, 96, 96), (1, 16, 64, 48), (1, 32, 48, 64), (3, 32, 16, 96),
                                          (1, 64, 32, 32), (1, 64, 48, 16), (2, 8, 48, 32)])
def test_conv_edges_of_the_plane_kernels(B, S, cin, cout):
    """Forward, masked input gradient and weight gradient at the smallest edge
    of the plane kernels (16: one tile line block, every halo wraps), odd
    batches, several planes per tile, each accumulator ring (16, 32 and 48
    channels per block) past its first lap, and the edge below (8).  bf16 results are held to the rounding of the output
    (2^-8) plus fp32 summation, as the module's other tests."""
    g = torch.Generator().manual_seed(1000 * S + cin + cout)
    x = rnd_bf16((B, S, S, S, cin), g)
    dy = rnd_bf16((B, S, S, S, cout), g)
    w32 = torch.randn((cout, 27, cin), generator=g) * (2.0 / (27 * cin)) ** 0.5
    bias = torch.randn(cout, generator=g) * 0.1
    wf = torch.empty(cout * 27 * cin, dtype=torch.int16, device=DEV)
    wd = torch.empty_like(wf)
    d_w32, d_x, d_dy, d_b = w32.to(DEV), x.to(DEV), dy.to(DEV), bias.to(DEV)
    y = torch.zeros((B, S, S, S, cout), dtype=torch.bfloat16, device=DEV)
    dx = torch.zeros((B, S, S, S, cin), dtype=torch.bfloat16, device=DEV)
    dw = torch.zeros((cout, 27, cin), device=DEV)
    L = lib()
    capi.check(L.dsmc_sg_pack_weights(stream(), P(d_w32), cout, cin, P(wf), P(wd)))
    capi.check(L.dsmc_sg_conv3(stream(), B, S, P(d_x), cin, 0, cin, P(wf), P(d_b), cout, P(y), cout, 0, 1, None, 0, 0))
    capi.check(L.dsmc_sg_conv3(stream(), B, S, P(d_dy), cout, 0, cout, P(wd), None, cin, P(dx), cin, 0, 0, P(d_x), cin,
                               0))
    capi.check(L.dsmc_sg_conv3_wgrad(stream(), B, S, P(d_dy), cout, 0, cout, P(d_x), cin, 0, cin, P(dw)))
    sync_ok()
    # fp64 on the GPU, tap by tap (the network's largest layers take torch's CPU operator minutes)
    xd, dyd, wb = d_x.double(), d_dy.double(), d_w32.to(torch.bfloat16).double()
    ry, rdx, rdw = d_b.double().expand(B, S, S, S, cout).clone(), torch.zeros_like(xd), torch.zeros_like(wb)
    for t in range(27):
        off = (t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1)
        ry += torch.roll(xd, tuple(-o for o in off), (1, 2, 3)) @ wb[:, t].T
        back = torch.roll(dyd, off, (1, 2, 3))
        rdx += back @ wb[:, t]
        rdw[:, t] = back.reshape(-1, cout).T @ xd.reshape(-1, cin)
    close_bf16(y, torch.relu(ry).cpu())
    close_bf16(dx, (rdx * (xd > 0)).cpu())
    assert rel_l2(dw.cpu().numpy(), rdw.cpu().numpy()) <= 1e-4


@pytest.mark.parametrize("B,cin,cout", [(1, 16, 16), (1, 96, 64), (2, 48, 48), (3, 64, 96), (5, 32, 32), (41, 96, 32)])
def test_conv_of_pairs_of_samples(B, cin, cout):
    """Edge 8, two samples per tile: even and odd batches, one and several
    planes per item, reads and writes through views of wider tensors, and the
    volume behind the last sample untouched.  bf16 results held to the
    rounding of the output, as the module's other tests."""
    S = 8
    g = torch.Generator().manual_seed(100 * B + cin + cout)
    xw = rnd_bf16((B, S, S, S, cin + 16), g)
    x = xw[..., 8:8 + cin]
    mask = rnd_bf16((B, S, S, S, cout), g)
    w32 = torch.randn((cout, 27, cin), generator=g) * (2.0 / (27 * cin)) ** 0.5
    bias = torch.randn(cout, generator=g) * 0.1
    wf = torch.empty(cout * 27 * cin, dtype=torch.int16, device=DEV)
    wd = torch.empty_like(wf)
    d_w32, d_xw, d_m, d_b = w32.to(DEV), xw.to(DEV), mask.to(DEV), bias.to(DEV)
    y = torch.full((B + 1, S, S, S, cout + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    ym = torch.full((B + 1, S, S, S, cout), 7.0, dtype=torch.bfloat16, device=DEV)
    L = lib()
    capi.check(L.dsmc_sg_pack_weights(stream(), P(d_w32), cout, cin, P(wf), P(wd)))
    capi.check(L.dsmc_sg_conv3(stream(), B, S, P(d_xw), cin + 16, 8, cin, P(wf), P(d_b), cout, P(y), cout + 8, 8, 1, None, 0, 0))
    capi.check(L.dsmc_sg_conv3(stream(), B, S, P(d_xw), cin + 16, 8, cin, P(wf), None, cout, P(ym), cout, 0, 0, P(d_m), cout, 0))
    sync_ok()
    xd, wb = x.to(DEV).double(), d_w32.to(torch.bfloat16).double()
    ref = torch.zeros((B, S, S, S, cout), dtype=torch.float64, device=DEV)
    for t in range(27):
        off = (t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1)
        ref += torch.roll(xd, tuple(-o for o in off), (1, 2, 3)) @ wb[:, t].T
    close_bf16(y[:B, ..., 8:], torch.relu(ref + d_b.double()).cpu())
    close_bf16(ym[:B], (ref * (d_m > 0)).cpu())
    assert (y[B] == 7.0).all() and (y[..., :8] == 7.0).all() and (ym[B] == 7.0).all()


@pytest.mark.parametrize("B,cin,cout", [(1, 16, 16), (2, 96, 64), (3, 48, 96), (5, 64, 48), (41, 32, 32), (8, 16, 160)])
def test_wgrad_of_pairs_of_samples(B, cin, cout):
    """Edge 8, two samples per tile: even and odd batches (what lies behind
    the last sample is NaN), both blocks of input channels, each width of output
    channels, through views.  Accumulators of at most 64 truncating additions
    (64 x 2^-24) and at most 21 partial sums added in fp32: 1e-5."""
    S = 8
    g = torch.Generator().manual_seed(10 * B + cin + cout)
    x = torch.full((B + 1, S, S, S, cin + 8), float("nan"), dtype=torch.bfloat16)
    dy = torch.full((B + 1, S, S, S, cout + 16), float("nan"), dtype=torch.bfloat16)
    x[:B] = rnd_bf16((B, S, S, S, cin + 8), g)
    dy[:B] = rnd_bf16((B, S, S, S, cout + 16), g)
    d_x, d_dy = x.to(DEV), dy.to(DEV)
    dw = torch.zeros((cout, 27, cin), device=DEV)
    capi.check(lib().dsmc_sg_conv3_wgrad(stream(), B, S, P(d_dy), cout + 16, 16, cout, P(d_x), cin + 8, 8, cin, P(dw)))
    sync_ok()
    xd, dyd = d_x[:B, ..., 8:].double(), d_dy[:B, ..., 16:].double().reshape(-1, cout)
    ref = torch.zeros((cout, 27, cin), dtype=torch.float64, device=DEV)
    for t in range(27):
        off = (t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1)
        ref[:, t] = dyd.T @ torch.roll(xd, tuple(-o for o in off), (1, 2, 3)).reshape(-1, cin)
    assert ((dw.double() - ref).norm() / ref.norm()).item() <= 1e-5


@pytest.mark.parametrize("B,S,c,cs,off", [(1, 4, 16, 16, 0), (3, 8, 48, 64, 16), (2, 16, 128, 128, 0), (1, 16, 8, 24, 8),
                                          (2, 8, 20, 24, 1), (1, 2, 128, 128, 0)])
def test_bias_gradient_shapes(B, S, c, cs, off):
    """16-byte chunks (channel counts whose chunks do and do not divide the
    block, fewer rows than blocks, a view) and the scalar kernel (20 channels
    at an odd offset) against fp64; fp32 sums of at most 8192 rows in blocks
    of a few hundred: relative error below 1e-4 of the sums' scale."""
    g = torch.Generator().manual_seed(c + S)
    x = rnd_bf16((B, S, S, S, cs), g)
    db = torch.ones(c, device=DEV)  # accumulated
    d = x.to(DEV)
    capi.check(lib().dsmc_sg_bias_grad(stream(), B, S, P(d), cs, off, c, P(db)))
    ref = 1.0 + x[..., off:off + c].double().sum(dim=(0, 1, 2, 3))
    scale = x[..., off:off + c].double().abs().sum(dim=(0, 1, 2, 3)).max().item()
    assert (db.cpu().double() - ref).abs().max().item() <= 1e-4 * scale


@pytest.mark.parametrize("B,S", [(1, 2), (3, 4), (2, 16)])
def test_loss_and_head_backward_rows(B, S):
    """Loss, head gradients and input gradient at few rows (fewer than a
    warp's eight), rows that do not fill the last turn, and many; fp32
    products summed in another order than fp64: 1e-4 of each tensor's norm,
    the bf16 input gradient to its rounding."""
    g = torch.Generator().manual_seed(S)
    e = torch.relu(torch.randn((B, S, S, S, 16), generator=g)).to(torch.bfloat16)
    wh = torch.randn((4, 16), generator=g)
    out, tgt = torch.randn((B, S, S, S, 4), generator=g), torch.randn((B, S, S, S, 4), generator=g)
    valid = (torch.rand((B, S, S, S), generator=g) < 0.6).to(torch.uint8)
    cw = torch.tensor([1.0, 4.0, 1.0, 0.5])
    coef = torch.randn(B, generator=g, dtype=torch.float64)
    inv = 1.0 / max(1, int(valid.sum()))
    d = [t.to(DEV) for t in (out, tgt, valid, cw, e, wh, coef)]
    dwh, dbh = torch.zeros((4, 16), device=DEV), torch.zeros(4, device=DEV)
    de = torch.zeros_like(d[4])
    loss = torch.zeros(1, dtype=torch.float64, device=DEV)
    capi.check(lib().dsmc_sg_loss_head_bwd(stream(), B, S, P(d[0]), P(d[1]), P(d[2]), P(d[3]), C.c_float(inv), P(d[4]), 16, 0,
                                           P(d[5]), P(dwh), P(dbh), P(de), 16, 0, P(loss), P(d[6]), 1))
    v = valid.double()[..., None]
    diff = (out - tgt).double() * v
    dout = 2.0 * cw.double() * diff * inv
    dout[..., 1] += coef.reshape(B, 1, 1, 1) * v[..., 0]
    ed = e.double()
    assert abs(loss.item() - float((cw.double() * diff ** 2).sum() * inv)) <= 1e-5 * abs(loss.item())
    assert rel_l2(dwh.cpu().numpy(), (dout.reshape(-1, 4).T @ ed.reshape(-1, 16)).numpy()) <= 1e-4
    assert rel_l2(dbh.cpu().numpy(), dout.reshape(-1, 4).sum(0).numpy()) <= 1e-4
    close_bf16(de, (dout @ wh.double()) * (ed > 0))


@pytest.mark.parametrize("B,S,ci,co", [(24, 32, 16, 96), (25, 32, 16, 96), (8, 64, 16, 48), (5, 64, 32, 48)])
def test_wgrad_at_the_longest_sums(B, S, ci, co):
    """Weight gradients on both sides of the number of additions per
    accumulator at which the gathering kernel takes over, against fp64 sums:
    an accumulator of n additions that each truncate by half an ulp on average is off by at
    most n 2^-24 of its size."""
    g = torch.Generator(device=DEV).manual_seed(B)
    x = torch.relu(torch.randn((B, S, S, S, ci), generator=g, device=DEV)).to(torch.bfloat16)
    dy = torch.randn((B, S, S, S, co), generator=g, device=DEV).to(torch.bfloat16)
    dw = torch.zeros((co, 27, ci), device=DEV)
    capi.check(lib().dsmc_sg_conv3_wgrad(stream(), B, S, P(dy), co, 0, co, P(x), ci, 0, ci, P(dw)))
    rows = B * S ** 3
    adds = rows * ((27 * co + 127) // 128) / (148 * 4) / 16
    dyd = dy.reshape(-1, co).double()
    for t in (0, 4, 13, 22, 26):
        d = (t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1)
        ref = dyd.T @ torch.roll(x, (-d[0], -d[1], -d[2]), (1, 2, 3)).reshape(-1, ci).double()
        assert ((dw[:, t].double() - ref).norm() / ref.norm()).item() <= adds * 2.0 ** -24, t


def test_pool_and_upsample_forward_and_backward():
    g = torch.Generator().manual_seed(11)
    B, S, Cc = 2, 16, 32
    x = rnd_bf16((B, S, S, S, Cc), g)
    act = rnd_bf16((B, S, S, S, Cc), g)
    skip = rnd_bf16((B, S, S, S, Cc), g)
    dyp = rnd_bf16((B, S // 2, S // 2, S // 2, Cc), g)
    L, s = lib(), stream()
    dx, dact, dskip, ddyp = x.to(DEV), act.to(DEV), skip.to(DEV), dyp.to(DEV)
    pooled = torch.zeros((B, S // 2, S // 2, S // 2, Cc), dtype=torch.bfloat16, device=DEV)
    capi.check(L.dsmc_sg_pool2(s, B, S, P(dx), Cc, 0, Cc, P(pooled), Cc, 0))
    pb = torch.zeros((B, S, S, S, Cc), dtype=torch.bfloat16, device=DEV)
    capi.check(L.dsmc_sg_pool2_bwd(s, B, S, P(ddyp), Cc, 0, P(dskip), Cc, 0, P(dact), Cc, 0, Cc, P(pb), Cc, 0))
    up = torch.zeros((B, S, S, S, Cc), dtype=torch.bfloat16, device=DEV)
    capi.check(L.dsmc_sg_up2(s, B, S, P(ddyp), Cc, 0, Cc, P(up), Cc, 0))
    ub = torch.zeros((B, S // 2, S // 2, S // 2, Cc), dtype=torch.bfloat16, device=DEV)
    capi.check(L.dsmc_sg_up2_bwd(s, B, S, P(dx), Cc, 0, None, 0, 0, Cc, P(ub), Cc, 0))
    sync_ok()
    X = to_ncdhw(x)
    close_bf16(to_ncdhw(pooled), F.avg_pool3d(X, 2))
    upref = to_ncdhw(dyp).repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
    assert torch.equal(to_ncdhw(up), upref)
    close_bf16(to_ncdhw(pb), (to_ncdhw(skip) + upref / 8) * (to_ncdhw(act) > 0))
    close_bf16(to_ncdhw(ub), F.avg_pool3d(X, 2) * 8)


def test_adam_matches_the_published_update():
    n = 1000
    g = torch.Generator().manual_seed(5)
    p0 = torch.randn(n, generator=g)
    grads = [torch.randn(n, generator=g) for _ in range(3)]
    p, m, v = p0.to(DEV), torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
    for k, gr in enumerate(grads, 1):
        gd = gr.to(DEV)
        capi.check(lib().dsmc_sg_adam(stream(), P(p), P(gd), P(m), P(v), n, C.c_float(1e-2), C.c_float(0.9),
                                      C.c_float(0.999), C.c_float(1e-8), k))
    torch.cuda.synchronize(DEV)
    q = p0.clone().to(torch.float64)
    mm = torch.zeros(n, dtype=torch.float64)
    vv = torch.zeros(n, dtype=torch.float64)
    for k, gr in enumerate(grads, 1):
        gr = gr.to(torch.float64)
        mm = 0.9 * mm + 0.1 * gr
        vv = 0.999 * vv + 0.001 * gr * gr
        q -= 1e-2 * (mm / (1 - 0.9 ** k)) / ((vv / (1 - 0.999 ** k)).sqrt() + 1e-8)
    assert torch.allclose(p.cpu().to(torch.float64), q, rtol=1e-5, atol=1e-6)


def sample_batch(B, S, seed):
    rng = np.random.default_rng(seed)
    solid = (rng.random((B, S, S, S)) < 0.35).astype(np.uint8)
    feature = rng.normal(0, 1, B).astype(np.float32)
    target = rng.normal(0, 1, (B, S, S, S, 4)).astype(np.float32)
    valid = (solid == 0).astype(np.uint8)
    return solid, feature, target, valid


def test_unet_forward_backward_matches_cpu_reference():
    from oracle.unet_ref import UNetRef
    B, S = 2, 16
    params = sgm.init_parameters(seed=3)
    # non-zero biases so every bias path is exercised
    lay, _ = sgm.parameter_layout()
    rng = np.random.default_rng(4)
    for k, (o, sh) in lay.items():
        if k.endswith(".b"):
            params[o:o + int(np.prod(sh))] = rng.normal(0, 0.05, int(np.prod(sh)))
    solid, feature, target, valid = sample_batch(B, S, 9)
    cw = np.array([1.0, 0.5, 0.25, 0.25], np.float32)
    net = sgm.UNet(0, params)
    out = net.forward(torch.tensor(solid, device=DEV), torch.tensor(feature, device=DEV))
    net.loss_acc.zero_()
    net.backward(torch.tensor(target, device=DEV), torch.tensor(valid, device=DEV), cw, flux_weight=3.0)
    sync_ok()
    ref = UNetRef(params, emulate_bf16=True)
    rout = ref.forward(solid, feature)
    loss = ref.loss(rout, target, valid, cw, flux_weight=3.0)
    loss.backward()
    o = out.detach().cpu().numpy()
    assert rel_l2(o, rout.detach().numpy()) <= 1e-2
    assert net.loss_acc.item() == pytest.approx(loss.item(), rel=1e-2)
    gg, rg = net.grads_host(), ref.grads()
    # bf16 itself moves the gradient by 1-9 % from the exact fp64 one; the
    # emulating reference reproduces most of that, and what is left (an fp32
    # sum on the other side of a rounding boundary, compounded through the
    # backward chain) must stay well inside it
    exact = UNetRef(params, emulate_bf16=False)
    exact.loss(exact.forward(solid, feature), target, valid, cw, flux_weight=3.0).backward()
    eg = exact.grads()
    for k in rg:
        e_gpu, e_bf16 = rel_l2(gg[k], rg[k]), rel_l2(rg[k], eg[k])
        assert e_gpu <= max(0.75 * e_bf16, 2e-3), (k, e_gpu, e_bf16)
    flat_g = np.concatenate([gg[k].ravel() for k in rg])
    flat_r = np.concatenate([rg[k].ravel() for k in rg])
    assert flat_g @ flat_r / (np.linalg.norm(flat_g) * np.linalg.norm(flat_r)) >= 0.999
    # the gradient is the derivative: one step along it lowers the fp64 loss
    ref2 = UNetRef(params - 1e-3 * net.g.cpu().numpy() / np.linalg.norm(net.g.cpu().numpy()), emulate_bf16=False)
    l2 = ref2.loss(ref2.forward(solid, feature), target, valid, cw, flux_weight=3.0).item()
    ref3 = UNetRef(params, emulate_bf16=False)
    l3 = ref3.loss(ref3.forward(solid, feature), target, valid, cw, flux_weight=3.0).item()
    assert l2 < l3


def test_training_on_one_batch_lowers_the_loss():
    B, S = 4, 16
    solid, feature, _, valid = sample_batch(B, S, 21)
    # a learnable target: a smooth function of the local openness
    open_ = 1.0 - solid.astype(np.float32)
    k = np.ones((3, 3, 3), np.float32) / 27
    from scipy.ndimage import convolve
    sm = np.stack([convolve(open_[b], k, mode="wrap") for b in range(B)])
    target = np.stack([sm, 0.5 * sm, -sm, sm * sm], -1).astype(np.float32)
    net = sgm.UNet(0, seed=1)
    d = [torch.tensor(a, device=DEV) for a in (solid, feature, target, valid)]
    losses = []
    for it in range(60):
        net.loss_acc.zero_()
        net.forward(d[0], d[1])
        net.backward(d[2], d[3], [1, 1, 1, 1])
        losses.append(net.loss_acc.item())
        net.adam(lr=3e-3)
    sync_ok()
    assert np.isfinite(losses).all()
    assert losses[-1] < 0.2 * losses[0], losses[::10]


@pytest.mark.parametrize("B,S,ci,co", [(50, 16, 96, 16), (7, 32, 96, 16), (49, 16, 48, 16), (41, 8, 96, 16), (8, 64, 16, 16)])
def test_wgrad_accumulators_take_no_more_additions_than_the_gathering_kernels(B, S, ci, co):
    """Positive data: every addition of an accumulator truncates by half an ulp
    on average and nothing cancels, so the sums' mean shortfall is proportional
    to the additions per accumulator. The same values as many boxes of edge
    4, which the gathering kernel takes, are split into accumulators by the same
    rule; the plane kernels' shortfall is at most that one (a tenth is left for
    the accumulators that end early in either). The lengths cover a whole item of planes longer
    than the limit (88, 100 and 44 additions) and limits of several items."""
    g = torch.Generator(device=DEV).manual_seed(S * B)
    rows = B * S ** 3
    x = (torch.rand((rows, ci), generator=g, device=DEV) + 0.5).to(torch.bfloat16)
    dy = (torch.rand((rows, co), generator=g, device=DEV) + 0.5).to(torch.bfloat16)
    short = []
    for b, s in ((B, S), (rows // 64, 4)):
        dw = torch.zeros((co, 27, ci), device=DEV)
        capi.check(lib().dsmc_sg_conv3_wgrad(stream(), b, s, P(dy), co, 0, co, P(x), ci, 0, ci, P(dw)))
        sync_ok()
        total, n = 0.0, 0
        for t in (0, 5, 13, 22):
            d = (t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1)
            xs = torch.roll(x.reshape(b, s, s, s, ci), tuple(-o for o in d), (1, 2, 3)).reshape(-1, ci)
            ref = sum(dy[k:k + 65536].double().T @ xs[k:k + 65536].double() for k in range(0, rows, 65536))
            total += ((ref - dw[:, t].double()) / ref).sum().item()
            n += ref.numel()
        short.append(total / n)
    assert 0.0 < short[0] <= 1.1 * short[1], short


@pytest.mark.parametrize("B,S,co", [(1, 8, 48), (3, 32, 16), (4, 32, 96), (5, 32, 16), (65, 16, 32)])
def test_wgrad_of_48_input_channels_in_one_launch_and_two(B, S, co):
    """Three blocks of 16 input channels in one launch (up to 131072 voxels) and
    blocks of 32 and 16 in two (above), the largest one-launch size included,
    through views.  Truncating sums of at most 304 additions (x 2^-24) and
    as many partial sums added in fp32: 3e-5."""
    ci = 48
    g = torch.Generator(device=DEV).manual_seed(B + S)
    rows = B * S ** 3
    x = torch.relu(torch.randn((B, S, S, S, ci + 16), generator=g, device=DEV)).to(torch.bfloat16)
    dy = torch.randn((B, S, S, S, co + 8), generator=g, device=DEV).to(torch.bfloat16)
    dw = torch.ones((co, 27, ci), device=DEV)  # accumulated
    capi.check(lib().dsmc_sg_conv3_wgrad(stream(), B, S, P(dy), co + 8, 8, co, P(x), ci + 16, 16, ci, P(dw)))
    sync_ok()
    dyd = dy[..., 8:].reshape(rows, co).double()
    for t in range(27):
        d = (t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1)
        ref = 1.0 + dyd.T @ torch.roll(x[..., 16:], tuple(-o for o in d), (1, 2, 3)).reshape(rows, ci).double()
        assert ((dw[:, t].double() - ref).norm() / ref.norm()).item() <= 3e-5, t
