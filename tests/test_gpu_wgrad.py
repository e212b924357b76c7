"""The network's weight gradients layer by layer at widths around the 128-pixel
strips of their kernels (8 to 1032 columns: levels of 1 to 1032 pixels, strips
of 1, 2, 4, 5, 8, 16 ... pixels left over) and at row counts that the row
groups do not divide.

Against the same forward and backward pass in torch (FP64) with every stored
activation and activation gradient rounded to BF16 where the device stores it
so. The weights make the convolutions copies (centre tap the identity, lift and
projection of signs) and the input is -1, 0 or 1, so every activation is a
multiple of 1/64 below 4 (exact in BF16) and no gradient of an activation goes
through a long FP32 sum whose order could round it the other way: both sides
contract the same operands, random in every tap. What is left is the FP32
accumulation of up to 25,000 terms of random sign, 2^-24 sqrt(25,000) ~ 1e-5 of
a sum's size; bound 1e-4 of a layer's largest tap. A strip's end or a row left
out of a gradient is off by more than 3 %."""
import numpy as np
import pytest

from test_gpu_learned import s_apply_ref

pytestmark = pytest.mark.gpu
C = 32


def _restated(params, x, t, st, NK):
    import torch
    import torch.nn.functional as F

    bf = lambda a: a.to(torch.bfloat16).to(torch.float64)

    def pad(a):     # periodic in x, zero beyond the rows
        return F.pad(F.pad(a[None], (1, 1, 0, 0), mode="circular"), (0, 0, 1, 1))

    def conv(a, w):                                   # w [9][cin][cout]
        return F.conv2d(pad(a), w.reshape(3, 3, w.shape[1], w.shape[2]).permute(3, 2, 0, 1))[0]

    def adjoint(d, w):
        return conv(d, torch.stack([w[8 - k].T for k in range(9)]))

    def wgrad(a, d):                                  # sum_p a[p + off] d[p] -> [9][cin][cout]
        p = pad(a)[0]
        H, W = d.shape[1:]
        return torch.stack([torch.einsum("ihw,ohw->io", p[:, dy:dy + H, dx:dx + W], d) for dy in range(3) for dx in range(3)])

    sum4 = lambda a: 4 * F.avg_pool2d(a[None], 2)[0]
    up = lambda a: a.repeat_interleave(2, 1).repeat_interleave(2, 2)
    lift, proj = params[:9 * C].reshape(9, 1, C), params[-9 * C:].reshape(9, C, 1)
    w = [bf(params[9 * C + j * 9 * C * C:9 * C + (j + 1) * 9 * C * C].reshape(9, C, C)) for j in range(6)]
    h, pl, u, g = [bf(conv(x[None], lift))], [None], [None] * 3, [None] * 3
    for l in range(1, 4):
        pl.append(bf(0.25 * sum4(h[l - 1])))
        h.append(bf(conv(pl[l], w[l - 1])))
    low = h[3]
    for l in (2, 1, 0):
        u[l] = bf(up(low) + h[l])
        g[l] = bf(conv(u[l], w[3 + (2 - l)]))
        low = g[l]
    z = conv(g[0], proj)[0]
    z[NK:] = 0.0
    Sz, St = s_apply_ref(z, st, NK), s_apply_ref(t, st, NK)
    a, b, c = (z * St).sum(), (z * Sz).sum(), (t * St).sum()
    dz = 2 * a / (b * c) * (a / b * Sz - St)
    dz[NK:] = 0.0
    out = [None] * 8
    out[7] = wgrad(g[0], dz[None])
    dg, du = bf(adjoint(dz[None], proj)), [None] * 3
    for l in range(3):
        du[l] = bf(adjoint(dg, w[3 + (2 - l)]))
        out[1 + 3 + (2 - l)] = wgrad(u[l], dg)
        dg = bf(sum4(du[l]))
    dh = dg
    for l in (3, 2, 1):
        dp = bf(adjoint(dh, w[l - 1]))
        out[1 + l - 1] = wgrad(pl[l], dh)
        du[l - 1] = bf(0.25 * up(dp) + du[l - 1])
        dh = du[l - 1]
    out[0] = wgrad(x[None], dh)
    return out


@pytest.mark.parametrize("NX,NZ", [(8, 9), (40, 17), (128, 33), (136, 41), (264, 24), (1032, 20)])
def test_weight_gradients_match_restatement(NX, NZ):
    import torch
    from vvm_b200 import build, gpu as G
    from vvm_b200.initial_state import warm_bubble
    build.build()
    st = warm_bubble(NX, NZ)
    g = G.VVMGpu(st.grid, solver=G.VVM_SOLVER_LEARNED)
    g.upload(st)
    H0, W0, n = g.learned_shape()
    NK = NZ - 1
    rng = np.random.default_rng(NX)
    sign = rng.choice((-1.0, 1.0), C)
    w = np.zeros(n, np.float32)
    w[4 * C:5 * C] = sign                                     # lift: tap 4 is the centre
    for j in range(6):
        w[9 * C + j * 9 * C * C:][4 * C * C:5 * C * C] = np.eye(C).reshape(-1)
    w[-9 * C:][4 * C:5 * C] = sign * 2.0 ** -rng.integers(3, 7, C)
    g.learned_weights(w)
    x, t = np.zeros((H0, W0), np.float32), np.zeros((H0, W0), np.float32)
    x[:NK] = rng.integers(-1, 2, (NK, W0))
    t[:NK] = rng.standard_normal((NK, W0))
    t += g.learned_eval(x)
    _, grad, _ = g.learned_eval(x, t)
    g.close()
    ref = _restated(*(torch.tensor(a.astype(np.float64)) for a in (w, x, t)), st, NK)
    at = 0
    for layer, r in enumerate(ref):
        b = r.reshape(9, -1).numpy()
        a = grad[at:at + b.size].reshape(9, -1)
        at += b.size
        most = max(np.linalg.norm(v) for v in b)
        for tap in range(9):
            assert np.linalg.norm(a[tap] - b[tap]) <= 1e-4 * most, (layer, tap, np.linalg.norm(a[tap] - b[tap]) / most)
