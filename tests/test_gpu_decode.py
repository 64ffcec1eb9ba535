"""The batched decode step at the sizes where its two kernels change hands and their loops end: rings around 32 slots and past what
the staged kernel keeps in shared memory, heads around 16, widths that rule out 16-byte pieces, positions before, at and
after the wrap and past the rotary table.  The reference is float64; a dot product of dk fp32 terms and a weighted mean of at
most `cap` rows stay within sqrt(dk + cap) * 2^-23 of it, 5e-6 leaves a factor of two at dk + cap = 400."""
import numpy as np
import pytest

from gpu_util import dev, host, normal, rel_err

pytestmark = pytest.mark.gpu


def reference(q_c, q_r, k_c, k_r, v_c, cos, sin, pos, kc, vc, H, dh, dr, cap, scale):
    N = len(pos)
    kc, vc, out = kc.copy(), vc.copy(), np.zeros((N, H * dh))

    def rotate(x, p):
        x = x.copy()
        if dr and p * (dr // 2) < len(cos):
            c, s = cos[p * (dr // 2):(p + 1) * (dr // 2)], sin[p * (dr // 2):(p + 1) * (dr // 2)]
            x[0::2], x[1::2] = x[0::2] * c - x[1::2] * s, x[0::2] * s + x[1::2] * c
        return x

    for n in range(N):
        p = int(pos[n]); slot, live = p % cap, min(p + 1, cap)
        for h in range(H):
            d, r = slice(h * dh, (h + 1) * dh), slice(h * dr, (h + 1) * dr)
            kc[n, h, slot] = np.concatenate([k_c[n, d], rotate(k_r[n, r], p)])
            vc[n, h, slot] = v_c[n, d]
            s = kc[n, h, :live] @ np.concatenate([q_c[n, d], rotate(q_r[n, r], p)]) * scale
            e = np.exp(s - s.max())
            out[n, d] = (e / e.sum()) @ vc[n, h, :live]
    return out, kc, vc


@pytest.mark.parametrize("N,H,dh,dr,cap", [(9, 4, 16, 16, 17), (5, 4, 32, 16, 17), (3, 1, 4, 4, 1), (3, 3, 8, 0, 33), (5, 2, 64, 32, 31), (3, 2, 128, 64, 12), (3, 1, 4, 0, 5),
                                           (3, 2, 12, 4, 32), (2, 2, 64, 64, 200), (5, 3, 6, 4, 9), (5, 3, 7, 2, 9)])
@pytest.mark.parametrize("offset", [0, 1])
def test_decode_step(talos, N, H, dh, dr, cap, offset):
    import torch
    ctx = talos.torch_context(0)
    steps = 40                                                   # rows of the rotary table
    q_c, k_c, v_c = (normal(i, (N, H * dh)) for i in (1, 2, 3))
    q_r, k_r = normal(4, (N, max(1, H * dr)))[:, :H * dr], normal(5, (N, max(1, H * dr)))[:, :H * dr]
    cos, sin = normal(6, (max(1, steps * (dr // 2)),)), normal(7, (max(1, steps * (dr // 2)),))
    pos = np.array([0, cap - 1, cap, 39, 40, 3 * cap + 1, 1, 5, 17][:N], dtype=np.int32)
    kc, vc = normal(8, (N, H, cap, dh + dr)), normal(9, (N, H, cap, dh))
    dk, dv = (dev(np.concatenate([np.zeros(offset), a.ravel(), np.full(4, 7.0)])) for a in (kc, vc))       # offset 1: caches off a 16-byte boundary
    out = torch.empty(N, H * dh, device="cuda")
    t = [dev(a) for a in (q_c, q_r, k_c, k_r, v_c, cos, sin, pos)]
    P = talos.ptr
    rot = [P(t[1]) if dr else None, P(t[3]) if dr else None, P(t[5]) if dr else None, P(t[6]) if dr else None]
    talos.lib.talos_mla_decode_step(ctx.handle, P(t[0]), rot[0], P(t[2]), rot[1], P(t[4]), rot[2], rot[3], steps * (dr // 2), P(t[7]), P(dk) + 4 * offset,
                                    P(dv) + 4 * offset, P(out), N, H, dh, dr, cap, 0.3)
    ref_out, ref_k, ref_v = reference(q_c, q_r, k_c, k_r, v_c, cos if dr else [], sin if dr else [], pos, kc, vc, H, dh, dr, cap, 0.3)
    ctx.synchronize()
    assert rel_err(out, ref_out) <= 5e-6
    got_k, got_v = host(dk)[offset:], host(dv)[offset:]
    assert rel_err(got_k[:kc.size], ref_k.ravel()) <= 1e-6 and np.array_equal(got_v[:vc.size], ref_v.ravel())
    assert np.all(got_k[kc.size:] == 7.0) and np.all(got_v[vc.size:] == 7.0)
