"""sem_element_step_noalloc: the update's vector and scalar accesses (16-byte aligned buffers and
buffers one float off), node counts with every remainder of four, rows shorter than a thread's
four nodes, and calls on different meshes in turn (each call leaves the accumulator zero for the
next).  Against a float64 evaluation of the same step in numpy; the element sums run in float with
atomics, tolerance as in test_zz_no_alloc.py (5e-6 against the oracle)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step64(semgb, ex, ey, ez, o, h, p, q, coef, sp):
    """One step in float64 (fields [y][z][x])."""
    xi, w, d = semgb.gll_tables(o)
    d = d.reshape(o + 1, o + 1)  # d[j][i] = phi_j'(xi_i)
    S = d @ np.diag(w) @ d.T
    kp = np.zeros_like(p)
    g = h / 2
    for iy in range(ey):
        for iz in range(ez):
            for ix in range(ex):
                sl = tuple(slice(i * o, i * o + o + 1) for i in (iy, iz, ix))
                e = p[sl]
                wz, wx = w[None, :, None], w[None, None, :]
                kp[sl] += g * (np.einsum("ab,bzx->azx", S, e) * wz * wx + np.einsum("ab,ybx->yax", S, e) * w[:, None, None] * wx
                               + np.einsum("ab,yzb->yza", S, e) * w[:, None, None] * wz)
    v = q.copy()
    i = (slice(1, -1),) * 3
    v[i] = (2 * p - q - coef * kp)[i]
    s = 1.0 if sp is None else sp[1][:, None, None] * sp[2][None, :, None] * sp[0][None, None, :]
    return s * v, s * p


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("sponge", [False, True])
def test_update_access_widths(semgb_lib, cuda_device, offset, sponge):
    import torch

    semgb = semgb_lib
    lib = semgb.lib()
    rng = np.random.default_rng(5)
    h = 10.0
    dev = torch.device("cuda", 0)
    boxes = [(1, 1, 1, 1), (1, 2, 3, 1), (2, 1, 1, 2), (3, 2, 2, 3), (5, 4, 3, 4), (2, 3, 2, 5), (4, 4, 4, 2)]
    for ex, ey, ez, o in boxes + boxes[::-1]:
        n = (ey * o + 1, ez * o + 1, ex * o + 1)
        N = int(np.prod(n))
        p, q = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
        coef = rng.uniform(0.5e-3, 1e-3, n).astype(np.float32)
        sp = [rng.uniform(0.9, 1.0, m).astype(np.float32) for m in (n[2], n[0], n[1])] if sponge else None
        want = _step64(semgb, ex, ey, ez, o, h, p.astype(np.float64), q.astype(np.float64), coef.astype(np.float64),
                       [a.astype(np.float64) for a in sp] if sponge else None)
        buf = []
        for a in (p, q, coef):
            t = torch.full((N + 8,), 7.0, device=dev)
            t[offset:offset + N] = torch.from_numpy(a.reshape(-1)).to(dev)
            buf.append(t)
        mesh = semgb.Mesh(ex, ey, ez, ex * h, ey * h, ez * h, o)
        conn = torch.from_numpy(mesh.connectivity()).to(dev)
        ptr = [C.c_void_p(t.data_ptr() + 4 * offset) for t in buf]
        s = [torch.from_numpy(a).to(dev) for a in sp] if sponge else []
        sptr = [C.c_void_p(t.data_ptr()) for t in s] if sponge else [None] * 3
        rc = lib.sem_element_step_noalloc(ex, ey, ez, ex * h, ey * h, ez * h, o, C.c_void_p(conn.data_ptr()), ptr[0],
                                          ptr[1], ptr[2], *sptr, C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == semgb.SEM_OK, lib.sem_last_error_string().decode()
        torch.cuda.synchronize()
        for t, w in ((buf[1], want[0]), (buf[0], want[1])):
            got = t.cpu().numpy()
            a = got[offset:offset + N].astype(np.float64).reshape(n)
            assert np.linalg.norm(a - w) <= 5e-6 * np.linalg.norm(w), (ex, ey, ez, o)
            assert np.all(got[:offset] == 7.0) and np.all(got[offset + N:] == 7.0)
        mesh.close()
