"""The FP32 operator of the mixed solve recomputed from rounded point records is
no further from the FP64 one than the FP64 matrices rounded to FP32 are: both
restated in numpy, in the kernels' order of operations, on elements of meshes
that were once solved with stored matrices (100,000 elements and more)."""
import numpy as np
import pytest

from specfem3d_geotech_gb300 import meshgen

F = np.float32
D = np.array([[-1.5, 2, -0.5], [-0.5, 0, 0.5], [0.5, -2, 1.5]])
NODES = np.array([[i % 3, i // 3 % 3, i // 9] for i in range(27)])
CORNERS = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])
W = np.prod(np.array([1, 4, 1])[NODES] / 3.0, axis=1)


def fma(a, b, c):
    return (np.float64(a) * np.float64(b) + np.float64(c)).astype(F)


def line(i, a):
    """Position of node i on its lattice line along a, and the line's nodes."""
    st = 3 ** a
    return NODES[i, a], i + st * (np.arange(3) - NODES[i, a])


def elements(mesh, sel):
    x = np.stack([mesh.x, mesh.y, mesh.z], 1)[mesh.conn[sel] - 1]
    p = NODES - 1.0
    f = 1 + CORNERS[None] * p[:, None]
    dn = np.stack([CORNERS[None, :, a] * np.prod(np.delete(f, a, 2), axis=2) / 8 for a in range(3)], 2)
    jac = np.einsum("qna,enb->eqab", dn, x)
    im = mesh.mat_id[sel] - 1
    e, nu = mesh.props[im, 1], mesh.props[im, 2]
    ef = e / ((1 + nu) * (1 - 2 * nu))
    wd = np.linalg.det(jac) * W
    c = [wd * k[:, None] for k in ((1 - nu) * ef, nu * ef, 0.5 * (1 - 2 * nu) * ef)]
    return np.einsum("qn,enb->eqb", np.prod(f, axis=2) / 8, x), np.linalg.inv(jac), c


def matrices(ji, c):
    dl = np.zeros((27, 27, 3))
    for i in range(27):
        for a in range(3):
            k, nd = line(i, a)
            dl[i, nd, a] += D[k]
    g = np.einsum("eqba,qna->eqnb", ji, dl)
    s = [np.einsum("eq,eqnc,eqmd->encmd", k, g, g) for k in c]
    trace = np.einsum("encmc->enm", s[2])
    out = np.zeros_like(s[0])
    for i in range(3):
        for j in range(3):
            out[:, :, i, :, j] = (s[0][:, :, i, :, i] + trace - s[2][:, :, i, :, i] if i == j
                                  else s[1][:, :, i, :, j] + s[2][:, :, j, :, i])
    return out.reshape(-1, 81, 81)


def stored(k, p):
    y = np.zeros(p.shape, F)
    for m in range(81):
        y = fma(k[:, :, m].astype(F), p[:, m:m + 1], y)
    return y


def recomputed(ji, c, p):
    ji, (c11, c12, c44), d32 = ji.astype(F), (k.astype(F) for k in c), D.astype(F)
    u = p.reshape(-1, 27, 3)
    gr, gp, t, fl = (np.zeros((len(u), 27, 3, 3), F) for _ in range(4))
    for q in range(27):
        for a in range(3):
            k, nd = line(q, a)
            s = d32[k, 0] * u[:, nd[0]]
            if k != 1:
                s = fma(d32[k, 1], u[:, nd[1]], s)
            gr[:, q, :, a] = fma(d32[k, 2], u[:, nd[2]], s)
    for i in range(3):
        for d in range(3):
            gp[:, :, i, d] = fma(ji[:, :, d, 0], gr[:, :, i, 0],
                                 fma(ji[:, :, d, 1], gr[:, :, i, 1], ji[:, :, d, 2] * gr[:, :, i, 2]))
    for i in range(3):
        j, k = (i + 1) % 3, (i + 2) % 3
        t[:, :, i, i] = fma(c11, gp[:, :, i, i], c12 * (gp[:, :, min(j, k), min(j, k)] + gp[:, :, max(j, k), max(j, k)]))
        t[:, :, i, j] = t[:, :, j, i] = c44 * (gp[:, :, i, j] + gp[:, :, j, i])
    for i in range(3):
        for r in range(3):
            fl[:, :, i, r] = fma(ji[:, :, 0, r], t[:, :, i, 0],
                                 fma(ji[:, :, 1, r], t[:, :, i, 1], ji[:, :, 2, r] * t[:, :, i, 2]))
    y = np.zeros(u.shape, F)
    for n in range(27):
        for a in range(3):
            k, nd = line(n, a)
            for i in range(3):
                if D[i, k]:
                    y[:, n] = fma(d32[i, k], fl[:, nd[i], :, a], y[:, n])
    return y.reshape(p.shape)


@pytest.mark.parametrize("dims", [(120, 40, 40), (100, 40, 30)])
def test_recomputed_operator_is_no_further_off(dims):
    rng = np.random.default_rng(0)
    mesh = meshgen.slope3d(*dims, seed=3)
    x, ji, c = elements(mesh, rng.choice(mesh.nelmt, 200, replace=False))
    k = matrices(ji, c)
    top, noise = mesh.z.max(), rng.standard_normal((200, 27, 3))

    def wave(n):
        a = 2 * np.pi * n / max(mesh.x.max(), top) * x
        return np.stack([np.sin(a[..., 0] + 0.3) * np.cos(0.5 * a[..., 2]), np.cos(a[..., 1] + 0.7),
                         np.sin(a[..., 2] + 0.1) * np.cos(0.7 * a[..., 0])], -1)

    settled = np.stack([2e-4 * x[..., 2], 0 * x[..., 1], -1e-3 * (top * x[..., 2] - 0.5 * x[..., 2] ** 2)], -1)
    fields = dict(noise=noise, settled=settled, rough=wave(8) + 1e-3 * noise, **{f"wave{n}": wave(n) for n in (1, 8, 40)})
    for name, f in fields.items():
        p = f.reshape(200, 81).astype(F)
        exact = np.einsum("eij,ej->ei", k, np.float64(p))
        a, b = (np.linalg.norm(y - exact) / np.linalg.norm(exact) for y in (stored(k, p), recomputed(ji, c, p)))
        print(name, "matrices %.2e, point records %.2e" % (a, b))
        assert b <= a, name
