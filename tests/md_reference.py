"""Two-electron integrals of a small molecule in numpy, from the mathematics alone: McMurchie-Davidson Hermite
expansions (J. Comput. Phys. 26, 218 (1978)), Boys functions by the incomplete gamma function, full Coulomb or
erf(omega r)/r (F_m(T) -> theta^(m+1/2) F_m(theta T), theta = omega^2 / (omega^2 + pq/(p+q))).  Shells up to d."""
import math

import numpy as np
from scipy.special import gamma, gammainc


def _components(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _outputs(l, cart):
    """Cartesian components -> output functions with libcint's factors."""
    if l < 2 or cart:
        return np.eye((l + 1) * (l + 2) // 2) * {0: math.sqrt(0.25 / math.pi), 1: math.sqrt(0.75 / math.pi)}.get(l, 1.0)
    t = np.zeros((6, 5))                                         # xx xy xz yy yz zz -> m = -2 .. 2
    a, b = math.sqrt(15.0 / (4.0 * math.pi)), math.sqrt(5.0 / (16.0 * math.pi))
    t[1, 0] = t[4, 1] = t[2, 3] = a
    t[[0, 3, 5], 2] = -b, -b, 2.0 * b
    t[[0, 3], 4] = 0.5 * a, -0.5 * a
    return t


def _boys(t, top):
    out = np.empty((top + 1,) + t.shape)
    for m in range(top + 1):
        big = np.maximum(t, 1e-6)
        out[m] = np.where(t < 1e-6, 1.0 / (2 * m + 1) - t / (2 * m + 3),
                          gamma(m + 0.5) * gammainc(m + 0.5, big) / (2.0 * big ** (m + 0.5)))
    return out


def _hermites(top):
    return [(t, u, v) for t in range(top + 1) for u in range(top + 1 - t) for v in range(top + 1 - t - u)]


def _expansion(i, j, t, a, b, ab):
    """Hermite coefficient E_t^ij of two Gaussians in one dimension."""
    p = a + b
    if t < 0 or t > i + j:
        return 0.0 * p
    if i == j == 0:
        return np.exp(-a * b / p * ab * ab)
    if j == 0:
        return (_expansion(i - 1, j, t - 1, a, b, ab) / (2 * p) - b * ab / p * _expansion(i - 1, j, t, a, b, ab)
                + (t + 1) * _expansion(i - 1, j, t + 1, a, b, ab))
    return (_expansion(i, j - 1, t - 1, a, b, ab) / (2 * p) + a * ab / p * _expansion(i, j - 1, t, a, b, ab)
            + (t + 1) * _expansion(i, j - 1, t + 1, a, b, ab))


def _pair(s, r, cart):
    """(p, P, E[primitive pair, output pair, Hermite], output AO pairs) of two shells."""
    a, b = (x.ravel() for x in np.meshgrid(s["exp"], r["exp"], indexing="ij"))
    e1 = [{(i, j, t): _expansion(i, j, t, a, b, s["at"][x] - r["at"][x])
           for i in range(s["l"] + 1) for j in range(r["l"] + 1) for t in range(i + j + 1)} for x in range(3)]
    zero = 0.0 * a
    e = np.array([[e1[0].get((f[0], g[0], t), zero) * e1[1].get((f[1], g[1], u), zero) * e1[2].get((f[2], g[2], v), zero)
                   for t, u, v in _hermites(s["l"] + r["l"])] for f in _components(s["l"]) for g in _components(r["l"])])
    e = np.einsum("chp,co->poh", e, np.kron(_outputs(s["l"], cart), _outputs(r["l"], cart)))
    cc = np.einsum("ix,jy->ijxy", s["c"], r["c"]).reshape(len(a), -1)             # contraction columns
    e = np.einsum("px,poh->pxoh", cc, e).reshape(len(a), -1, e.shape[-1])
    n, m = (_outputs(x["l"], cart).shape[1] for x in (s, r))
    ao = [(s["ao"] + x * n + i, r["ao"] + y * m + j) for x in range(s["c"].shape[1]) for y in range(r["c"].shape[1])
          for i in range(n) for j in range(m)]
    return a + b, (np.outer(a, s["at"]) + np.outer(b, r["at"])) / (a + b)[:, None], e, np.array(ao), s["l"] + r["l"]


def _block(bra, ket, omega):
    (p, rp, eb, _, lb), (q, rq, ek, _, lk) = bra, ket
    p, q = p[:, None], q[None]
    rho = p * q / (p + q)
    d = rp[:, None] - rq[None]
    theta = omega ** 2 / (omega ** 2 + rho) if omega else np.ones_like(rho)
    f = _boys(theta * rho * (d * d).sum(-1), lb + lk)
    pre = 2.0 * math.pi ** 2.5 / (p * q * np.sqrt(p + q)) * np.sqrt(theta)
    level = {}
    for m in range(lb + lk, -1, -1):                            # R_tuv^m from R^(m+1)
        now = {(0, 0, 0): pre * (-2.0 * rho * theta) ** m * f[m]}
        for h in _hermites(lb + lk - m)[1:]:
            x = max(range(3), key=lambda i: h[i])
            one, two = (tuple(h[i] - k * (i == x) for i in range(3)) for k in (1, 2))
            now[h] = d[..., x] * level[one] + ((h[x] - 1) * level[two] if h[x] > 1 else 0.0)
        level = now
    out = 0.0
    for i, h in enumerate(_hermites(lb)):
        for j, g in enumerate(_hermites(lk)):
            r = level[tuple(x + y for x, y in zip(h, g))] * (-1.0) ** sum(g)
            out = out + eb[:, :, i].T @ r @ ek[:, :, j]
    return out


def eri(atm, bas, env, cart):
    """(n, n, n, n) integrals of libcint tables; env[8] = omega > 0 selects the erf-attenuated operator."""
    shells, n = [], 0
    for at, l, nprim, nctr, _, pe, pc, *_ in bas.tolist():
        c = env[pc:pc + nprim * nctr].reshape(nctr, nprim).T
        shells.append({"l": l, "exp": env[pe:pe + nprim], "c": c, "at": env[atm[at, 1]:atm[at, 1] + 3], "ao": n})
        n += nctr * _outputs(l, cart).shape[1]
    pairs = [_pair(s, r, cart) for i, s in enumerate(shells) for r in shells[:i + 1]]
    full = np.zeros((n, n, n, n))
    for x, bra in enumerate(pairs):
        for ket in pairs[:x + 1]:
            v = _block(bra, ket, float(env[8]))
            (i, j), (k, l) = bra[3].T[:, :, None], ket[3].T[:, None]
            for a, b in ((i, j), (j, i)):
                for c, e in ((k, l), (l, k)):
                    full[a, b, c, e] = v
                    full[c, e, a, b] = v
    return full
