"""Coordinate products of J/K for every class up to (ff|ff): order 1 against central differences of J/K, order 2 and
the order-2 VJP against central differences of order 1.  The step 1e-4 leaves h^2/6 times a third derivative, with
exponents up to 1e4 on the oxygen core at most 1e-7 of the elements here, and rounding 1e-16/h of them: 2e-7 and
3e-7 relative, the bounds of the reference's own difference tests; the VJP's scalar sums elements of such errors with
the cotangents as weights.

The VJP of order 1 is the adjoint of the JVP: <cotangents, JVP(u)> = VJP . u, two sums of the same n^4 FP64 terms by
different kernels (2e-14 of values up to 10 measured, 1e-12 allowed).  With every quartet in FP32 its elements move by
up to 4.2e-7 of the largest one; four times that."""
import ctypes
import sys
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs CUDA")]

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
from gradscf_b200 import _capi  # noqa: E402
from gradscf_b200 import jk as J  # noqa: E402
from tests.gpu_util import WATER, psd_density, tables  # noqa: E402


@pytest.mark.parametrize("cart,omega", [(False, 0.0), (True, 0.0), (False, 0.33)])
def test_geometry_products_of_every_class_match_differences(cart, omega):
    top, par, sa, atm, bas, env = tables("O 0 0 0; H 0.1 0.7572 0.5865", "cc-pvtz", cart)
    env[8] = omega
    rng = np.random.default_rng(3)
    d = psd_density(top.nao, 5, 2)
    slots = (atm[:, 1][:, None] + np.arange(3)[None, :]).ravel()
    u, v = np.zeros((2, len(env)))
    u[slots], v[slots] = 0.17 * rng.normal(size=(2, slots.size))
    h = 1e-4

    def close(a, b, atol=2e-7):
        np.testing.assert_allclose(a, b, atol=atol, rtol=3e-7)

    def jk(e):
        return torch.stack(J.direct_jk(atm, bas, e, d, cart=cart)).cpu().numpy()

    def first(e):
        return torch.stack(J.direct_jk_geometry_jvp(atm, bas, e, d, u, cart=cart)).cpu().numpy()

    close(first(env), (jk(env + h * u) - jk(env - h * u)) / (2 * h))
    plus, minus = first(env + h * v), first(env - h * v)
    close(torch.stack(J.direct_jk_geometry_jvp(atm, bas, env, d, u, v, cart=cart)).cpu().numpy(),
          (plus - minus) / (2 * h))
    cot = np.stack([np.cos(d), np.sin(d)])
    g = J.direct_jk_geometry_hvp(atm, bas, env, d, u, tuple(cot), cart=cart)
    close(g @ v, np.sum(cot * (plus - minus)) / (2 * h), atol=2e-7 * np.linalg.norm(cot))


@pytest.mark.parametrize("omega", [0.0, 0.33])
@pytest.mark.parametrize("atom,basis,cart", [("O 0 0 0; H 0.1 0.7572 0.5865", "cc-pvtz", False),
                                             ("O 0 0 0; H 0.1 0.7572 0.5865", "cc-pvtz", True),
                                             (WATER, "cc-pvdz", False)])
def test_vjp_of_every_class_is_the_adjoint_of_the_jvp(atom, basis, cart, omega):
    top, par, sa, atm, bas, env = tables(atom, basis, cart)
    env[8] = omega
    n = top.nao
    rng = np.random.default_rng(3)
    d = torch.as_tensor(rng.normal(size=(2, n, n)) / n, device="cuda")
    cot = torch.as_tensor(rng.normal(size=(2, 2, n, n)), device="cuda")
    slots = atm[:, 1][:, None] + np.arange(3)[None, :]
    u = np.zeros(len(env))
    u[slots.ravel()] = rng.normal(size=slots.size)
    plan = J.cached_plan(atm, bas, env, cart=cart, cutoff=0.0)

    def vjp(precision, cut):
        g = torch.empty((len(atm), 3), dtype=torch.float64, device="cuda")
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _capi.check(_capi.lib().b200jk_direct_jk_geom_vjp_precision(
            plan._h, ctypes.c_void_p(d.data_ptr()), 2, ctypes.c_void_p(cot.data_ptr()), 1, 1, precision, cut,
            ctypes.c_void_p(g.data_ptr()), stream))
        return g.cpu().numpy()

    g = vjp(_capi.FP64, 0.0)
    j, k = J.direct_jk_geometry_jvp(atm, bas, env, d, u, cart=cart)
    assert abs((g * u[slots]).sum() - (cot * torch.stack([j, k])).sum().item()) < 1e-12
    assert np.abs(vjp(_capi.SPLIT, 1e9) - g).max() < 1.7e-6 * np.abs(g).max()
