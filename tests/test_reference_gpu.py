"""Packed integrals and direct J/K, full Coulomb and erf-attenuated, against an evaluation that shares no code or
method with the kernels (tests/md_reference.py).  J and K sum n^2 FP64 products of order one in another order:
n^2 eps |element| < 1e-11; the integrals themselves, some hundred eps of values up to 5, < 1e-12.  All quartets in
FP32 (a boundary above every bound): elements up to 6e-7 of the largest one were measured; four times that."""
import sys
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs CUDA")]

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
from gradscf_b200 import jk as J  # noqa: E402
from tests import md_reference  # noqa: E402
from tests.gpu_util import WATER, tables  # noqa: E402


@pytest.mark.parametrize("omega", [0.0, 0.33])
@pytest.mark.parametrize("basis,cart", [("sto-3g", False), ("6-31g*", True), ("cc-pvdz", False)])
def test_integrals_and_jk_match_an_independent_evaluation(basis, cart, omega):
    top, par, sa, atm, bas, env = tables(WATER, basis, cart)
    env[8] = omega
    n = top.nao
    eri = md_reference.eri(atm, bas, env, cart)
    i, j = np.tril_indices(n)
    s4 = eri[i[:, None], j[:, None], i[None], j[None]]
    assert np.abs(J.packed_eri(atm, bas, env, cart=cart, aosym="s4").cpu().numpy() - s4).max() < 1e-12
    a, b = np.tril_indices(len(s4))
    assert np.abs(J.packed_eri(atm, bas, env, cart=cart).cpu().numpy() - s4[a, b]).max() < 1e-12
    d = np.random.default_rng(4).normal(size=(2, n, n)) / n
    for dens in (d, d + d.transpose(0, 2, 1)):
        ref = (np.einsum("pqrs,ers->epq", eri, dens), np.einsum("prqs,ers->epq", eri, dens))
        for x, y in zip(J.direct_jk(atm, bas, env, dens, cart=cart), ref):
            assert np.abs(x.cpu().numpy() - y).max() < 1e-11
        for x, y in zip(J.direct_jk(atm, bas, env, dens, cart=cart, precision="split", fp32_cut=1e9), ref):
            assert np.abs(x.cpu().numpy() - y).max() < 2.4e-6 * np.abs(y).max()
