"""Small builds, whose items hold few kets and share quartets among lanes: J/K of the direct build against the
packed integrals of the same molecule, contracted in torch.  Both sum the same n^2 FP64 products per element;
their different orders differ by n^2 eps |element| < 1e-11 here."""
import sys
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs CUDA")]

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
from gradscf_b200 import jk as J  # noqa: E402
from gradscf_b200 import workloads as W  # noqa: E402
from tests.gpu_util import tables  # noqa: E402


def packed_to_full(eri, n):
    i, j = torch.meshgrid(torch.arange(n), torch.arange(n), indexing="ij")
    pos = (torch.maximum(i, j) * (torch.maximum(i, j) + 1) // 2 + torch.minimum(i, j)).reshape(-1).to(eri.device)
    return eri[pos][:, pos].reshape(n, n, n, n)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("split", 2e-6)])   # split: FP32 quartets below 1e-6
@pytest.mark.parametrize("hermi", [True, False])
@pytest.mark.parametrize("waters,basis,cart", [(1, "sto-3g", False), (1, "6-31g*", True), (1, "cc-pvdz", False),
                                               (2, "cc-pvdz", False), (3, "6-31g*", False), (1, "cc-pvtz", False)])
def test_small_direct_builds_match_packed_integrals(waters, basis, cart, hermi, precision, tol):
    top, par, sa, atm, bas, env = tables(W.water_cluster(waters, 5), basis, cart)
    n = top.nao
    eri = packed_to_full(J.packed_eri(atm, bas, env, cart=cart, aosym="s4"), n)
    rng = np.random.default_rng(waters)
    d = torch.as_tensor(rng.normal(size=(2, n, n)) / n, device=eri.device)
    if hermi:
        d = d + d.transpose(1, 2)
    j0 = torch.einsum("pqrs,ers->epq", eri, d)
    k0 = torch.einsum("prqs,ers->epq", eri, d)
    j, k = J.DirectJKPlan([(atm, bas, env)], cart=cart).jk(d, hermi=hermi, precision=precision)
    assert (j - j0).abs().max().item() < tol
    assert (k - k0).abs().max().item() < tol
