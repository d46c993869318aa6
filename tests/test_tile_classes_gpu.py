"""The tile path (blocks that do not fit one thread's registers: d and f shells): J, K and their combinations against
the packed integrals, contracted in torch.  Both sum the same n^2 FP64 products per element, in another order:
n^2 eps |element| < 1e-11 here.  Two waters give items whose last pass is ragged for every number of quartets a
block takes (12, 7, 4, 3, 2 or 1), triple zeta every class up to (ff|ff).  Split-precision bounds: test_small_builds_gpu."""
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
from tests.test_small_builds_gpu import PRECISIONS, packed_to_full  # noqa: E402


@pytest.fixture(scope="module", params=[(2, "cc-pvtz", False), (1, "cc-pvtz", True), (2, "cc-pvdz", True)])
def molecule(request):
    waters, basis, cart = request.param
    top, par, sa, atm, bas, env = tables(W.water_cluster(waters, 11), basis, cart)
    eri = packed_to_full(J.packed_eri(atm, bas, env, cart=cart, aosym="s4"), top.nao)
    return (atm, bas, env), cart, top.nao, eri


@pytest.mark.parametrize("with_j,with_k,hermi,nb", [(True, True, True, 1), (True, False, True, 3),
                                                    (False, True, True, 2), (True, True, False, 3),
                                                    (False, True, False, 1)])
@pytest.mark.parametrize("precision,cut,tol,rel", PRECISIONS)
def test_tile_classes_match_packed_integrals(molecule, with_j, with_k, hermi, nb, precision, cut, tol, rel):
    mol, cart, n, eri = molecule
    rng = np.random.default_rng(nb)
    d = torch.as_tensor(rng.normal(size=(nb, n, n)) / n, device=eri.device)
    if hermi:
        d = d + d.transpose(1, 2)
    j, k = J.DirectJKPlan([mol], cart=cart).jk(d, with_j=with_j, with_k=with_k, hermi=hermi, precision=precision,
                                               fp32_cut=cut)
    for on, x, path in ((with_j, j, "pqrs,ers->epq"), (with_k, k, "prqs,ers->epq")):
        y = torch.einsum(path, eri, d)
        assert not on or (x - y).abs().max().item() < tol + rel * y.abs().max().item()
