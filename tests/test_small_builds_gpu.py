"""Small builds, whose items hold few kets and share quartets among lanes: J/K of the direct build against the
packed integrals of the same molecule, contracted in torch (the packed integrals themselves are checked against an
independent evaluation in test_reference_gpu).  Both sum the same n^2 FP64 products per element; their different
orders differ by n^2 eps |element| < 1e-11 here.  Split precision: at the default boundary elements differ from the
FP64 build by up to 5e-12, with every quartet in FP32 by up to 9e-7 of the largest element (both measured over these
molecules and those of test_tile_classes_gpu); four times that on top of the FP64 bound.  With the attenuated operator the bounds of
pairs of p and d shells fall below the terms that cancel in them, whose rounding stays: 1.9e-10 at the default
boundary (the quadrature that these kernels replaced: 1.9e-10 too), four times that."""
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


# (precision, FP32 boundary, absolute bound, bound relative to the largest element)
PRECISIONS = [("fp64", 1e-6, 1e-11, 0.0), ("split", 1e-6, 3e-11, 0.0), ("split", 1e9, 1e-11, 3.6e-6)]


@pytest.mark.parametrize("omega", [0.0, 0.33])
@pytest.mark.parametrize("precision,cut,tol,rel", PRECISIONS)
@pytest.mark.parametrize("hermi", [True, False])
@pytest.mark.parametrize("waters,basis,cart", [(1, "sto-3g", False), (1, "6-31g*", True), (1, "cc-pvdz", False),
                                               (2, "cc-pvdz", False), (3, "6-31g*", False), (1, "cc-pvtz", False)])
def test_small_direct_builds_match_packed_integrals(waters, basis, cart, hermi, precision, cut, tol, rel, omega):
    top, par, sa, atm, bas, env = tables(W.water_cluster(waters, 5), basis, cart)
    env[8] = omega
    n = top.nao
    eri = packed_to_full(J.packed_eri(atm, bas, env, cart=cart, aosym="s4"), n)
    rng = np.random.default_rng(waters)
    d = torch.as_tensor(rng.normal(size=(2, n, n)) / n, device=eri.device)
    if hermi:
        d = d + d.transpose(1, 2)
    j0 = torch.einsum("pqrs,ers->epq", eri, d)
    k0 = torch.einsum("prqs,ers->epq", eri, d)
    j, k = J.DirectJKPlan([(atm, bas, env)], cart=cart).jk(d, hermi=hermi, precision=precision, fp32_cut=cut)
    if omega and precision == "split":
        tol = 8e-10
    for x, y in ((j, j0), (k, k0)):
        assert (x - y).abs().max().item() < tol + rel * y.abs().max().item()
