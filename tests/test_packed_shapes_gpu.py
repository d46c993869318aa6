"""Packed J/K at the edges of its tiles (32 x 32 of a row's triangle, 1024 columns and 128 rows of the pair
matrix) and of its density groups (three for J, two for K; no limit on their number), s4 and s8, symmetric and nonsymmetric densities,
against torch on the unpacked integrals.  The integrals need no basis: any symmetric pair matrix.  Both sides
sum up to n^2 products of order one in FP64; 4 n^2 eps max|element| bounds their difference."""
import sys
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs CUDA")]

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
from gradscf_b200 import jk as J  # noqa: E402


@pytest.mark.parametrize("layout", ["s4", "s8"])
@pytest.mark.parametrize("hermi", [True, False])
@pytest.mark.parametrize("n,nb", [(1, 1), (2, 3), (7, 2), (31, 1), (32, 4), (33, 2), (45, 5), (64, 1), (65, 3),
                                  (33, 200)])   # a batch of more than 6400 rows
def test_packed_jk_shapes(n, nb, hermi, layout):
    gen = torch.Generator(device="cuda").manual_seed(n * 8 + nb)
    npair = n * (n + 1) // 2
    m = torch.randn((npair, npair), dtype=torch.float64, device="cuda", generator=gen)
    m = m + m.T
    d = torch.randn((nb, n, n), dtype=torch.float64, device="cuda", generator=gen)
    if hermi:
        d = d + d.transpose(1, 2)
    else:
        d[0] = d[0] + d[0].T      # one symmetric density among the others
    i, j = torch.meshgrid(torch.arange(n, device="cuda"), torch.arange(n, device="cuda"), indexing="ij")
    pos = torch.maximum(i, j) * (torch.maximum(i, j) + 1) // 2 + torch.minimum(i, j)
    if layout == "s4":
        eri = m
    else:
        r, c = torch.tril_indices(npair, npair, device="cuda")
        eri = m[r, c]
    full = m[pos.reshape(-1)][:, pos.reshape(-1)].reshape(n, n, n, n)
    j0 = torch.einsum("pqrs,ers->epq", full, d)
    k0 = torch.einsum("prqs,ers->epq", full, d)
    tol = 4 * n * n * 2.3e-16 * 100.0
    for with_j, with_k in ((True, True), (True, False), (False, True)):
        jj, kk = J.packed_jk(eri, d, with_j=with_j, with_k=with_k)
        assert (jj - (j0 if with_j else 0 * j0)).abs().max().item() <= tol
        assert (kk - (k0 if with_k else 0 * k0)).abs().max().item() <= tol
