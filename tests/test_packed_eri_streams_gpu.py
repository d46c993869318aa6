"""Packed integrals of one plan from several host threads and streams at a time, and inside a captured graph: the same
integrals as a call alone.  Elements of diagonal shell pairs are written from both orders, which differ in rounding
(some hundred eps of integrals up to 5: below 1e-12); a lost order between the zeroing of the output and the kernels
loses whole integrals."""
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs CUDA")]

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
from gradscf_b200 import jk as J  # noqa: E402
from gradscf_b200 import workloads as W  # noqa: E402
from tests.gpu_util import tables  # noqa: E402


def test_packed_eri_from_threads_and_in_a_graph():
    atm, bas, env = tables(W.water_cluster(2, 3), "cc-pvdz", False)[3:]
    ref = J.packed_eri(atm, bas, env, cart=False)

    def call(_):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            out = [J.packed_eri(atm, bas, env, cart=False) for _ in range(4)]
            same = [(x - ref).abs().max().item() < 1e-12 for x in out]
        stream.synchronize()
        return same

    with ThreadPoolExecutor(max_workers=6) as pool:
        assert all(all(same) for same in pool.map(call, range(24)))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = J.packed_eri(atm, bas, env, cart=False)
    for _ in range(2):
        out.fill_(float("nan"))
        graph.replay()
        assert (out - ref).abs().max().item() < 1e-12
