"""Small cases at the edges of the kernels' tiles, steps and dispatch rules, against the CPU oracle or bit for bit against
another route to the same result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import quant  # noqa: E402
from test_cuda_moe import FULL, Layer, QT, check_layer, dev, make, pkg  # noqa: E402,F401


@pytest.mark.parametrize("n,dims", [(16, dict(H=128, E=2, K=2, F=128, S=128)), (17, dict(H=256, E=3, K=1, F=128, S=384)),
                                    (191, dict(H=128, E=2, K=2, F=128, S=128)), (192, dict(H=128, E=2, K=2, F=256, S=128)),
                                    (193, dict(H=384, E=2, K=2, F=128, S=256)), (385, dict(H=128, E=4, K=2, F=128, S=128))])
def test_fp16_grouped_gemm_at_tile_edges(pkg, port, n, dims):
    """fp16 weights by TMA: K of two blocks up (fewer than the ring's stages), ragged token tiles, one to several weight tiles."""
    L, hidden, resid = make(300 + n, dims, "f16", n)
    check_layer(pkg, port, L, hidden, resid, gemm=True)


def test_fp16_grouped_gemm_honours_a_mixed_layer(pkg, port):
    """Quantised experts beside an fp16 shared MLP: both weight operands of the kernel in one call."""
    L, hidden, resid = make(41, dict(H=256, E=4, K=2, F=128, S=256), "q8_0", 70, shared_qname="f16")
    check_layer(pkg, port, L, hidden, resid, gemm=True)
