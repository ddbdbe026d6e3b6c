"""Routes that a rule on sizes picks, against the general route of the same call: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from owoinfer_b200 import ops as o
    return o


def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


@pytest.mark.parametrize("m", [1, 127, 256, 257, 297, 384, 512])
@pytest.mark.parametrize("n,k", [(64, 512), (1000, 528), (3072, 3072), (3064, 8192)])
def test_gemm_tiles_that_share_k_give_the_bits_of_whole_tiles(ops, m, n, k):
    """Few rows: AUTO takes tiles whose K range a cluster shares where whole ones would leave SMs idle. Edges: one row, the
    edges of 128- and 256-row tiles, columns that end inside a 64-column unit, K blocks that do not divide evenly."""
    g = _gen(m * 7 + n + k)
    x = torch.randint(-127, 128, (m, k), dtype=torch.int8, device="cuda", generator=g)
    w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    xs, ws = torch.rand(m, device="cuda", generator=g) * 1e-3, torch.rand(n, device="cuda", generator=g) * 1e-3
    bias, gate = (torch.randn(n, device="cuda", generator=g).bfloat16() for _ in range(2))
    res = torch.randn((m, n), device="cuda", generator=g).bfloat16()
    want, want_res = ops.int8_gemm(x, xs, w, ws, bias, tile=ops.TILE_128x128), res.clone()
    ops.int8_gemm_gated_residual(x, xs, w, ws, gate, want_res, tile=ops.TILE_128x128)
    got = ops.int8_gemm(x, xs, w, ws, bias)
    ops.int8_gemm_gated_residual(x, xs, w, ws, gate, res)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(res.view(torch.int16), want_res.view(torch.int16))
    assert ops.kernel_status() == (0, 0)
