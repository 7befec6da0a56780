"""The float32 product of few rows: rows of w in turn through one block, chunks of x, every number of rows per warp."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows of x at the edges of a block's 1, 2, 4, 8 and 16; one chunk of x, several, and a short last one (2,048 elements
# up to 4 rows, 1,024 up to 8, 512 beyond); fewer rows of w than one warp has, ragged ones, and more than
# all SMs hold at once, with one chunk and with several
@pytest.mark.parametrize("rows_per_warp", [0, 1, 2, 4])
@pytest.mark.parametrize("m,n,k", [(1, 3, 4), (1, 9603, 2048), (2, 9603, 2052), (3, 20001, 2176), (4, 70, 8960), (5, 20001, 1028),
                                   (8, 9603, 1536), (9, 20001, 516), (16, 300, 3588), (17, 9603, 640), (48, 77, 132),
                                   (8, 592, 1028), (5, 593, 1028), (6, 100, 1024), (2, 150001, 132)])
def test_few_rows(m, n, k, rows_per_warp):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(m + n + k)
    x, w, bias = (torch.randn(shape, generator=generator, device="cuda") for shape in ((m, k + 4), (n, k), (n,)))
    x = x[:, 4:]
    want = x.double() @ w.double().T + bias.double()
    out = torch.full((m, n + 3), float("nan"), device="cuda")
    ops.gemm_f32(x, w, bias, out=out[:, :n], kind="rows", rows_per_warp=rows_per_warp)
    # 32 partial sums of k / 32 products each, then a tree of 5: at most (k / 32 + 6) roundings of 2^-24 of the sum of |x w|
    bound = (k / 32 + 6) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + bias.double().abs())
    assert ((out[:, :n].double() - want).abs() <= bound).all()
    assert torch.isnan(out[:, n:]).all()
    # the order of the sums depends on neither the rows beside a row nor the rows per warp
    alone = ops.gemm_f32(x[m // 2:m // 2 + 1], w, bias, kind="rows")
    assert torch.equal(alone[0], out[m // 2, :n])
