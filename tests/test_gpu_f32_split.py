"""The float32 product on the tensor cores (operands in three bfloat16 parts) against 64-bit products: over more than
one stage of k no further off than the FFMA kernel, at the edges of tiles, stages and rounds of tiles, and with numbers that
the parts cannot hold."""

import pytest
import torch

pytestmark = pytest.mark.gpu

BLOCKS = 148


def product(x, w, bias=None, out=None, blocks=BLOCKS):
    from from_scratch_inference_engine_b200.kernels import ops
    rows, n, k = x.shape[0], w.shape[0], w.shape[1]
    planes, notes = ops.gemm_f32_split_room(rows, n, k)
    out = torch.full((rows, n), float("nan"), device="cuda") if out is None else out
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.gemm_f32_split(x, w, bias, out, torch.empty(planes, dtype=torch.bfloat16, device="cuda"),
                             torch.full((notes,), 7, dtype=torch.int32, device="cuda"), error, blocks)
    assert error.item() == 0
    return got


def ffma(x, w, bias=None):
    from from_scratch_inference_engine_b200.kernels import ops
    return ops.gemm_f32(x, w, bias, kind="tiles")


def distance(got, want):
    return ((got.double() - want).norm() / want.norm().clamp_min(1e-300)).item()


# rows, n, k: single elements, edges of a tile (256) and of a stage (64), one stage per tile, several rounds
# of tiles on few pairs, k where the FFMA sums drift furthest, tiles for all pairs and more
SIZES = [(1, 1, 4), (5, 7, 8), (127, 129, 60), (128, 128, 64), (129, 255, 68), (256, 256, 128), (257, 513, 132),
         (300, 3000, 64), (49, 2048, 1536), (700, 1300, 2052), (64, 300, 18944), (1668, 17920, 1536)]


@pytest.mark.parametrize("rows,n,k", SIZES)
@pytest.mark.parametrize("held", ["any", "positive", "bfloat16", "mixed"])
def test_split_product(rows, n, k, held):
    torch.manual_seed(rows + n + k)
    x, w, bias = torch.randn(rows, k, device="cuda"), torch.randn(n, k, device="cuda"), torch.randn(n, device="cuda")
    if held == "positive":
        x, w = x.abs(), w.abs()
    elif held == "bfloat16":                 # the parts of w beyond the first are zero
        w = w.bfloat16().float()
    elif held == "mixed":                    # in some stages and rows only
        w[: n // 2] = w[: n // 2].bfloat16().float()
        w[:, : k // 8 * 4] = w[:, : k // 8 * 4].bfloat16().float()
        x *= torch.exp(4 * torch.randn(rows, 1, device="cuda"))
    want = x.double() @ w.double().T
    got = product(x, w)
    # Errors are measured against the sums of |x w|: where a sum cancels, what is left of it says nothing.  Over more
    # than one stage of k never further off than FFMA; within one, where FFMA has next to no error, the four truncated
    # steps of the stage may show: 4 x 2^-23 at most, half of that on average.
    size = x.abs().double() @ w.abs().double().T
    allowed = 2.0 ** -22 if k <= 64 else 0.0

    def off(got, want, size):
        return ((got.double() - want).norm() / size.norm()).item()
    assert off(got, want, size) <= max(off(ffma(x, w), want, size), allowed)
    # no single output is far off either: of operands of both signs by the steps of a stage and its sum, of positive ones,
    # whose stages all err to one side, by a few more roundings of a long sum
    assert ((got.double() - want).abs() / size).max().item() < (2e-6 if held == "positive" else 5 * 2.0 ** -23)
    size = size + bias.double().abs()
    biased = product(x, w, bias, blocks=6 if rows < 1000 else BLOCKS)   # three pairs: several tiles each
    want += bias.double()
    assert off(biased, want, size) <= max(off(ffma(x, w, bias), want, size), allowed)
    alone = product(x[rows // 2:rows // 2 + 1].contiguous(), w)
    assert torch.equal(alone[0], got[rows // 2])


@pytest.mark.parametrize("parts", [2, 3])
def test_whole_numbers_are_exact(parts):
    """Whole numbers whose sums stay below 2^24 come out exactly: a plane of w that either block's tensor core reads
    before its warps have filled it, in any stage, tile or launch, changes a result.  w is another one at every launch and
    needs `parts` planes; three pairs of blocks have several tiles each."""
    torch.manual_seed(parts)
    rows, n, k = 300, 2000, 1536
    x = torch.randint(-3, 4, (rows, k), device="cuda").float()
    if parts == 3:                               # 20 bits of w: room for few terms
        x = torch.where(torch.rand(rows, k, device="cuda") < 4 / k, x.clamp(-1, 1), torch.zeros_like(x))
        assert x.abs().sum(1).max() < 16
    for launch in range(30):
        w = torch.randint(-2 ** (11 if parts == 2 else 20), 2 ** (11 if parts == 2 else 20), (n, k), device="cuda").float()
        got = product(x, w, blocks=(6, BLOCKS)[launch % 2])
        assert torch.equal(got.double(), x.double() @ w.double().T)


@pytest.mark.parametrize("offset", [1, 4])
def test_split_product_of_views(offset):
    """x as columns of a wider matrix, the result into one whose rows do (4) or do not (1) start on 16 bytes."""
    torch.manual_seed(offset)
    wide, w = torch.randn(200, 140, device="cuda"), torch.randn(131, 132, device="cuda")
    room = torch.full((200, 140 + offset), float("nan"), device="cuda")
    x = wide[:, 4:136]
    product(x, w, None, room[:, offset:offset + 131])
    want = x.double() @ w.double().T
    assert distance(room[:, offset:offset + 131], want) < 2e-7
    assert torch.isnan(room[:, :offset]).all() and torch.isnan(room[:, offset + 131:]).all()


def test_split_product_of_infinities():
    """Infinite, NaN, overflowing and largest inputs give what the FFMA kernel gives."""
    torch.manual_seed(2)
    x, w = torch.randn(300, 200, device="cuda"), torch.randn(600, 200, device="cuda")
    x[3, 5], x[40, 7], x[200, 9] = float("inf"), float("nan"), -float("inf")
    x[260, 11], w[17, 11] = 3.4e38, 0.5          # finite, but rounds to infinity as bfloat16
    x[261], w[300] = 1e30, 1e30                  # overflows in the sum
    got, want = product(x, w), ffma(x, w)
    same = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got[~same & ~torch.isnan(want)], want[~same & ~torch.isnan(want)])
    quiet = torch.ones(300, dtype=torch.bool, device="cuda")
    quiet[[3, 40, 200, 260, 261]] = False
    exact = x[quiet].double() @ w.double().T
    keep = torch.ones(600, dtype=torch.bool, device="cuda")
    keep[300] = False
    assert distance(got[quiet][:, keep], exact[:, keep]) < 4e-7


@pytest.mark.parametrize("x_power,w_power", [(-115, 0), (0, -118), (-117, -20), (-75, -75), (-140, 40), (60, -130), (70, -70),
                                             (40, 0), (22, 22), (23, 24), (63, 63), (90, -90), (-120, 100), (127, -127)])
def test_split_product_of_small_and_large_numbers(x_power, w_power):
    """Operands of any size, subnormal numbers and results among them: no further off than FFMA, which rounds at every
    k (a unit of the smallest result beside it); sums that overflow are infinite in both."""
    torch.manual_seed(x_power + w_power)
    rows, n, k = 130, 270, 192
    x = ((torch.rand(rows, k, device="cuda").double() + 1) * 2.0 ** x_power).float()
    w = (torch.randn(n, k, device="cuda").double() * 2.0 ** w_power).float()
    assert torch.isfinite(x).all() and torch.isfinite(w).all()
    got, plain, want = product(x, w), ffma(x, w), x.double() @ w.double().T
    finite = torch.isfinite(plain)
    assert torch.equal(torch.isfinite(got), finite)
    torch.testing.assert_close(got[~finite], plain[~finite], rtol=0, atol=0, equal_nan=True)
    off = [(v.double() - want)[finite].norm().item() for v in (got, plain)]
    assert off[0] <= off[1] + 2.0 ** -150 * got.numel() ** 0.5


@pytest.mark.parametrize("bias", [False, True])
def test_rows_beside_infinities_keep_their_bits(bias):
    """A row with an infinity, a NaN, an overflow in its sums or in its planes changes no bit of the rows beside it."""
    torch.manual_seed(4)
    x, w = torch.randn(260, 320, device="cuda"), torch.randn(300, 320, device="cuda")
    b = torch.randn(300, device="cuda") if bias else None
    calm = product(x, w, b)
    rows = torch.ones(260, dtype=torch.bool, device="cuda")
    for row, value in ((3, float("inf")), (70, float("nan")), (130, 3e38), (131, 1e25), (259, -float("inf"))):
        x[row, 9], rows[row] = value, False
    got = product(x, w, b)
    assert torch.equal(got[rows], calm[rows])
    assert not torch.isfinite(got[[3, 70, 259]]).any() and not torch.isfinite(got[130]).all()
    assert torch.isfinite(got[131]).all()                # beyond the room of the planes, not of float32
    size = x[131].double().abs() @ w.double().abs().T
    want = x[131].double() @ w.double().T + (b.double() if bias else 0)
    assert ((got[131].double() - want).abs() <= 2e-6 * size).all()


def test_split_product_refuses():
    from from_scratch_inference_engine_b200.kernels.ops import KernelError
    with pytest.raises(KernelError):
        product(torch.randn(64, 6, device="cuda"), torch.randn(8, 6, device="cuda"))
    with pytest.raises(KernelError):
        product(torch.randn(64, 13, device="cuda")[:, 1:9], torch.randn(8, 8, device="cuda"))


@pytest.mark.parametrize("rows,n,k", [(49, 64, 16), (64, 16384, 4), (300, 5000, 8), (2048, 4096, 32), (17, 17920, 64),
                                      (48, 17920, 256)])
@pytest.mark.parametrize("sign", ["normal", "positive"])
def test_products_over_a_short_k_lose_nothing(rows, n, k, sign):
    """What a step's product of these sizes gives is no further from 64 bits than FFMA (whichever of its kernels
    takes the rows), also where the sums of a stage, truncated, would be."""
    from from_scratch_inference_engine_b200.engine.runtime import Runtime
    from from_scratch_inference_engine_b200.kernels import ops
    torch.manual_seed(rows + k)
    x, w = torch.randn(rows, k, device="cuda"), torch.randn(n, k, device="cuda")
    if sign == "positive":
        x, w = x.abs(), w.abs()
    want = x.double() @ w.double().T
    got = Runtime(dtype="float32").linear(x, w, None)
    assert distance(got, want) <= distance(ops.gemm_f32(x, w, None), want)
