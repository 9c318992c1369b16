"""Short reduced axes: rows of one to eight vectors on teams of two to eight lanes, kept indexes walked in
tiles whose last ones are smaller, outer reductions with a warp to a tile, grids of a block for every few
rows or 256 vectors.  Against 64-bit arithmetic; maxima, moves and integer sums exactly."""
import pytest
import torch

import inductor_x_b200  # noqa: F401

pytestmark = pytest.mark.gpu
# sums of n terms of size one in 32 bits, rounded once to the type
EPS = {torch.float32: 2.0 ** -22, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def compiled(fn, *args):
    torch._dynamo.reset()
    return torch.compile(fn, dynamic=False)(*args)


def data(cuda, shape, dtype):
    g = torch.Generator(device=cuda).manual_seed(sum(shape))
    return (torch.rand(*shape, generator=g, device=cuda) * 2 - 1).to(dtype)


def close(got, want, dtype, terms):
    scale = want.abs().clamp_min(float(want.square().mean().sqrt()))
    assert float(((got.double() - want).abs() / scale).max()) <= EPS[dtype] * (4 if dtype != torch.float32 else 4 + terms ** 0.5)


# extents of the two kept digits below, at and past one tile of 16, and past several; rows of one vector to 24
@pytest.mark.parametrize("b,c,dtype,d", [(2, 15, torch.float32, 4), (33, 16, torch.float32, 16), (16, 17, torch.bfloat16, 64),
                                         (130, 70, torch.float16, 24), (47, 31, torch.float32, 96)])
def test_rows_in_smaller_tiles(cuda, b, c, dtype, d):
    x = data(cuda, (37, b, c, d), dtype)
    close(compiled(lambda x: x.permute(0, 2, 1, 3).sum(3), x), x.double().permute(0, 2, 1, 3).sum(3), dtype, d)


# the same where so much is read that the smaller tiles at the ends are taken
@pytest.mark.parametrize("shape,dtype", [((200, 33, 70, 96), torch.float32), ((37, 130, 1000, 16), torch.float32), ((100, 47, 700, 64), torch.float16)])
def test_rows_in_smaller_tiles_of_large_operands(cuda, shape, dtype):
    x = data(cuda, shape, dtype)
    assert torch.equal(compiled(lambda x: x.permute(0, 2, 1, 3).amax(3), x), x.permute(0, 2, 1, 3).amax(3))


# 1, 2 (ragged), 4, 5 and 6 vectors of four; one row, rows for a few blocks, and more than three batches of
# what is resident (blocks that see one batch)
@pytest.mark.parametrize("d", [4, 7, 16, 20, 24])
def test_rows_of_a_few_vectors(cuda, d):
    for rows in (1, 1003, 300007):
        x = data(cuda, (rows, d), torch.float32)
        close(compiled(lambda x: x.sum(-1), x), x.double().sum(-1), torch.float32, d)
        y = compiled(lambda x: torch.softmax(x, -1), x)
        assert float((y.double() - torch.softmax(x.double(), -1)).abs().max()) <= 1e-6


# 7 and 8 vectors of four: four lanes of two, and a team of eight
@pytest.mark.parametrize("d", [28, 32])
def test_rows_of_seven_and_eight_vectors(cuda, d):
    test_rows_of_a_few_vectors(cuda, d)


# steps of the reduced axis around those of a warp's thread rows (8, 4, 2 and 1 of them) and of a batch of
# four, tiles enough for a warp each
@pytest.mark.parametrize("dtype,r,d", [(torch.bfloat16, 2, 32), (torch.bfloat16, 33, 32), (torch.float16, 26, 128), (torch.float32, 9, 100)])
def test_outer_reductions_with_a_warp_to_a_tile(cuda, dtype, r, d):
    x = data(cuda, (4003, r, d), dtype)
    assert torch.equal(compiled(lambda x: x.amax(1), x), x.amax(1))
    if r == 33:
        close(compiled(lambda x: x.sum(1), x), x.double().sum(1), dtype, r)
        i = (x * 1000).to(torch.int32)
        assert torch.equal(compiled(lambda i: i.sum(1), i), i.sum(1))


@pytest.mark.parametrize("n", [1, 2041, 3000001])
def test_grids_of_a_block_for_256_vectors(cuda, n):
    a, b = data(cuda, (n,), torch.bfloat16), data(cuda, (n,), torch.bfloat16)
    assert torch.equal(compiled(lambda a, b: a + b, a, b), a + b)
    if n > 1:   # bases off a boundary
        assert torch.equal(compiled(lambda a, b: a + b, a[1:], b[1:]), a[1:] + b[1:])


@pytest.mark.parametrize("dtype,shape", [(torch.float16, (3, 320, 64)), (torch.float32, (5, 128, 96))])
def test_register_tiles(cuda, dtype, shape):
    x = data(cuda, shape, dtype)
    assert torch.equal(compiled(lambda x: (x.transpose(1, 2) + 1.0).contiguous(), x), x.transpose(1, 2) + 1.0)
