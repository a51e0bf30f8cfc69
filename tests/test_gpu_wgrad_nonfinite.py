"""The weight gradient with a non-finite cell: only the weights that the cell
meets inside the grid become non-finite.  A cell beyond the grid adds nothing,
whatever its partner holds (the zeros that pad the tiles are not numbers to be
multiplied)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import guess  # noqa: E402


def _reference(x, dy, dims):
    """Per tap, the sum over the cells whose neighbour there is in the grid
    (float64; x, dy channels-last)."""
    nx, ny, nz = dims
    X = x.double().view(nz, ny, nx, -1)
    Y = dy.double().view(nz, ny, nx, -1)
    out = []
    for t in range(27):
        d = (t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1)
        a = [slice(max(0, -o), m - max(0, o)) for o, m in zip(d, (nz, ny, nx))]
        b = [slice(max(0, o), m - max(0, -o)) for o, m in zip(d, (nz, ny, nx))]
        yc = Y[a[0], a[1], a[2]].reshape(-1, Y.shape[3])
        xc = X[b[0], b[1], b[2]].reshape(-1, X.shape[3])
        # (a product and a sum: a matrix product may pad with zeros as well)
        out.append((yc[:, :, None] * xc[:, None, :]).sum(0))
    return torch.stack(out)


# one whole 32 x BY tile; ragged tiles along x and y; both roles of the operands
@pytest.mark.parametrize("dims,cin,cout", [((32, 8, 6), 16, 16), ((20, 9, 7), 16, 16),
                                           ((33, 5, 6), 96, 32), ((20, 9, 7), 16, 48),
                                           ((20, 9, 7), 48, 16), ((1, 1, 3), 32, 32)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("which", ["x", "dy"])
def test_only_pairs_inside_the_grid_count(dims, cin, cout, value, which):
    nx, ny, nz = dims
    n = nx * ny * nz
    gen = torch.Generator().manual_seed(n + cin)
    X = torch.randn(n, cin, generator=gen).bfloat16().cuda()
    Y = torch.randn(n, cout, generator=gen).bfloat16().cuda()
    bulk = _reference(X.abs(), Y.abs(), dims)      # the sums' absolute terms
    mid = (nx // 2, ny // 2, nz // 2)
    cells = [mid, (0, mid[1], mid[2]), (nx - 1, mid[1], mid[2]), (mid[0], 0, mid[2]),
             (mid[0], ny - 1, mid[2]), (mid[0], mid[1], 0), (mid[0], mid[1], nz - 1),
             (0, 0, 0), (nx - 1, ny - 1, nz - 1)]
    for c in cells:
        x, y = X.clone(), Y.clone()
        (x if which == "x" else y)[c[0] + nx * (c[1] + ny * c[2]), 5] = value
        ref = _reference(x, y, dims)
        got = guess.conv3d_wgrad_raw(guess.blocked(x), guess.blocked(y), dims).double()
        assert torch.equal(got.isnan(), ref.isnan()), c
        assert torch.equal(got.isinf(), ref.isinf()), c
        inf = ref.isinf()
        assert torch.equal(got[inf], ref[inf]), c
        fin = torch.isfinite(ref)
        # FP32 sums of at most n exact products: n roundings of the absolute sum
        assert ((got - ref).abs()[fin] <= (n + 8) * 2.0 ** -24 * bulk[fin]).all(), c
    guess.check_errors()


def test_the_sums_are_added_to_what_is_there():
    """dw += with a non-finite cell at a face: the finite weights' earlier
    contents stay."""
    dims, n = (20, 9, 7), 20 * 9 * 7
    gen = torch.Generator().manual_seed(3)
    x = torch.randn(n, 16, generator=gen).bfloat16().cuda()
    y = torch.randn(n, 16, generator=gen).bfloat16().cuda()
    bulk = _reference(x.abs(), y.abs(), dims)
    x[0, 2] = float("inf")
    bx, by = guess.blocked(x), guess.blocked(y)
    dw = torch.full((27, 16, 16), 64.0, device="cuda")
    rc = guess._lib().hmfem_conv3d_wgrad(bx.data_ptr(), by.data_ptr(), dw.data_ptr(), *dims, 16,
                                         16, guess._err_buf(dw.device).data_ptr(),
                                         torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    guess.check_errors()
    ref = _reference(x, y, dims) + 64.0
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(dw), fin)
    assert ((dw.double() - ref).abs()[fin] <= (n + 8) * 2.0 ** -24 * (bulk[fin] + 64.0)).all()
