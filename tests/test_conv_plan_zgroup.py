"""The forward convolution's grouped z taps, checked on the CPU: a numpy
emulation of the kernel's walk -- run columns, input planes, one operand per
plane and (dx, dy) pair that feeds up to three output planes lying next to
each other in tensor memory, N = COUT to 3 COUT at the ends, the weights as
[dx dy][dz][COUT], a plane's first MMA not accumulating -- must reproduce a
direct 3x3x3 convolution.  Accumulators start as NaN, so one that is read
before its first write shows, as does a row past the halo."""
import numpy as np
import pytest

from hmfem_b200 import guess
from test_conv_plan import SMEM_MAX, _check_limits, direct, emulate


def emulate_zg(x, w, dims, p):
    nx, ny, nz = dims
    cin, cout = x.shape[1], w.shape[1]
    W, H, bx, by, bz, rp = p["W"], p["H"], p["bx"], p["by"], p["bz"], p["rp"]
    grid = x.reshape(nz, ny, nx, cin)
    out = np.full((nz, ny, nx, cout), np.nan)
    written = np.zeros((nz, ny, nx), np.int32)
    offs = [(g % 3 - 1) + W * (g // 3 - 1) for g in range(9)]
    # the weight box [9][3][COUT][CIN]: tap (dz, g) = 9 dz + g
    wb = w.reshape(3, 9, cout, cin).transpose(1, 0, 2, 3).reshape(27 * cout, cin)
    for tz in range(p["ntz"]):
        for ty in range(p["nty"]):
            for tx in range(p["ntx"]):
                x0, y0, z0 = tx * bx - 1, ty * by - 1, tz * bz - 1
                halo = np.full((p["hcp"], cin), np.nan)
                hq = np.arange(p["hc"])
                zi, rem = divmod(hq, W * H)
                yi, xi = divmod(rem, W)
                gx, gy, gz = x0 + xi, y0 + yi, z0 + zi
                g = (gx >= 0) & (gx < nx) & (gy >= 0) & (gy < ny) & (gz >= 0) & (gz < nz)
                halo[:p["hc"]] = 0.0
                halo[hq[g]] = grid[gz[g], gy[g], gx[g]]
                acc = np.full((128, p["runs"] * cout), np.nan)

                def mma(col, row, wrow, ncols, accumulate, kc):
                    assert 0 <= row and row + 128 <= p["hcp"]
                    assert 0 <= col and col + ncols <= acc.shape[1]
                    assert 16 <= ncols <= 256 and wrow + ncols <= wb.shape[0]
                    d = halo[row:row + 128, kc] @ wb[wrow:wrow + ncols, kc].T
                    acc[:, col:col + ncols] = d + (acc[:, col:col + ncols] if accumulate else 0.0)

                for c in range(cin // 16):
                    kc = slice(16 * c, 16 * c + 16)
                    for j in range(rp):
                        row_j = 1 + (W * (j + 1) if p["row_mode"] else W + 128 * j)
                        for zi in range(bz + 2):
                            lo = 0 if zi < bz else zi - bz + 1
                            hi = zi if zi < 2 else 2
                            row = row_j + W * H * zi
                            col = (j * bz + bz - 1 - zi + lo) * cout
                            ncols = (hi - lo + 1) * cout
                            if c == 0 and zi < bz:     # the plane that starts here
                                mma(col, row + offs[0], 0, cout, False, kc)
                                if hi > 0:
                                    mma(col + cout, row + offs[0], cout, hi * cout, True, kc)
                            else:
                                mma(col, row + offs[0], lo * cout, ncols, True, kc)
                            for g in range(1, 9):
                                mma(col, row + offs[g], (3 * g + lo) * cout, ncols, True, kc)
                for r in range(p["runs"]):
                    if p["row_mode"]:
                        plane, line = divmod(r, by)
                        q0 = 1 + W * (line + 1) + W * H * (plane + 1)
                    else:
                        plane, j = divmod(r, rp)
                        line, q0 = -1, 1 + W + W * H * (plane + 1) + 128 * j
                    col = ((r - plane * rp) * bz + bz - 1 - plane) * cout
                    pos = q0 + np.arange(128)
                    zi, rem = divmod(pos, W * H)
                    yi, xi = divmod(rem, W)
                    gx, gy, gz = x0 + xi, y0 + yi, z0 + zi
                    v = (zi == plane + 1) & (yi >= 1) & (yi <= by) & (xi >= 1) & (xi <= bx)
                    if line >= 0:
                        v &= yi == line + 1
                    v &= (gx < nx) & (gy < ny) & (gz < nz)
                    out[gz[v], gy[v], gx[v]] = acc[v, col:col + cout]
                    written[gz[v], gy[v], gx[v]] += 1
    assert (written == 1).all()
    return out.reshape(-1, cout)


# a device of a few SMs groups taps on grids small enough to emulate: plane and
# row mode, several run columns, ragged tiles along y and z, one and
# several chunks of channels
@pytest.mark.parametrize("dims,cin,cout,nsm", [
    ((20, 16, 12), 16, 16, 2), ((20, 16, 12), 32, 32, 2), ((33, 20, 9), 96, 32, 4),
    ((12, 11, 13), 32, 16, 1), ((40, 9, 10), 16, 16, 1), ((130, 5, 9), 16, 16, 2),
    ((128, 9, 8), 16, 32, 2)])
def test_grouped_taps_match_direct_convolution(dims, cin, cout, nsm):
    p = guess.conv_plan(dims, cin, cout, nsm, SMEM_MAX)
    assert p["zg"] + p["xg"] == 1      # (32 -> 16 at 12x11x13: x taps)
    assert 3 * cout <= 256 and (p["xg"] or p["bz"] >= 4)
    _check_limits(p, cin, cout)
    rng = np.random.default_rng(sum(dims) + cin)
    n = dims[0] * dims[1] * dims[2]
    x = rng.standard_normal((n, cin))
    w = rng.standard_normal((27, cout, cin))
    out = emulate_zg(x, w, dims, p) if p["zg"] else emulate(x, w, dims, p)
    np.testing.assert_allclose(out, direct(x, w, dims), rtol=1e-12,
                               atol=1e-10)


def test_both_forms_are_chosen_by_the_planner():
    """The headline network's full-resolution layers group z taps, the flat
    grids do not; x and z taps are never grouped together."""
    seen = set()
    for dims in [(128, 128, 128), (64, 64, 64), (256, 256, 256), (20, 16, 12), (200, 4, 3)]:
        for cin, cout in sorted(guess._SHAPES):
            p = guess.conv_plan(dims, cin, cout)
            assert not (p["xg"] and p["zg"])
            seen.add((p["xg"], p["zg"]))
    assert seen == {(0, 0), (1, 0), (0, 1)}
