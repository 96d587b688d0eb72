"""CPU emulation of the shared-memory layouts of two tcgen05 kernels (csrc/sf_conv_tc.cuh): the z-line convolution with
three taps an MMA from one x plane a stage, and the weight gradient with M = 64, with a box a tap pair or one halo'd box for nine.
The emulation places TMA boxes as the unit does (out-of-grid elements zero), reads the operands through the descriptors'
addressing, multiplies as the MMA does, and compares with a direct convolution; every byte read lies in its buffer, and the
first MMA on an accumulator overwrites it."""
import numpy as np
import pytest

from test_tc_layouts import SLACK, _const, _direct_forward, _read_plain, _read_sw32, _write_sw32

LZ, LX = _const("kLineZ"), _const("kLineX")


@pytest.mark.parametrize("shape,ci,co,Y", [((4, 6, 128), 16, 16, 4), ((3, 7, 130), 16, 32, 4), ((3, 6, 128), 32, 16, 4),
                                           ((3, 9, 150), 32, 32, 4), ((4, 10, 128), 16, 16, 8), ((3, 17, 129), 32, 16, 8)])
def test_line_kernel_plane_stages(shape, ci, co, Y):
    nx, ny, nz = shape
    kp = ci // 16
    rng = np.random.default_rng(1)
    X = rng.standard_normal(shape + (ci,))
    W = rng.standard_normal((27, co, ci))
    Wp = np.stack([W[3 * (t % 9) + t // 9] for t in range(27)])  # taps (dz, dx, dy)
    stage_bytes = LZ * (Y + 2) * 32
    wch = (27 * co * 32 + 1023) // 1024 * 1024
    wbuf = np.zeros(kp * wch // 2)
    for c in range(kp):
        _write_sw32(wbuf, c * wch, Wp[:, :, 16 * c:16 * c + 16].reshape(-1, 16))
    Xp = np.zeros((nx + 3 + LX, ny + 2 + Y, nz + 2 + LZ, ci))
    Xp[1:1 + nx, 1:1 + ny, 1:1 + nz] = X
    out = np.zeros((nx, ny, nz, co))
    bz_n, by_n, bx_n = -(-nz // LZ), -(-ny // Y), -(-nx // LX)
    for br in range(bz_n * by_n * bx_n):
        z0, y0, x0 = LZ * (br % bz_n), Y * ((br // bz_n) % by_n), LX * (br // (bz_n * by_n))
        acc = np.full((128, Y * LX * co), np.nan)

        def mma(col, a_at, b_at, n, add, stage):
            A, ma = _read_sw32(stage, a_at, 128)
            B, mb = _read_sw32(wbuf, b_at, n)
            assert ma < stage_bytes and mb < (b_at // wch + 1) * wch and 0 <= col and col + n <= acc.shape[1]
            assert n % 16 == 0 and n <= 256 and b_at % 256 == 0
            acc[:, col:col + n] = A @ B.T + (acc[:, col:col + n] if add else 0.0)

        for st in range(3 * kp):
            dz, jp = st // kp, st % kp
            for xb in range(LX + 2):
                stage = np.zeros(stage_bytes // 2)
                _write_sw32(stage, 0, Xp[x0 + xb, y0:y0 + Y + 2, z0 + dz:z0 + dz + LZ,
                                         16 * jp:16 * jp + 16].reshape(-1, 16))
                for xx in range(LX):
                    dx = xb - xx
                    if dx < 0 or dx > 2:
                        continue
                    b0 = jp * wch + (9 * dz + 3 * dx) * co * 32
                    first = dx == 0 and st == 0
                    if first:
                        for yb in range(Y):
                            mma((xx * Y + Y - 1 - yb) * co, 4096 * yb, b0, co, False, stage)
                    for yb in range(Y + 2):
                        lo, dy1 = (0 if yb < Y else yb - Y + 1), min(yb, 2)
                        dy0 = 1 if first and lo == 0 else lo
                        if dy0 <= dy1:
                            mma((xx * Y + Y - 1 - (yb - dy0)) * co, 4096 * yb, b0 + dy0 * co * 32, (dy1 - dy0 + 1) * co,
                                True, stage)
        for xt in range(LX):
            for yt in range(Y):
                if x0 + xt < nx and y0 + yt < ny:
                    zz = min(LZ, nz - z0)
                    col = (xt * Y + Y - 1 - yt) * co
                    out[x0 + xt, y0 + yt, z0:z0 + zz] = acc[:zz, col:col + co]
    ref = _direct_forward(X, W)
    assert np.abs(out - ref).max() <= 1e-9 * np.abs(ref).max()


@pytest.mark.parametrize("shape,ci,co,halo", [((4, 6, 32), 16, 16, True), ((5, 7, 40), 16, 32, True),
                                              ((4, 9, 26), 16, 16, True), ((3, 5, 40), 16, 32, False),
                                              ((3, 5, 26), 32, 16, False), ((2, 4, 32), 64, 64, False)])
def test_weight_gradient_m64(shape, ci, co, halo):
    nx, ny, nz = shape
    bx = 2 if ci == 16 else 1
    N = 3 * ci
    rng = np.random.default_rng(2)
    X = rng.standard_normal(shape + (ci,))
    dY = rng.standard_normal(shape + (co,))
    nzh = (nz + 7) // 8

    def chmajor(src, C, shifts):  # [zh][x][y][shift, c][8 z]
        out = np.zeros((nzh, nx, ny, len(shifts), C, 8))
        for s, sh in enumerate(shifts):
            for z in range(nz):
                if 0 <= z + sh < nz:
                    out[z // 8, :, :, s, :, z % 8] = src[:, :, z + sh, :]
        return out.reshape(nzh, nx, ny, len(shifts) * C, 8)

    def box(T, y, x, zh0, by, bxx, bz):
        b = np.zeros((bz, bxx, by) + T.shape[3:])
        for a in range(bz):
            for i in range(bxx):
                for j in range(by):
                    if 0 <= zh0 + a < nzh and 0 <= x + i < nx and 0 <= y + j < ny:
                        b[a, i, j] = T[zh0 + a, x + i, y + j]
        return b.reshape(-1)

    dYT, XT = chmajor(dY, co, [0]), chmajor(X, ci, [-1, 0, 1])
    a_bytes = 256 * co * bx
    acc = np.zeros((9, 64, N))
    bz_n, by_n, bx_n = -(-nz // 32), -(-ny // 4), -(-nx // bx)
    for br in range(bz_n * by_n * bx_n):
        z0, y0, x0 = 32 * (br % bz_n), 4 * ((br // bz_n) % by_n), bx * (br // (bz_n * by_n))
        abuf = np.concatenate([box(dYT, y0, x0, z0 // 8, 4, bx, 4), np.zeros(SLACK // 2)])
        if halo:
            for jj in range(4):
                bbuf = box(XT, y0 - 1, x0 - 1, z0 // 8 + jj, 6, bx + 2, 1)
                for dx in range(3):
                    for p in range(2 * bx):  # p = y / 2 + 2 x
                        A, ma = _read_plain(abuf, 16 * (jj * 4 * bx * co + 2 * p * co), co * 16, 128, 64)
                        B, mb = _read_plain(bbuf, 16 * (2 * (p % 2) + 6 * (p // 2 + dx)) * N, N * 16, 128, 3 * N)
                        assert ma < a_bytes + SLACK and mb < bbuf.size * 2
                        acc[3 * dx:3 * dx + 3] += (A @ B.T).reshape(64, 3, N).transpose(1, 0, 2)
        else:
            for pr in range(9):
                bbuf = box(XT, y0 + pr % 3 - 1, x0 + pr // 3 - 1, z0 // 8, 4, bx, 4)
                for p in range(8 * bx):
                    A, ma = _read_plain(abuf, 2 * p * co * 16, co * 16, 128, 64)
                    B, mb = _read_plain(bbuf, 2 * p * N * 16, N * 16, 128, N)
                    assert ma < a_bytes + SLACK and mb < bbuf.size * 2
                    acc[pr] += A @ B.T
    got = np.zeros((27, co, ci))
    for pr in range(9):
        for sz in range(3):
            got[3 * pr + sz] = acc[pr, :co, sz * ci:(sz + 1) * ci]
    Xp = np.pad(X, ((1, 1), (1, 1), (1, 1), (0, 0)))
    ref = np.zeros((27, co, ci))
    for t in range(27):
        dx, dy, dz = t // 9, (t // 3) % 3, t % 3
        ref[t] = np.einsum("xyzo,xyzi->oi", dY, Xp[dx:dx + nx, dy:dy + ny, dz:dz + nz])
    assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
