"""CPU emulation of the tile-staged smoothers and residual (opentm_b200/csrc/otm_tile.cuh, otm_ctile.cuh).

The kernels' index arithmetic is restated here line by line (tile origins of both tilings, the
periodic wrap of shifted tiles, the parity-split and padded shared-memory site order, the thread ->
register-block mapping and which of a pass's neighbours come from the block, the six-plane streaming of
a pass, the right-hand side's two-wide loads, the staged coarse block and the quad-wise prolongation, the
write-back from registers; on coarse levels also the copies of the stencils into shared memory) and every
shared-memory and global access is checked to stay in bounds before the kernels run on a GPU.
Within a pass no thread may read the values (.xyz) of a site that another thread writes in the
same pass, and the write-back must cover each vertex once. The emulated arithmetic is then compared
with an independent block Gauss-Seidel (whole 27-point rows, colour pairs in order, halo frozen,
tiles of either tiling) and an independent residual, so the streaming algebra (which plane's
conductivities feed which coefficient) is checked too."""
import numpy as np
import pytest

TX, TY, TZ = 16, 16, 8  # interior vertices of a tile
SX, SY, SZ = TX + 2, TY + 2, TZ + 2
SHALF = SX // 2
SROW = SX + 1  # padded row pitch
SPLANE, SSITES = SROW * SY, SROW * SY * SZ
THREADS, SEG, RTHREADS = 128, 4, 256
CX, CY, CZ = TX // 2 + 2, TY // 2 + 2, TZ // 2 + 2
CSITES = CX * CY * CZ
OP = dict(c0=0.35, c2=-0.08, c3=-0.095)  # distinct c2 / c3 so that a mix-up shows
NBR = [(-1, -1), (0, -1), (1, -1), (-1, 0), (1, 0), (-1, 1), (0, 1), (1, 1)]


def wrapm(a, n):
    assert -n <= a < 2 * n
    return a + n if a < 0 else (a - n if a >= n else a)


def tsite(lx, ly, lz):
    assert 0 <= lx < SX and 0 <= ly < SY and 0 <= lz < SZ
    return lz * SPLANE + ly * SROW + ((SHALF + (lx >> 1)) if (lx & 1) else (lx >> 1))


def rsite(lx, ly, lz):
    assert 0 <= lx < SX and 0 <= ly < SY and 0 <= lz < SZ
    return lz * SPLANE + ly * SROW + lx


def gidx(d, x, y, z):
    nx, ny, nz = d
    assert 0 <= x < nx and 0 <= y < ny and 0 <= z < nz
    return x + nx * (y + ny * z)


def tile_origin(d, b, shift):
    nx, ny, nz = d
    ntx, nty = nx // TX, ny // TY
    q = b // ntx
    return ((b - q * ntx) * TX + shift * (TX // 2), (q % nty) * TY + shift * (TY // 2),
            (q // nty) * TZ + shift * (TZ // 2))


def plane_coef(K):
    c2, c3 = OP["c2"], OP["c3"]
    return [c3 * K[0], c2 * (K[0] + K[1]), c3 * K[1], c2 * (K[0] + K[2]), c2 * (K[1] + K[3]), c3 * K[2],
            c2 * (K[2] + K[3]), c3 * K[3]]


class Smem:
    """Shared memory of one CTA with access checks."""

    def __init__(self, n):
        self.v = np.zeros((n, 4))
        self.n = n
        self.writes = {}
        self.reads = {}

    def rd(self, i, who, comp="xyzw"):
        assert 0 <= i < self.n, i
        self.reads.setdefault(i, set()).add((who, comp))
        return self.v[i]

    def wr(self, i, val, who):
        assert 0 <= i < self.n, i
        self.writes.setdefault(i, set()).add(who)
        self.v[i] = val

    def check_pass(self):
        for i, ws in self.writes.items():
            assert len(ws) == 1, f"site {i} written by {ws}"
            (w,) = ws
            for (who, comp) in self.reads.get(i, ()):
                assert who == w or comp == "w", f"site {i} written by {w}, read by {who}"
        self.writes, self.reads = {}, {}


class Block:
    """A thread's register block: 2 x 2 columns from (lx, ly), planes lz0 .. lz0 + 3; value of column
    c = cx + 2 cy, plane q in v[c][q] (u of the three cases and the conductivity)."""

    def __init__(self, sm, t):
        self.lx, self.ly, self.lz0 = 2 * (t & 7) + 1, 2 * ((t >> 3) & 7) + 1, 1 + SEG * (t >> 6)
        assert self.lx + 1 <= TX and self.ly + 1 <= TY and self.lz0 + SEG - 1 <= TZ
        self.v = [[list(sm.rd(tsite(self.lx + (c & 1), self.ly + (c >> 1), self.lz0 + q), t)) for q in range(SEG)]
                  for c in range(4)]


def tile_rhs(d, f, blk, x0, y0, z0, py):
    """tile_rhs<PY>: the right-hand side of row py of the block, both columns by one 8-byte load."""
    nx, ny, nz = d
    nv = nx * ny * nz
    X, Y = wrapm(x0 + blk.lx - 1, nx), wrapm(y0 + blk.ly - 1 + py, ny)
    out = []
    for q in range(SEG):
        g = gidx(d, X, Y, wrapm(z0 + blk.lz0 - 1 + q, nz))
        assert g % 2 == 0 and X + 1 < nx, "an aligned pair inside the row"
        out.append([(f[c * nv + g], f[c * nv + g + 1]) for c in range(3)])
    return out


def emulate_pass(sm, blocks, rhs, px, py, last, fs):
    """tile_pass<PX, PY, kLast>: every thread updates column (px, py) of its block, 6 planes streamed."""
    oL, oR = (SHALF - 1, SHALF) if px else (-SHALF, -SHALF + 1)
    kcol = px + 2 * py
    for t in range(THREADS):
        own = blocks[t]
        lx, ly, lz0 = own.lx, own.ly, own.lz0
        cx0, cy0 = lx + px, ly + py
        # the compile-time neighbour offsets equal the site order's
        assert tsite(cx0 - 1, cy0, 1) - tsite(cx0, cy0, 1) == oL and tsite(cx0 + 1, cy0, 1) - tsite(cx0, cy0, 1) == oR
        col = tsite(cx0, cy0, lz0 - 1)
        Kp, Cp = [0.0] * 4, None
        accA, accB, accC = [0.0] * 3, [0.0] * 3, [0.0] * 3
        dA = dB = 0.0
        for s in range(SEG + 2):
            P = lz0 - 1 + s
            b = col + s * SPLANE
            assert b == tsite(cx0, cy0, P)
            nb = []
            for ox, oy in NBR:
                cx, cy = px + ox, py + oy
                if 1 <= s <= SEG and 0 <= cx <= 1 and 0 <= cy <= 1:
                    nb.append(own.v[cx + 2 * cy][s - 1])
                else:
                    i = b + (oL if ox < 0 else (oR if ox > 0 else 0)) + oy * SROW
                    assert i == tsite(cx0 + ox, cy0 + oy, P)
                    nb.append(sm.rd(i, t))
            kown = 0.0
            if 1 <= s <= SEG:
                kown = own.v[kcol][s - 1][3]
            elif s == 0:
                kown = sm.rd(b, t, "w")[3]
            K = [nb[0][3], nb[1][3], nb[3][3], kown]
            sK = (K[0] + K[1]) + (K[2] + K[3])
            C = plane_coef(K) if s <= SEG else None
            dC = 0.0
            if s < SEG:
                accC = [rhs[t][s][c][px] * fs[c] for c in range(3)]
                for n in range(8):
                    for c in range(3):
                        accC[c] -= C[n] * nb[n][c]
                dC = sK
            if 1 <= s <= SEG:
                for q, n in enumerate((0, 2, 5, 7)):
                    w = OP["c2"] * (Kp[q] + K[q])
                    for c in range(3):
                        accB[c] -= w * nb[n][c]
                dB += sK
            if s >= 2:
                for n in range(8):
                    for c in range(3):
                        accA[c] -= Cp[n] * nb[n][c]
                inv = 1.0 / (OP["c0"] * dA)
                own.v[kcol][s - 2][:3] = [accA[c] * inv for c in range(3)]
                if not last:
                    sm.wr(tsite(cx0, cy0, lz0 + s - 2), own.v[kcol][s - 2], t)
            accA, accB = accB, accC
            accC = [0.0] * 3
            dA, dB = dB, dC
            Kp, Cp = K, C
    sm.check_pass()


def prolong_site(cb, ux, uy, uz, c0x, c0y, c0z):
    ax0, ay0, az0 = (ux >> 1) - c0x, (uy >> 1) - c0y, (uz >> 1) - c0z
    ax1, ay1, az1 = ax0 + (ux & 1), ay0 + (uy & 1), az0 + (uz & 1)
    for a, n in ((ax0, CX), (ax1, CX), (ay0, CY), (ay1, CY), (az0, CZ), (az1, CZ)):
        assert 0 <= a < n
    wx1, wy1, wz1 = [0.5 if (q & 1) else 0.0 for q in (ux, uy, uz)]
    wx0, wy0, wz0 = 1 - wx1, 1 - wy1, 1 - wz1
    r00, r10 = (ay0 + CY * az0) * CX, (ay1 + CY * az0) * CX
    r01, r11 = (ay0 + CY * az1) * CX, (ay1 + CY * az1) * CX
    out = []
    for c in range(3):
        u = cb[:, c]
        out.append(wz0 * (wy0 * (wx0 * u[r00 + ax0] + wx1 * u[r00 + ax1]) +
                          wy1 * (wx0 * u[r10 + ax0] + wx1 * u[r10 + ax1])) +
                   wz1 * (wy0 * (wx0 * u[r01 + ax0] + wx1 * u[r01 + ax1]) +
                          wy1 * (wx0 * u[r11 + ax0] + wx1 * u[r11 + ax1])))
    return out


def prolong_quad(cb, xs, uy, uz, c0x, c0y, c0z):
    """The quad-wise prolongation: 3 coarse columns per coarse row, 4 fine sites."""
    assert xs % 2 == 0
    ax = (xs >> 1) - c0x
    ay0, az0 = (uy >> 1) - c0y, (uz >> 1) - c0z
    ay1, az1 = ay0 + (uy & 1), az0 + (uz & 1)
    wy1, wz1 = (0.5 if uy & 1 else 0.0), (0.5 if uz & 1 else 0.0)
    wy0, wz0 = 1 - wy1, 1 - wz1
    rows = [(ay0 + CY * az0) * CX + ax, (ay1 + CY * az0) * CX + ax, (ay0 + CY * az1) * CX + ax,
            (ay1 + CY * az1) * CX + ax]
    for r in rows:
        assert 0 <= r and r + 2 < CSITES and (r % CX) + 2 < CX
    v = [[cb[r + a] for a in range(3)] for r in rows]
    # each coarse column interpolated over (y, z), then over x: even sites take a column, odd
    # sites the mean of two
    col = [[wz0 * (wy0 * v[0][a][c] + wy1 * v[1][a][c]) + wz1 * (wy0 * v[2][a][c] + wy1 * v[3][a][c])
            for c in range(3)] for a in range(3)]
    out = [col[0], [0.5 * (col[0][c] + col[1][c]) for c in range(3)], col[1],
           [0.5 * (col[1][c] + col[2][c]) for c in range(3)]]
    # the values of the per-site prolongation, summed in another order
    for e in range(4):
        ref = prolong_site(cb, xs + e, uy, uz, c0x, c0y, c0z)
        assert all(abs(out[e][c] - ref[c]) <= 1e-6 * (1.0 + abs(ref[c])) for c in range(3))
    return out


def emulate_sweep(d, dc, ks, u_in, uc, f, start, shift, reverse, fs=(1.0, 1.0, 1.0)):
    """k_tile_sweep<start> over all tiles of tiling `shift`. start: 0 zero, 1 u_in, 2 u_in + P uc."""
    nx, ny, nz = d
    nv = nx * ny * nz
    ntiles = (nx // TX) * (ny // TY) * (nz // TZ)
    out = np.full(3 * nv, np.nan)
    written = np.zeros(nv, dtype=int)
    pos = sorted(tsite(lx, ly, lz) for lz in range(SZ) for ly in range(SY) for lx in range(SX))
    assert len(set(pos)) == SX * SY * SZ and pos[-1] < SSITES, "the site order is one-to-one and in bounds"
    for b in range(ntiles):
        x0, y0, z0 = tile_origin(d, b, shift)
        sm = Smem(SSITES)
        c0x, c0y, c0z = x0 // 2 - 1, y0 // 2 - 1, z0 // 2 - 1
        cb = np.zeros((CSITES, 4))
        if start == 2:
            cnx, cny, cnz = dc
            nvc = cnx * cny * cnz
            for s in range(CSITES):
                ax, ay, az = s % CX, (s // CX) % CY, s // (CX * CY)
                g = gidx(dc, wrapm(c0x + ax, cnx), wrapm(c0y + ay, cny), wrapm(c0z + az, cnz))
                cb[s] = [uc[g], uc[nvc + g], uc[2 * nvc + g], 0.0]
        staged = {}
        for w in range(SY * SZ * (TX // 4)):
            q, row = w & 3, w >> 2
            ly, lz = row % SY, row // SY
            uy, uz = y0 - 1 + ly, z0 - 1 + lz
            g = gidx(d, wrapm(x0 + 4 * q, nx), wrapm(uy, ny), wrapm(uz, nz))
            assert g % 4 == 0 and g + 3 < nv and (g + 3) // nx == g // nx  # one aligned 4-wide vector in a row
            p = prolong_quad(cb, x0 + 4 * q, uy, uz, c0x, c0y, c0z) if start == 2 else None
            for e in range(4):
                v = [0.0, 0.0, 0.0, ks[g + e]]
                if start >= 1:
                    v = [u_in[c * nv + g + e] for c in range(3)] + [ks[g + e]]
                if start == 2:
                    v = [v[c] + p[e][c] for c in range(3)] + [ks[g + e]]
                i = tsite(1 + 4 * q + e, ly, lz)
                staged[i] = staged.get(i, 0) + 1
                sm.wr(i, v, -1)
        for w in range(SY * SZ * 2):
            side, row = w & 1, w >> 1
            ly, lz = row % SY, row // SY
            lx = SX - 1 if side else 0
            ux, uy, uz = x0 - 1 + lx, y0 - 1 + ly, z0 - 1 + lz
            g = gidx(d, wrapm(ux, nx), wrapm(uy, ny), wrapm(uz, nz))
            v = [0.0, 0.0, 0.0, ks[g]]
            if start >= 1:
                v = [u_in[c * nv + g] for c in range(3)] + [ks[g]]
            if start == 2:
                p = prolong_site(cb, ux, uy, uz, c0x, c0y, c0z)
                v = [v[c] + p[c] for c in range(3)] + [ks[g]]
            i = tsite(lx, ly, lz)
            staged[i] = staged.get(i, 0) + 1
            sm.wr(i, v, -1)
        assert len(staged) == SX * SY * SZ and set(staged.values()) == {1}, "every site staged once"
        sm.writes, sm.reads = {}, {}
        blocks = [Block(sm, t) for t in range(THREADS)]
        sm.writes, sm.reads = {}, {}
        pa = 1 if reverse else 0
        pb = 1 - pa
        rhs = [tile_rhs(d, f, blk, x0, y0, z0, pa) for blk in blocks]
        emulate_pass(sm, blocks, rhs, pa, pa, False, fs)
        rhs2 = [tile_rhs(d, f, blk, x0, y0, z0, pb) for blk in blocks]
        emulate_pass(sm, blocks, rhs, pb, pa, False, fs)
        emulate_pass(sm, blocks, rhs2, pa, pb, False, fs)
        emulate_pass(sm, blocks, rhs2, pb, pb, True, fs)
        for blk in blocks:
            X = wrapm(x0 + blk.lx - 1, nx)
            for q in range(SEG):
                for e in range(2):
                    g = gidx(d, X, wrapm(y0 + blk.ly - 1 + e, ny), wrapm(z0 + blk.lz0 - 1 + q, nz))
                    assert g % 2 == 0 and X + 1 < nx
                    for px in range(2):
                        written[g + px] += 1
                        for c in range(3):
                            out[c * nv + g + px] = blk.v[2 * e + px][q][c]
    assert (written == 1).all()
    return out


def emulate_resid(d, ks, u, f, fs=(1.0, 1.0, 1.0)):
    """k_tile_resid over all tiles of tiling 0: 256 threads, one column each, 10 planes streamed."""
    nx, ny, nz = d
    nv = nx * ny * nz
    r = np.full(3 * nv, np.nan)
    written = np.zeros(nv, dtype=int)
    for b in range((nx // TX) * (ny // TY) * (nz // TZ)):
        x0, y0, z0 = tile_origin(d, b, 0)
        sm = np.full((SSITES, 4), np.nan)
        for w in range(SY * SZ * (TX // 4)):
            q, row = w & 3, w >> 2
            ly, lz = row % SY, row // SY
            g = gidx(d, wrapm(x0 + 4 * q, nx), wrapm(y0 - 1 + ly, ny), wrapm(z0 - 1 + lz, nz))
            for e in range(4):
                sm[rsite(1 + 4 * q + e, ly, lz)] = [u[g + e], u[nv + g + e], u[2 * nv + g + e], ks[g + e]]
        for w in range(SY * SZ * 2):
            side, row = w & 1, w >> 1
            ly, lz = row % SY, row // SY
            lx = SX - 1 if side else 0
            g = gidx(d, wrapm(x0 - 1 + lx, nx), wrapm(y0 - 1 + ly, ny), wrapm(z0 - 1 + lz, nz))
            sm[rsite(lx, ly, lz)] = [u[g], u[nv + g], u[2 * nv + g], ks[g]]
        for t in range(RTHREADS):
            lx, ly = 1 + (t & 15), 1 + (t >> 4)
            pl = nx * ny
            col = gidx(d, x0 + lx - 1, y0 + ly - 1, z0)
            fn = [f[c * nv + col] for c in range(3)]  # right-hand side of vertex P + 1
            Kp, Cp = [0.0] * 4, None
            accA, accB, accC = [0.0] * 3, [0.0] * 3, [0.0] * 3
            dA = dB = 0.0
            uA, uB = [0.0] * 3, [0.0] * 3
            for P in range(SZ):
                b0 = rsite(lx, ly, P)
                offs = [-SROW - 1, -SROW, -SROW + 1, -1, 1, SROW - 1, SROW, SROW + 1]
                for n, (ox, oy) in enumerate(NBR):
                    assert b0 + offs[n] == rsite(lx + ox, ly + oy, P)
                nb = [sm[b0 + o] for o in offs]
                own = sm[b0]
                assert not np.isnan(own).any() and not any(np.isnan(x).any() for x in nb), "read a staged site"
                K = [nb[0][3], nb[1][3], nb[3][3], own[3]]
                sK = (K[0] + K[1]) + (K[2] + K[3])
                C = plane_coef(K)
                dC = 0.0
                if P + 1 <= TZ:
                    accC = [fn[c] * fs[c] for c in range(3)]
                    if P + 2 <= TZ:
                        assert col + (P + 1) * pl < nv
                        fn = [f[c * nv + col + (P + 1) * pl] for c in range(3)]
                    for n in range(8):
                        for c in range(3):
                            accC[c] -= C[n] * nb[n][c]
                    dC = sK
                if 1 <= P <= TZ:
                    for q, n in enumerate((0, 2, 5, 7)):
                        w = OP["c2"] * (Kp[q] + K[q])
                        for c in range(3):
                            accB[c] -= w * nb[n][c]
                    dB += sK
                    uB = list(own[:3])
                if P >= 2:
                    for n in range(8):
                        for c in range(3):
                            accA[c] -= Cp[n] * nb[n][c]
                    diag = OP["c0"] * dA
                    g = col + (P - 2) * pl
                    assert 0 <= g < nv
                    written[g] += 1
                    for c in range(3):
                        r[c * nv + g] = accA[c] - diag * uA[c]
                accA, accB, accC = accB, accC, [0.0] * 3
                uA = uB
                dA, dB = dB, dC
                Kp, Cp = K, C
    assert (written == 1).all()
    return r


# ---- independent restatements: whole 27-point rows ----------------------------------------
def row_coefs(d, ks, x, y, z):
    """A(v, v+o) for the 27 offsets of vertex (x,y,z) with c1 = 0."""
    nx, ny, nz = d
    k8 = {}
    for bz in (0, 1):
        for by in (0, 1):
            for bx in (0, 1):
                k8[(bx, by, bz)] = ks[gidx(d, (x - 1 + bx) % nx, (y - 1 + by) % ny, (z - 1 + bz) % nz)]
    c = {0: OP["c0"], 1: 0.0, 2: OP["c2"], 3: OP["c3"]}
    out = {}
    for oz in (-1, 0, 1):
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                nzc = (ox != 0) + (oy != 0) + (oz != 0)
                ssum = 0.0
                for (bx, by, bz), kv in k8.items():
                    ok = all((o > 0 and b == 1) or (o < 0 and b == 0) or o == 0
                             for o, b in ((ox, bx), (oy, by), (oz, bz)))
                    if ok:
                        ssum += kv
                out[(ox, oy, oz)] = c[nzc] * ssum
    return out


def block_gs(d, ks, u0, f, order, shift):
    """One colour-pair Gauss-Seidel sweep per 16 x 16 x 8 block of tiling `shift` (blocks shifted by
    half a block along every axis for shift 1, wrapping periodically), the halo (every neighbour
    outside the block, periodic images of the block's own vertices included) frozen at u0."""
    nx, ny, nz = d
    nv = nx * ny * nz
    sx, sy, sz = shift * TX // 2, shift * TY // 2, shift * TZ // 2
    out = u0.copy()
    for z0 in range(sz, nz + sz, TZ):
        for y0 in range(sy, ny + sy, TY):
            for x0 in range(sx, nx + sx, TX):
                loc = u0.copy()
                for p in order:
                    px, py = p & 1, p >> 1
                    for z in range(z0, z0 + TZ):
                        for y in range(y0 + py, y0 + TY, 2):
                            for x in range(x0 + px, x0 + TX, 2):
                                A = row_coefs(d, ks, x % nx, y % ny, z % nz)
                                v = gidx(d, x % nx, y % ny, z % nz)
                                for c in range(3):
                                    s = f[c * nv + v]
                                    for (ox, oy, oz), a in A.items():
                                        if (ox, oy, oz) == (0, 0, 0):
                                            continue
                                        inside = (x0 <= x + ox < x0 + TX and y0 <= y + oy < y0 + TY
                                                  and z0 <= z + oz < z0 + TZ)
                                        src = loc if inside else u0  # the halo stays at u0
                                        s -= a * src[c * nv + gidx(d, (x + ox) % nx, (y + oy) % ny, (z + oz) % nz)]
                                    loc[c * nv + v] = s / A[(0, 0, 0)]
                for z in range(z0, z0 + TZ):
                    for y in range(y0, y0 + TY):
                        for x in range(x0, x0 + TX):
                            v = gidx(d, x % nx, y % ny, z % nz)
                            for c in range(3):
                                out[c * nv + v] = loc[c * nv + v]
    return out


def residual(d, ks, u, f):
    nx, ny, nz = d
    nv = nx * ny * nz
    r = np.zeros(3 * nv)
    for z in range(nz):
        for y in range(ny):
            for x in range(nx):
                A = row_coefs(d, ks, x, y, z)
                v = gidx(d, x, y, z)
                for c in range(3):
                    s = f[c * nv + v]
                    for (ox, oy, oz), a in A.items():
                        s -= a * u[c * nv + gidx(d, (x + ox) % nx, (y + oy) % ny, (z + oz) % nz)]
                    r[c * nv + v] = s
    return r


def prolong(d, dc, uc):
    nx, ny, nz = d
    cnx, cny, cnz = dc
    nv, nvc = nx * ny * nz, cnx * cny * cnz
    out = np.zeros(3 * nv)
    for z in range(nz):
        for y in range(ny):
            for x in range(nx):
                v = gidx(d, x, y, z)
                for c in range(3):
                    a = 0.0
                    for (X, wx) in ((x // 2, 1.0),) if x % 2 == 0 else ((x // 2, 0.5), ((x // 2 + 1) % cnx, 0.5)):
                        for (Y, wy) in ((y // 2, 1.0),) if y % 2 == 0 else ((y // 2, 0.5), ((y // 2 + 1) % cny, 0.5)):
                            for (Z, wz) in ((z // 2, 1.0),) if z % 2 == 0 else ((z // 2, 0.5), ((z // 2 + 1) % cnz, 0.5)):
                                a += wx * wy * wz * uc[c * nvc + gidx(dc, X, Y, Z)]
                    out[c * nv + v] = a
    return out


@pytest.fixture(scope="module")
def fields():
    rng = np.random.default_rng(7)
    d = (32, 16, 16)  # two tiles along x and z: halos cross tile faces, shifted tiles wrap
    dc = (16, 8, 8)
    nv, nvc = 32 * 16 * 16, 16 * 8 * 8
    ks = 0.001 + rng.random(nv)
    f = rng.standard_normal(3 * nv)
    u_in = rng.standard_normal(3 * nv)
    uc = rng.standard_normal(3 * nvc)
    return d, dc, ks, f, u_in, uc


def test_sweep_from_zero_forward_tiling0(fields):
    d, dc, ks, f, u_in, uc = fields
    got = emulate_sweep(d, dc, ks, None, None, f, start=0, shift=0, reverse=False)
    ref = block_gs(d, ks, np.zeros_like(f), f, (0, 1, 2, 3), 0)
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


def test_sweep_from_u_forward_shifted_tiling(fields):
    d, dc, ks, f, u_in, uc = fields
    got = emulate_sweep(d, dc, ks, u_in, None, f, start=1, shift=1, reverse=False)
    ref = block_gs(d, ks, u_in, f, (0, 1, 2, 3), 1)
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


def test_sweep_with_prolongation_reverse_shifted_tiling(fields):
    d, dc, ks, f, u_in, uc = fields
    got = emulate_sweep(d, dc, ks, u_in, uc, f, start=2, shift=1, reverse=True)
    ref = block_gs(d, ks, u_in + prolong(d, dc, uc), f, (3, 2, 1, 0), 1)
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


def test_residual_indices_and_values(fields):
    d, dc, ks, f, u_in, uc = fields
    got = emulate_resid(d, ks, u_in, f)
    ref = residual(d, ks, u_in, f)
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


# ---- coarse levels: otm_ctile.cuh -----------------------------------------------------------
CTX, CTY, CTZ = 16, 8, 8
CSX, CSY, CSZ = CTX + 2, CTY + 2, CTZ + 2
CSHALF, CSROW = CSX // 2, CSX + 1
CSPLANE, CSSITES = CSROW * CSY, CSROW * CSY * CSZ
CTHREADS = (CTX // 2) * (CTY // 2) * (CTZ // 2)
CCX, CCY, CCZ = CTX // 2 + 2, CTY // 2 + 2, CTZ // 2 + 2
CCSITES = CCX * CCY * CCZ


def csite(lx, ly, lz):
    assert 0 <= lx < CSX and 0 <= ly < CSY and 0 <= lz < CSZ
    return lz * CSPLANE + ly * CSROW + ((CSHALF + (lx >> 1)) if (lx & 1) else (lx >> 1))


def ctile_origin(d, b, shift):
    nx, ny, nz = d
    ntx, nty = nx // CTX, ny // CTY
    q = b // ntx
    return ((b - q * ntx) * CTX + shift * (CTX // 2), (q % nty) * CTY + shift * (CTY // 2),
            (q // nty) * CTZ + shift * (CTZ // 2))


def cb_index(d, x, y, z):
    nx, ny, nz = d
    hx, hy = nx // 2, ny // 2
    colour = (x & 1) + 2 * (y & 1) + 4 * (z & 1)
    return colour * (nx * ny * nz // 8) + (x >> 1) + hx * ((y >> 1) + hy * (z >> 1))


def cprolong_site(cb, ux, uy, uz, c0x, c0y, c0z):
    ax0, ay0, az0 = (ux >> 1) - c0x, (uy >> 1) - c0y, (uz >> 1) - c0z
    ax1, ay1, az1 = ax0 + (ux & 1), ay0 + (uy & 1), az0 + (uz & 1)
    for a, n in ((ax0, CCX), (ax1, CCX), (ay0, CCY), (ay1, CCY), (az0, CCZ), (az1, CCZ)):
        assert 0 <= a < n
    wx1, wy1, wz1 = [0.5 if (q & 1) else 0.0 for q in (ux, uy, uz)]
    wx0, wy0, wz0 = 1 - wx1, 1 - wy1, 1 - wz1
    r = lambda ay, az: (ay + CCY * az) * CCX
    out = []
    for c in range(3):
        u = cb[:, c]
        out.append(wz0 * (wy0 * (wx0 * u[r(ay0, az0) + ax0] + wx1 * u[r(ay0, az0) + ax1]) +
                          wy1 * (wx0 * u[r(ay1, az0) + ax0] + wx1 * u[r(ay1, az0) + ax1])) +
                   wz1 * (wy0 * (wx0 * u[r(ay0, az1) + ax0] + wx1 * u[r(ay0, az1) + ax1]) +
                          wy1 * (wx0 * u[r(ay1, az1) + ax0] + wx1 * u[r(ay1, az1) + ax1])))
    return out


def emulate_csweep(d, dc, st, u_in, uc, f, start, shift, reverse):
    """k_ctile_sweep<start> over all coarse tiles of tiling `shift`."""
    nx, ny, nz = d
    nv = nx * ny * nz
    out = np.full(3 * nv, np.nan)
    written = np.zeros(nv, dtype=int)
    pos = [csite(lx, ly, lz) for lz in range(CSZ) for ly in range(CSY) for lx in range(CSX)]
    assert len(set(pos)) == len(pos) and max(pos) < CSSITES
    for b in range((nx // CTX) * (ny // CTY) * (nz // CTZ)):
        x0, y0, z0 = ctile_origin(d, b, shift)
        c0x, c0y, c0z = x0 // 2 - 1, y0 // 2 - 1, z0 // 2 - 1
        cb = np.zeros((CCSITES, 4))
        if start == 2:
            cnx, cny, cnz = dc
            nvc = cnx * cny * cnz
            for q in range(CCSITES):
                ax, ay, az = q % CCX, (q // CCX) % CCY, q // (CCX * CCY)
                g = gidx(dc, wrapm(c0x + ax, cnx), wrapm(c0y + ay, cny), wrapm(c0z + az, cnz))
                cb[q] = [uc[g], uc[nvc + g], uc[2 * nvc + g], 0.0]
        sm = Smem(CSSITES)
        for q in range(CSX * CSY * CSZ):
            lx, ly, lz = q % CSX, (q // CSX) % CSY, q // (CSX * CSY)
            ux, uy, uz = x0 - 1 + lx, y0 - 1 + ly, z0 - 1 + lz
            v = [0.0, 0.0, 0.0, 0.0]
            if start >= 1:
                g = gidx(d, wrapm(ux, nx), wrapm(uy, ny), wrapm(uz, nz))
                v = [u_in[c * nv + g] for c in range(3)] + [0.0]
                if start == 2:
                    p = cprolong_site(cb, ux, uy, uz, c0x, c0y, c0z)
                    v = [v[c] + p[c] for c in range(3)] + [0.0]
            sm.wr(csite(lx, ly, lz), v, -1)
        sm.writes, sm.reads = {}, {}
        order = list(range(8))[::-1] if reverse else list(range(8))
        for col in order:
            cx, cy, cz = col & 1, (col >> 1) & 1, col >> 2
            oL, oR = (-CSHALF, -CSHALF + 1) if cx == 0 else (CSHALF - 1, CSHALF)
            for t in range(CTHREADS):
                i, j, k = t & 7, (t >> 3) & 3, t >> 5
                lx, ly, lz = 1 + 2 * i + cx, 1 + 2 * j + cy, 1 + 2 * k + cz
                X, Y, Z = wrapm(x0 + lx - 1, nx), wrapm(y0 + ly - 1, ny), wrapm(z0 + lz - 1, nz)
                v = gidx(d, X, Y, Z)
                sb = cb_index(d, X, Y, Z)
                assert 0 <= sb < nv
                s = [st[o * nv + sb] for o in range(27)]
                acc = [f[c * nv + v] for c in range(3)]
                base = csite(lx, ly, lz)
                for o in range(27):
                    if o == 13:
                        continue
                    ox, oy, oz = o % 3 - 1, (o // 3) % 3 - 1, o // 9 - 1
                    off = (oL if ox < 0 else (oR if ox > 0 else 0)) + oy * CSROW + oz * CSPLANE
                    assert base + off == csite(lx + ox, ly + oy, lz + oz)
                    n = sm.rd(base + off, t)
                    for c in range(3):
                        acc[c] -= s[o] * n[c]
                sm.wr(base, [acc[c] / s[13] for c in range(3)] + [0.0], t)
            sm.check_pass()
        for q in range(CTX * CTY * CTZ):
            lx, ly, lz = 1 + q % CTX, 1 + (q // CTX) % CTY, 1 + q // (CTX * CTY)
            g = gidx(d, wrapm(x0 + lx - 1, nx), wrapm(y0 + ly - 1, ny), wrapm(z0 + lz - 1, nz))
            written[g] += 1
            o = sm.v[csite(lx, ly, lz)]
            for c in range(3):
                out[c * nv + g] = o[c]
    assert (written == 1).all()
    return out


# few tiles: k_ctile_sweep_small
SMALL_THREADS = 3 * CTHREADS
SMALL_ROW = 20
SMALL_PLANE, SMALL_CASE = SMALL_ROW * CSY, SMALL_ROW * CSY * CSZ
SMALL_STENCILS = 8 * 27 * CTHREADS


def cspos(lx, ly, lz):
    assert 0 <= lx < CSX and 0 <= ly < CSY and 0 <= lz < CSZ
    return lz * SMALL_PLANE + ly * SMALL_ROW + ((CSHALF + (lx >> 1)) if (lx & 1) else (lx >> 1))


def small_stencils(d, st, x0, y0, z0, reverse):
    """The copies of a CTA's stencils, 16 bytes each, and after which copy group each word has landed."""
    nx, ny, nz = d
    nv, nsub = nx * ny * nz, nx * ny * nz // 8
    hx, hy, hz = nx // 2, ny // 2, nz // 2
    sm = np.full(SMALL_STENCILS, np.nan)
    group = np.full(SMALL_STENCILS, -1)
    for warp in range(SMALL_THREADS // 32):
        for lane in range(32):
            h, r = lane & 1, lane >> 1
            X, Y, Z = wrapm(x0 // 2 + 4 * h, hx), wrapm(y0 // 2 + (r & 3), hy), wrapm(z0 // 2 + (r >> 2), hz)
            src, dst = X + hx * (Y + hy * Z), r * 8 + h * 4
            assert X + 4 <= hx, "half a row never crosses the periodic boundary"
            q = warp
            for p in range(8):
                c = 7 - p if reverse else p
                for _ in range(3):
                    if q < 27 * (p + 1):
                        o = q - 27 * p
                        assert 0 <= o < 27
                        a, g = dst + (c * 27 + o) * CTHREADS, src + o * nv + c * nsub
                        assert a % 4 == 0 and g % 4 == 0 and 0 <= g and g + 3 < 27 * nv
                        assert (group[a:a + 4] == -1).all(), "every word copied once"
                        sm[a:a + 4], group[a:a + 4] = st[g:g + 4], p
                        q += SMALL_THREADS // 32
            assert q >= 27 * 8
    assert (group >= 0).all()
    return sm, group


def emulate_csmall(d, dc, st, u_in, uc, f, start, shift, reverse):
    """k_ctile_sweep_small<start, reverse> over all coarse tiles of tiling `shift`: a lane per vertex of a
    colour and load case, stencils in shared memory."""
    nx, ny, nz = d
    nv = nx * ny * nz
    out = np.full(3 * nv, np.nan)
    written = np.zeros(3 * nv, dtype=int)
    pos = [cspos(lx, ly, lz) for lz in range(CSZ) for ly in range(CSY) for lx in range(CSX)]
    assert len(set(pos)) == len(pos) and max(pos) < SMALL_CASE
    for b in range((nx // CTX) * (ny // CTY) * (nz // CTZ)):
        x0, y0, z0 = ctile_origin(d, b, shift)
        st_sm, group = small_stencils(d, st, x0, y0, z0, reverse)
        c0x, c0y, c0z = x0 // 2 - 1, y0 // 2 - 1, z0 // 2 - 1
        cb = np.zeros((CCSITES, 4))
        if start == 2:
            cnx, cny, cnz = dc
            nvc = cnx * cny * cnz
            for q in range(3 * CCSITES):
                c, s = q // CCSITES, q % CCSITES
                ax, ay, az = s % CCX, (s // CCX) % CCY, s // (CCX * CCY)
                cb[s, c] = uc[c * nvc + gidx(dc, wrapm(c0x + ax, cnx), wrapm(c0y + ay, cny), wrapm(c0z + az, cnz))]
        sites = np.full(3 * SMALL_CASE, np.nan)
        nsites = CSX * CSY * CSZ
        for q in range(3 * nsites):
            c, s = q // nsites, q % nsites
            lx, ly, lz = s % CSX, (s // CSX) % CSY, s // (CSX * CSY)
            ux, uy, uz = x0 - 1 + lx, y0 - 1 + ly, z0 - 1 + lz
            v = u_in[c * nv + gidx(d, wrapm(ux, nx), wrapm(uy, ny), wrapm(uz, nz))] if start >= 1 else 0.0
            if start == 2:
                v += cprolong_site(cb, ux, uy, uz, c0x, c0y, c0z)[c]
            sites[c * SMALL_CASE + cspos(lx, ly, lz)] = v
        for p in range(8):
            C = 7 - p if reverse else p
            cx, cy, cz = C & 1, (C >> 1) & 1, C >> 2
            oL, oR = (-CSHALF, -CSHALF + 1) if cx == 0 else (CSHALF - 1, CSHALF)
            reads, writes = [], {}
            for t in range(SMALL_THREADS):
                warp, lane = t >> 5, t & 31
                i, j, k, cs = lane & 7, lane >> 3, warp & 3, warp >> 2
                X, Y, Z = (wrapm(x0 + 2 * i + cx, nx), wrapm(y0 + 2 * j + cy, ny), wrapm(z0 + 2 * k + cz, nz))
                sp = C * 27 * CTHREADS + i + 8 * j + 32 * k
                assert (group[sp:sp + 27 * CTHREADS:CTHREADS] <= p).all(), "the pass waits for its copies"
                assert all(st_sm[sp + o * CTHREADS] == st[o * nv + cb_index(d, X, Y, Z)] for o in (0, 13, 26))
                base = cs * SMALL_CASE + cspos(1 + 2 * i + cx, 1 + 2 * j + cy, 1 + 2 * k + cz)
                acc = f[cs * nv + gidx(d, X, Y, Z)]
                for o in range(27):
                    if o == 13:
                        continue
                    ox, oy, oz = o % 3 - 1, (o // 3) % 3 - 1, o // 9 - 1
                    off = (oL if ox < 0 else (oR if ox > 0 else 0)) + oy * SMALL_ROW + oz * SMALL_PLANE
                    assert base + off == cs * SMALL_CASE + cspos(1 + 2 * i + cx + ox, 1 + 2 * j + cy + oy, 1 + 2 * k + cz + oz)
                    reads.append(base + off)
                    acc -= st_sm[sp + o * CTHREADS] * sites[base + off]
                assert base not in writes
                writes[base] = acc / st_sm[sp + 13 * CTHREADS]
            assert not set(reads) & set(writes), "no lane reads what another writes in the pass"
            for a, v in writes.items():
                sites[a] = v
        for t in range(SMALL_THREADS):
            cs = t // CTHREADS
            for it in range(CTX * CTY * CTZ // CTHREADS):
                s = t - cs * CTHREADS + it * CTHREADS
                lx, ly, lz = 1 + s % CTX, 1 + (s // CTX) % CTY, 1 + s // (CTX * CTY)
                g = cs * nv + gidx(d, wrapm(x0 + lx - 1, nx), wrapm(y0 + ly - 1, ny), wrapm(z0 + lz - 1, nz))
                written[g] += 1
                out[g] = sites[cs * SMALL_CASE + cspos(lx, ly, lz)]
    assert (written == 1).all()
    return out


def block_gs_stencil(d, st, u0, f, order, shift):
    """Colour Gauss-Seidel with 27-point stencils per 16 x 8 x 8 block of tiling `shift`, halo frozen."""
    nx, ny, nz = d
    nv = nx * ny * nz
    sx, sy, sz = shift * CTX // 2, shift * CTY // 2, shift * CTZ // 2
    out = u0.copy()
    for z0 in range(sz, nz + sz, CTZ):
        for y0 in range(sy, ny + sy, CTY):
            for x0 in range(sx, nx + sx, CTX):
                loc = u0.copy()
                for col in order:
                    cx, cy, cz = col & 1, (col >> 1) & 1, col >> 2
                    for z in range(z0 + cz, z0 + CTZ, 2):
                        for y in range(y0 + cy, y0 + CTY, 2):
                            for x in range(x0 + cx, x0 + CTX, 2):
                                X, Y, Z = x % nx, y % ny, z % nz
                                v, sb = gidx(d, X, Y, Z), cb_index(d, X, Y, Z)
                                for c in range(3):
                                    s = f[c * nv + v]
                                    for o in range(27):
                                        if o == 13:
                                            continue
                                        ox, oy, oz = o % 3 - 1, (o // 3) % 3 - 1, o // 9 - 1
                                        inside = (x0 <= x + ox < x0 + CTX and y0 <= y + oy < y0 + CTY
                                                  and z0 <= z + oz < z0 + CTZ)
                                        src = loc if inside else u0
                                        s -= st[o * nv + sb] * src[c * nv + gidx(d, (x + ox) % nx, (y + oy) % ny,
                                                                                   (z + oz) % nz)]
                                    loc[c * nv + v] = s / st[13 * nv + sb]
                for z in range(z0, z0 + CTZ):
                    for y in range(y0, y0 + CTY):
                        for x in range(x0, x0 + CTX):
                            v = gidx(d, x % nx, y % ny, z % nz)
                            for c in range(3):
                                out[c * nv + v] = loc[c * nv + v]
    return out


@pytest.fixture(scope="module")
def cfields():
    rng = np.random.default_rng(11)
    d, dc = (32, 16, 16), (16, 8, 8)
    nv, nvc = 32 * 16 * 16, 16 * 8 * 8
    st = rng.random(27 * nv) - 0.5
    st[13 * nv:14 * nv] = 20.0 + rng.random(nv)  # a dominant diagonal
    f = rng.standard_normal(3 * nv)
    u_in = rng.standard_normal(3 * nv)
    uc = rng.standard_normal(3 * nvc)
    return d, dc, st, f, u_in, uc


def test_coarse_sweep_from_zero_tiling0(cfields):
    d, dc, st, f, u_in, uc = cfields
    got = emulate_csweep(d, dc, st, None, None, f, start=0, shift=0, reverse=False)
    ref = block_gs_stencil(d, st, np.zeros_like(f), f, list(range(8)), 0)
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


def test_coarse_sweep_with_prolongation_reverse_shifted(cfields):
    d, dc, st, f, u_in, uc = cfields
    got = emulate_csweep(d, dc, st, u_in, uc, f, start=2, shift=1, reverse=True)
    ref = block_gs_stencil(d, st, u_in + prolong(d, dc, uc), f, list(range(8))[::-1], 1)
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("start,shift,reverse", [(0, 0, False), (1, 1, False), (2, 1, True), (1, 0, True)])
def test_small_coarse_sweep(cfields, start, shift, reverse):
    d, dc, st, f, u_in, uc = cfields
    got = emulate_csmall(d, dc, st, u_in, uc, f, start, shift, reverse)
    u0 = [np.zeros_like(f), u_in, u_in + prolong(d, dc, uc)][start]
    ref = block_gs_stencil(d, st, u0, f, list(range(8))[::-1] if reverse else list(range(8)), shift)
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()
