"""The streamed smoother (k_wave in imau-ice_b200/csrc/solver.cu), restated on the CPU with its
ring of columns, schedule and ghost writes: within a step the roles run in random order on
what the previous steps left (NaN where nothing was copied), every ring and plane index is
checked, and the result must equal the level-wide colour sweeps bit for bit, for every
'zero'/'infinite' side, ragged strips and chunks, and coarsening by 2 or not along each
direction."""
import itertools
import random

import numpy as np
import pytest

INF, ZERO = 0, 1
PRE, COARSE = 3, 8


class Level:
    def __init__(self, nx, ny, bc):
        self.nx, self.ny, self.bc = nx, ny, bc          # bc: (uW,uE,uS,uN,vW,vE,vS,vN)
        self.ld = (ny + 15) // 16 * 16

    def interior(self, comp, j, i):
        if comp == 0:
            return 1 <= i <= self.nx - 3 and 1 <= j <= self.ny - 2
        return 1 <= i <= self.nx - 2 and 1 <= j <= self.ny - 3

    def src(self, comp, j, i):
        """Source of a value (u_src / v_src), None for zero."""
        if self.interior(comp, j, i):
            return j, i
        ie, jn = (self.nx - 2, self.ny - 1) if comp == 0 else (self.nx - 1, self.ny - 2)
        W, E, S, N = i == 0, i == ie, j == 0, j == jn
        b = self.bc[4 * comp:4 * comp + 4]
        kinds = [b[k] for k, on in enumerate((W, E, S, N)) if on]
        if ZERO in kinds:
            return None
        return (1 if S else jn - 1 if N else j), (1 if W else ie - 1 if E else i)


def row_apply(comp, rd, co, j, i, idx):
    """Same-shape stand-in for the operator's rows: 4 same-component neighbours, itself, 4 of the other."""
    u, v = rd
    c = co[j % 3 + 3 * (i % 3) + 9 * comp]
    if comp == 0:
        pts = [(u, j, i + 1), (u, j, i - 1), (u, j + 1, i), (u, j - 1, i), (u, j, i), (v, j, i), (v, j, i + 1),
               (v, j - 1, i), (v, j - 1, i + 1)]
    else:
        pts = [(v, j + 1, i), (v, j - 1, i), (v, j, i + 1), (v, j, i - 1), (v, j, i), (u, j + 1, i - 1),
               (u, j + 1, i), (u, j, i - 1), (u, j, i)]
    s = 0.0
    for k, (f, jj, ii) in enumerate(pts):
        s += c[k] * idx(f, jj, ii)
    return s


def colour_pass(L, x, b, co, comp, color):
    """One level-wide colour pass, boundary unknowns read through their sources."""
    def rd(f, j, i):
        p = L.src(f, j, i)
        return 0.0 if p is None else x[f][p]
    new = []
    for i in range(L.nx):
        for j in range(L.ny):
            if (i + j) % 2 == color and L.interior(comp, j, i):
                r = b[comp][j, i] - row_apply(comp, (0, 1), co, j, i, rd)
                new.append((j, i, x[comp][j, i] + 0.1 * r))
    for j, i, val in new:
        x[comp][j, i] = val


def scatter(f, fac, cell):
    if fac == 1:
        return [(f, 1.0)]
    c = f >> 1
    if cell:
        return [(c, 0.75), (c - 1 if f % 2 == 0 else c + 1, 0.25)]
    return [(c, 1.0)] if f % 2 == 0 else [(c, 0.5), (c + 1, 0.5)]


def prolong(K, comp, j, i, fx, fy, val):
    s = 0.0
    for Cj, wj in scatter(j, fy, comp == 1):
        for Ci, wi in scatter(i, fx, comp == 0):
            s += wj * wi * val(comp, Cj, Ci)
    return s


def wave(L, x0, b, co, nu, rows, chunk, up, K=None, xc=None, fx=1, fy=1, rng=None):
    """k_wave over the whole level: (x, r) for the descent, x for the ascent."""
    NP, H = 4 * nu, 4 * nu + 1
    TJ, HB = 64 - 2 * NP, (H + 3) // 4 * 4
    RP, NC = (HB + TJ + H + 3) // 4 * 4, 2 * PRE + 3 * NP + 6
    CP = RP + 8
    assert rows <= TJ and rows % 4 == 0
    out = np.full((2, L.ny, L.nx), np.nan)
    res = np.full((2, L.ny, L.nx), np.nan)
    for tj0, ti0 in itertools.product(range(0, L.ny, rows), range(0, L.nx, chunk)):
        j0, i0 = tj0 - HB, ti0 - H
        tw = min(chunk, L.nx - ti0)
        ncols = tw + 2 * H
        CJ0 = ((j0 >> 1) - 2) & ~1 if fy == 2 else j0 - 2
        X = np.full((NC, 2, RP), np.nan)
        C = np.full((COARSE, 2, CP), np.nan)
        state = dict(bad=0)

        def coarse_col(Cc, comp):
            last = K.nx - 2 if comp == 0 else K.nx - 1
            I = min(max(Cc, 0), last)
            w, e = K.bc[4 * comp], K.bc[4 * comp + 1]
            if I == 0:
                return 1 if w == INF else -1
            if I == last:
                return last - 1 if e == INF else -1
            return I

        def load_coarse(Cc):
            for comp in (0, 1):
                I = coarse_col(Cc, comp)
                if I >= 0:
                    for r in range(CP):
                        if 0 <= CJ0 + r < K.ny:
                            C[Cc & (COARSE - 1), comp, r] = xc[comp][CJ0 + r, I]

        def issue(t):
            for h in (0, 1):
                i, sl = i0 + 2 * t + h, (2 * t + h) % NC
                X[sl] = 0.0 if not up else np.nan
                if up and 0 <= i < L.nx:
                    for r in range(RP):
                        if 0 <= j0 + r < L.ny:
                            X[sl, :, r] = x0[:, j0 + r, i]
            if up:
                i = i0 + 2 * t
                Cb = i + 1 if fx == 1 else ((i + 1) >> 1) + 1
                for Cc in range(i if fx == 1 else Cb - 3 if t == 0 else Cb, Cb + 1):
                    load_coarse(Cc)

        def at(cc, dc, j):
            assert 0 <= j - j0 < RP
            return (cc + dc) % NC, j - j0

        def ghosts(comp, cc, j, i, val):
            il, jl = (L.nx - 3, L.ny - 2) if comp == 0 else (L.nx - 2, L.ny - 3)
            w, e, s_, n = L.bc[4 * comp:4 * comp + 4]
            for on, dc, jg in ((s_ == INF and j == 1, 0, 0), (n == INF and j == jl, 0, jl + 1),
                               (w == INF and i == 1, -1, j), (e == INF and i == il, 1, j)):
                if on:
                    sl, r = at(cc, dc, jg)
                    X[sl, comp, r] = val

        def reader(cc, i):
            def rd(f, j, ii):
                sl, r = at(cc, ii - i, j)
                return X[sl, f, r]
            return rd

        def do_pass(q, s):
            p = q & 3
            p = 3 - p if up else p
            comp, color, reach = p >> 1, p & 1, H - 1 - q
            il, jl = (L.nx - 3, L.ny - 2) if comp == 0 else (L.nx - 2, L.ny - 3)
            jlo = tj0 - reach
            jmin, jmax = max(jlo, 1), min(tj0 + rows + reach - 1, jl)
            new = []
            for lane in range(32):
                cc = 2 * s - 3 - 3 * q + ((lane >> 3) & 1)
                i = i0 + cc
                if not (max(H - reach, 1 - i0) <= cc <= min(H + tw + reach - 1, il - i0)):
                    continue
                jA = jlo + ((color + i + jlo) & 1) + 2 * ((lane & 7) | ((lane >> 4) << 3))
                for j in (jA, jA + 32):
                    if jmin <= j <= jmax:
                        sl, r = at(cc, 0, j)
                        val = X[sl, comp, r] + 0.1 * (b[comp][j, i] - row_apply(comp, (0, 1), co, j, i, reader(cc, i)))
                        new.append((comp, cc, j, i, val))
            assert jmax < jlo + 64                                       # a warp covers the rows of the colour
            return new

        def do_prolong(s):
            new = []
            for cc in (2 * s, 2 * s + 1):
                i = i0 + cc
                for r in range(RP - 1):
                    j = j0 + r
                    for comp in (0, 1):
                        if cc < ncols and i >= 1 and j >= 1 and L.interior(comp, j, i):
                            def tap(cp, Cj, Ci):
                                lj, li = (K.ny - 1, K.nx - 2) if cp == 0 else (K.ny - 2, K.nx - 1)
                                J, I = min(max(Cj, 0), lj), min(max(Ci, 0), li)
                                if J in (0, lj) or I in (0, li):
                                    p = K.src(cp, J, I)
                                    if p is None:
                                        return 0.0
                                    J = p[0]
                                assert 0 <= J - CJ0 < CP
                                return C[Ci & (COARSE - 1), cp, J - CJ0]
                            sl, rr = at(cc, 0, j)
                            new.append((comp, cc, j, i, X[sl, comp, rr] + prolong(K, comp, j, i, fx, fy, tap)))
            return new

        def do_out(s):
            for cc in (2 * s - 3 - 3 * NP, 2 * s - 2 - 3 * NP):
                i = i0 + cc
                if not H <= cc < H + tw:
                    continue
                for jj in range(min(rows, L.ny - tj0)):
                    j = tj0 + jj
                    for comp in (0, 1):
                        sl, r = at(cc, 0, j)
                        inner = L.interior(comp, j, i)
                        out[comp, j, i] = X[sl, comp, r] if (inner or not up) else 0.0
                        res[comp, j, i] = ((b[comp][j, i] - row_apply(comp, (0, 1), co, j, i, reader(cc, i)))
                                           if inner else 0.0)

        def commit(new):
            for comp, cc, j, i, val in new:
                sl, r = at(cc, 0, j)
                X[sl, comp, r] = val
                ghosts(comp, cc, j, i, val)

        npair = tw // 2 + H + (tw & 1)
        issued = min(PRE, npair)
        for t in range(issued):
            issue(t)
        for s in range((tw + H + 3 * NP + 2) // 2 + 1):
            roles = [("pass", q) for q in range(NP)] + [("out", 0), ("copy", 0)] + ([("prolong", 0)] if up else [])
            rng.shuffle(roles)
            for kind, q in roles:            # any order within a step
                if kind == "pass":
                    commit(do_pass(q, s))
                elif kind == "out":
                    do_out(s)
                elif kind == "copy":
                    if s + PRE < npair:
                        issue(s + PRE)
                else:
                    commit(do_prolong(s))
    return out, res


SIDES = [(INF,) * 8, (ZERO,) * 8, (ZERO, INF, INF, INF, ZERO, INF, ZERO, ZERO), (INF, ZERO, ZERO, INF, INF, INF, INF, ZERO)]


@pytest.mark.parametrize("nx,ny,nu,rows,chunk", [(23, 17, 1, 8, 7), (14, 41, 2, 12, 5), (9, 9, 2, 48, 9), (31, 12, 2, 4, 31)])
@pytest.mark.parametrize("bc", SIDES)
def test_streamed_sweeps_equal_the_colour_sweeps(nx, ny, nu, rows, chunk, bc):
    rng = np.random.default_rng(nx + ny)
    order = random.Random(nx * ny)
    L = Level(nx, ny, bc)
    co = rng.normal(0, 0.3, (18, 9))
    b = rng.normal(0, 1, (2, ny, nx))
    # descent: x = 0, forward sweeps, residual
    x = np.zeros((2, ny, nx))
    for _ in range(nu):
        for p in range(4):
            colour_pass(L, x, b, co, p >> 1, p & 1)
    got, res = wave(L, None, b, co, nu, rows, chunk, False, rng=order)
    for comp in (0, 1):
        m = np.array([[L.interior(comp, j, i) for i in range(nx)] for j in range(ny)])
        assert np.array_equal(got[comp][m], x[comp][m])

        def rd(f, j, i):
            q = L.src(f, j, i)
            return 0.0 if q is None else x[f][q]
        want = [b[comp][j, i] - row_apply(comp, (0, 1), co, j, i, rd) for j, i in zip(*np.nonzero(m))]
        assert np.array_equal(res[comp][m], np.array(want)) and not res[comp][~m].any()
    # ascent: prolongation, backward sweeps, from the descent's x (its ghosts included)
    for fx, fy in ((2, 2), (1, 2), (2, 1)):
        K = Level((nx + 2) // 2 if fx == 2 else nx, (ny + 2) // 2 if fy == 2 else ny, bc)
        xc = rng.normal(0, 1, (2, K.ny, K.nx))

        def coarse(cp, Cj, Ci):
            lj, li = (K.ny - 1, K.nx - 2) if cp == 0 else (K.ny - 2, K.nx - 1)
            q = K.src(cp, min(max(Cj, 0), lj), min(max(Ci, 0), li))
            return 0.0 if q is None else xc[cp][q]
        y = x.copy()
        for comp in (0, 1):
            for j in range(ny):
                for i in range(nx):
                    if L.interior(comp, j, i):
                        y[comp][j, i] += prolong(K, comp, j, i, fx, fy, coarse)
        for _ in range(nu):
            for p in (3, 2, 1, 0):
                colour_pass(L, y, b, co, p >> 1, p & 1)
        got2, _ = wave(L, got, b, co, nu, rows, chunk, True, K, xc, fx, fy, rng=order)
        for comp in (0, 1):
            m = np.array([[L.interior(comp, j, i) for i in range(nx)] for j in range(ny)])
            assert np.array_equal(got2[comp][m], y[comp][m]) and not got2[comp][~m].any()
