"""Host-side emulation of the address arithmetic of the precision form's step
kernel (fall3d_gb300/csrc/f3d_fused2.cu, step_tile) for both tile shapes, on
grids of many sizes and for every way step_chunks cuts their columns: every
global load and store falls inside its array under the guard it is made under,
pairs are 8-byte aligned, every tensor copy starts on a 16-byte boundary and
brings the planes its iteration reads, the shared-memory reads a row beyond a
staged field or exchange plane stay inside the block's allocation, and every
value of the result is stored exactly once.

The layout's numbers are read from the sources, and the expressions that the
emulation restates are compared with the sources' text: a change of either
makes this file fail until the emulation follows."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fall3d_gb300", "csrc")


def _source(name):
    """A source without its comments."""
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def _squeeze(s):
    return re.sub(r"\s+", "", s)


SRC, MATH, HEAD, CTX = (_source(n) for n in ("f3d_fused2.cu", "f3d_fused_math.cuh", "f3d_fused.h", "f3d_ctx.cu"))


def _const(name):
    return int(re.search(rf"\b{name} = (\d+)\b", SRC).group(1))


def _pin(src, *texts):
    flat = _squeeze(src)
    for t in texts:
        assert _squeeze(t) in flat, t


HX, GUARD = _const("HX"), _const("GUARD")
TX, RS = HX - 6, HX + 4
FIELDS = re.findall(r"\w+", re.search(r"enum : int \{ (F_C = 0[^}]*)\}", MATH).group(1).replace("= 0", ""))
assert FIELDS[-1] == "NF"
NF = len(FIELDS) - 1
F = {n: i for i, n in enumerate(FIELDS)}
_members = re.search(r"struct ZTab \{(.*?)\};", HEAD, re.S).group(1)
ZTAB = 4 * sum(int(n) if n else 1 for n in re.findall(r"\b(?:a|b|rdz|dtdzz|dtrdz|pad)\b(?:\[(\d+)\])?", _members))
# region rows and warps of the two shapes
SHAPES = {"Tall": (_const("HY"), _const("NW")),
          "Flat": tuple(int(v) for v in re.search(r"using Flat = Shape<(\d+), (\d+)>", SRC).groups())}


def plane_of(f):
    """field_plane: the plane of field f in iteration t, minus t"""
    return 2 if f == F["F_C"] else 1 if f == F["F_VK"] else -1 if f >= F["F_FZ"] else 0


def test_the_sources_say_what_is_emulated():
    assert len(re.findall(r"\bfloat\b", _members)) == 5 and ZTAB == 32  # all of its members were counted
    _pin(SRC, "using Tall = Shape<HY, NW>;")
    _pin(MATH, "return f == F_C ? 2 : f == F_VK ? 1 : f >= F_FZ ? -1 : 0;")
    _pin(HEAD, "inline int halo_pitch(int nx) { return (nx + 2 + 3) & ~3; }")
    # the shapes, shared memory, tensor maps
    _pin(SRC, "NT = 32 * NW_, RPW = HY_ / NW_, TY = HY_ - 6, FS = RS * HY_, NP = HX * HY_",
         "return GUARD + sizeof(float) * ((size_t)2 * NF * S::FS + 3 * (size_t)S::NP + HX) + "
         "sizeof(ZTab) * (size_t)(nz + 2) + 64;",
         "float* stage = reinterpret_cast<float*>(smem_raw + GUARD); float* P0s = stage + 2 * NF * FS; "
         "float* Ws = P0s + NP; float* P1s = Ws + NP; ZTab* tab = reinterpret_cast<ZTab*>(P1s + NP + HX); "
         "unsigned long long* mbar = reinterpret_cast<unsigned long long*>(tab + (a.d.nz + 2));",
         "const cuuint64_t dim[3] = {(cuuint64_t)d.px, (cuuint64_t)(d.ny + 2), (cuuint64_t)planes};",
         "const cuuint32_t box[3] = {(cuuint32_t)RS, q ? 16u : 32u, 1u};",
         "const long long np = a.d.nz + 2;", "f == F2Maps::VK ? np * a.ncls : np")
    # positions, the piece's levels and the staging
    _pin(SRC, "const int i0 = 1 + (tile % tiles_x) * TX, j0 = 1 + (tile / tiles_x) * TY;",
         "const int gx0 = i0 - 3, gy0 = j0 - 3;", "const int gi = gx0 + 2 * lane;", "const int gj0 = gy0 + RPW * warp;",
         "const int oi1 = min(nx, i0 + TX - 1), oj1 = min(ny, j0 + TY - 1);", "const int xs = gx0 & ~3;",
         "const int k0 = chunk == 0 ? 1 : a.kfirst + 1 + (chunk - 1) * a.klen;",
         "const int k1 = chunk == 0 ? (a.nchunk > 1 ? a.kfirst : nz) : min(nz, k0 + a.klen - 1);",
         "const int ts = max(1, k0 - 1), te = k1 + 1;",
         "const int f_z = warp <= F_VK ? cls * (nz + 2) : 0;", "const bool ok = p >= 1 && p <= nz;",
         "tma_load3(stage0 + 4u * (buf * NF + warp) * FS, f_map, xs, gy0, f_z + p, bar);",
         "const bool pair_in = gi >= 0 && gi < px;", "return gj0 + r >= 0 && gj0 + r <= ny + 1;",
         "const int h0 = gi + px * gj0;")
    # the window, ghosts and edge arrays
    _pin(SRC, "const bool in = pair_in && row_in(r);", "o0[r] = C(ts); o1[r] = C(ts + 1); vk[r] = V(ts);",
         "const float2 cm = C(ts - 1), cmm = C(ts - 2), vm = V(ts - 1), vmm = V(ts - 2);",
         "cin + h + (gj == 0 ? px : -px) + ts * cs", "if (t < min(te, nz) && pair_in)",
         "cin + h0 + r * px + (lo ? px : -px) + (t + 1) * cs",
         "if (k < k0) continue;", "if (xedge && (gi == 0 || gi == nx || gi + 1 == nx) && row_in(r))",
         "a.f.ex + (gi == 0 ? 0 : (nz + 2) * (ny + 2)) + k * (ny + 2) + gj",
         "if ((gj == 1 || gj == ny) && pair_in) ey[r] = ldg2(a.f.ey + (gj == 1 ? 0 : (nz + 2) * px) + k * px + gi);",
         "const int h = pair_in && row_in(r) ? h0 + r * px : 0;", "ldg2(a.f.ez + h)", "ldg2(a.f.fz + h)",
         "ldg2(a.f.fz + h + nz * cs)", "ldg2(a.f.fz + h + (nz + 1) * cs)",
         "cout[h0 + r * px + c + (nz + 1) * cs] = clip0(cmp(c2, c));", "float* const q = cout + (h0 + k * cs);")
    # what is staged is read under these conditions, at these rows
    _pin(SRC, "if (STEADY || t + 1 <= nz) { vkp = lds2(at(F_VK, r)); if (STEADY || t + 2 <= nz) { c2 = lds2(at(F_C, r));",
         "for (int r = 0; r <= RPW; ++r) cfy[r] = lds2(at(F_FY, r - 1));", "lds2(P0 - HX), ca = lds2(P0 + RPW * HX)",
         "lds2(W - HX), Fa = r < RPW ? F[r] : lds2(W + RPW * HX)", "lds2(P1 - HX), qa = lds2(P1 + RPW * HX)")
    _pin(SRC, "const int len = (nz + n - 1) / n, first = std::max(len, nwet), rest = nz - first;",
         "if (len < 4 || rest < 4 * (n - 1)) break;", "const int each = (rest + n - 2) / (n - 1);",
         "if (rest - each * (n - 2) < 4) continue;", "for (int n = 2; n <= 16; ++n) {")
    # the arrays' sizes
    _pin(CTX, "hsz = (size_t)d.halo(), hpl = (size_t)d.px * (d.ny + 2);", "A(sf.vk, hsz * nc);",
         "A(sf.ex, 2 * (size_t)(d.nz + 2) * (d.ny + 2));", "A(sf.ey, 2 * (size_t)(d.nz + 2) * d.px);", "A(sf.ez, hpl);",
         "A(sf.tab, (size_t)d.nz + 2);")


def cuts(nz):
    """Every (nchunk, kfirst, klen) that step_chunks may return for nz levels:
    the uncut column, and each n it considers for each wet level."""
    out = {(1, nz, nz)}
    for nwet in range(nz + 1):
        for n in range(2, 17):
            size = -(-nz // n)
            first = max(size, nwet)
            rest = nz - first
            if size < 4 or rest < 4 * (n - 1):
                break
            each = -(-rest // (n - 1))
            if rest - each * (n - 2) < 4:
                continue
            assert first >= nwet
            out.add((n, first, each))
    return sorted(out)


def pieces(nz, cut):
    n, first, each = cut
    out = []
    for chunk in range(n):
        k0 = 1 if chunk == 0 else first + 1 + (chunk - 1) * each
        k1 = (first if n > 1 else nz) if chunk == 0 else min(nz, k0 + each - 1)
        out.append((k0, k1, max(1, k0 - 1), k1 + 1))
    return out


@pytest.mark.parametrize("nz", [3, 4, 7, 8, 9, 12, 13, 17, 25, 33, 50, 80, 128, 1000])
def test_pieces_cover_the_column_and_stage_what_they_read(nz):
    for cut in cuts(nz) if nz < 200 else cuts(nz)[::97]:
        levels = []
        for k0, k1, ts, te in pieces(nz, cut):
            assert k0 <= k1
            levels += range(k0, k1 + 1)
            # the window: c at ts..ts+1, and inside the column ts-2..ts+1; vz+vset up to ts
            assert ts == 1 or ts - 2 >= 1
            assert ts + 1 <= nz
            for t in range(ts, te + 1) if nz < 200 else (ts, ts + 1, te - 1, te):
                loaded = {f for f in range(NF) if 1 <= t + plane_of(f) <= nz}
                need = set()
                if t <= nz:
                    need |= {F[f] for f in ("F_UX", "F_KX", "F_UY", "F_KY", "F_L")}
                    if t + 1 <= nz:
                        need.add(F["F_VK"])
                    if t + 2 <= nz:
                        need.add(F["F_C"])
                    if t > ts:
                        need.add(F["F_FZ"])
                if t - 1 >= k0:
                    need |= {F["F_FX"], F["F_FY"]}
                assert need <= loaded, (cut, t, need - loaded)
        assert levels == list(range(1, nz + 1)), cut


def _positions(nx, ny, shape):
    """The positions of every lane's pair: tile, warp, lane, row r of the warp."""
    hy, nw = SHAPES[shape]
    ty = hy - 6
    tx = -(-nx // TX)
    tile = np.arange(tx * -(-ny // ty))
    T, W, L, R = np.meshgrid(tile, np.arange(nw), np.arange(32), np.arange(hy // nw), indexing="ij")
    i0, j0 = 1 + (T % tx) * TX, 1 + (T // tx) * ty
    return dict(i0=i0, j0=j0, oi1=np.minimum(nx, i0 + TX - 1), oj1=np.minimum(ny, j0 + ty - 1), gi=i0 - 3 + 2 * L,
                gj=j0 - 3 + hy // nw * W + R, gx0=i0 - 3)


def _in(idx, size, what):
    assert idx.size == 0 or (idx.min() >= 0 and idx.max() < size), (what, int(idx.min()), int(idx.max()), size)


def _pair(idx, size, what):
    _in(idx, size - 1, what)
    assert np.all(idx % 2 == 0), what + " is not 8-byte aligned"


GRIDS = [(nx, ny, nz) for nx in (3, 4, 5, 57, 58, 59, 60, 64, 116, 117, 175) for ny in (3, 4, 10, 11, 20, 25, 26, 27, 53)
         for nz in (3, 4)] + [(61, 28, 17), (5, 12, 25), (117, 53, 41)]


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("nx,ny,nz", GRIDS)
def test_global_accesses_stay_in_their_arrays(nx, ny, nz, shape):
    p = _positions(nx, ny, shape)
    gi, gj, i0, j0 = p["gi"], p["gj"], p["i0"], p["j0"]
    px = (nx + 2 + 3) & ~3
    cs, pl = px * (ny + 2), nx * ny
    size = cs * (nz + 2)  # a class of c and of vz+vset; a field
    assert size % 4 == 0  # class blocks keep the pairs' and copies' alignment
    pair_in = (gi >= 0) & (gi < px)
    row_in = (gj >= 0) & (gj <= ny + 1)
    both = pair_in & row_in
    h = gi + px * gj
    edge = ~((p["gx0"] >= 1) & (p["gx0"] + HX - 1 <= nx) & (j0 - 3 >= 1) & (j0 - 3 + SHAPES[shape][0] - 1 <= ny))
    xedge = (p["gx0"] <= 1) | (p["gx0"] + HX - 1 >= nx)
    ghost_row = (gj == 0) | (gj == ny + 1)
    ya = np.where(gj == 0, px, -px)
    g = np.stack([gi, gi + 1], -1)
    rows = ((gj >= j0) & (gj <= p["oj1"]))[..., None]
    cols = (g >= i0[..., None]) & (g <= p["oi1"][..., None])
    out = rows & cols
    gjj = gj[..., None] + 0 * g
    ghost = (rows & (((g == 0) & (i0 == 1)[..., None]) | ((g == nx + 1) & (p["oi1"] == nx)[..., None]))) | \
            (cols & (((gjj == 0) & (j0 == 1)[..., None]) | ((gjj == ny + 1) & (p["oj1"] == ny)[..., None])))
    stored = out | ghost

    # tensor copies: the box's first column on 16 bytes, the region inside the box
    xs = p["gx0"] & ~3
    assert np.all(xs % 4 == 0) and px % 4 == 0
    assert np.all((p["gx0"] - xs >= 0) & (p["gx0"] - xs + HX <= RS))
    # ghost cells that the kernel forms are in an edge tile; the ends of x lines in an xedge one
    assert np.all(edge[ghost_row & pair_in]) and np.all(edge[both & ((gi == 0) | (gi + 1 == nx + 1) | (gi == nx + 1))])
    assert np.all(xedge[both & ((gi == 0) | (gi == nx) | (gi + 1 == nx))])

    for cut in cuts(nz):
        for chunk, (k0, k1, ts, te) in enumerate(pieces(nz, cut)):
            for k in (ts, ts + 1) if ts == 1 else (ts - 2, ts - 1, ts, ts + 1):
                _pair((h + k * cs)[both], size, "window")
            if ts == 1:
                inner = (g >= 1) & (g <= nx) & (gjj >= 1) & (gjj <= ny)
                _in(((g - 1) + nx * (gjj - 1))[inner], pl, "vdep, rkver1")
            for k in range(ts, min(te, nz) + 1):  # first at ts, then t+1 <= min(te, nz)
                _pair((h + ya + k * cs)[edge & ghost_row & both], size, "row beside a ghost row")
            for k in {k0, k1}:
                m = edge & xedge & ((gi == 0) | (gi == nx) | (gi + 1 == nx)) & row_in
                _in((np.where(gi == 0, 0, (nz + 2) * (ny + 2)) + k * (ny + 2) + gj)[m], 2 * (nz + 2) * (ny + 2), "ex")
                m = edge & ((gj == 1) | (gj == ny)) & pair_in
                _pair((np.where(gj == 1, 0, (nz + 2) * px) + k * px + gi)[m], 2 * (nz + 2) * px, "ey")
                for f in range(NF):
                    for t in (ts, te):
                        pk = t + plane_of(f)
                        if 1 <= pk <= nz:
                            assert pk < nz + 2
                _in(((g + px * gjj) + k * cs)[stored], size, "store")
                pairs = stored.all(-1)
                _pair((h + k * cs)[pairs], size, "pair store")
            hh = np.where(both, h, 0)
            if k0 == 1:
                _pair(hh, cs, "ez, fz plane 0")
                _in((g + px * gjj)[out], size, "bottom ghost")
            if k1 == nz:
                _pair(hh + nz * cs, size, "fz plane nz")
                _pair(hh + (nz + 1) * cs, size, "fz plane nz+1")
                _in((g + px * gjj + (nz + 1) * cs)[out], size, "top ghost")
            _in(((g - 1) + nx * (gjj - 1))[out], pl, "2-D fields of output cells")

    # each output cell and each face ghost of a plane is stored once
    cells = (g + px * gjj)[stored]
    J, I = np.meshgrid(np.arange(ny + 2), np.arange(nx + 2), indexing="ij")
    corner = ((I == 0) | (I == nx + 1)) & ((J == 0) | (J == ny + 1))
    assert np.array_equal(np.sort(cells), np.sort((I + px * J)[~corner]))
    # the mixing-height scan of the tile's columns
    hy = SHAPES[shape][0]
    o = np.arange(TX * (hy - 6))
    for a, b in {(int(x), int(y)) for x, y in zip(i0.ravel(), j0.ravel())}:
        oi, oj = a + o % TX, b + o // TX
        m = (oi <= min(nx, a + TX - 1)) & (oj <= min(ny, b + hy - 7))
        _in(((oi - 1) + nx * (oj - 1))[m], pl, "zi")


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("nz", [3, 25, 80])
def test_shared_memory_stays_in_the_block(shape, nz):
    hy, nw = SHAPES[shape]
    rpw, fs, np_ = hy // nw, RS * hy, HX * hy
    smem = GUARD + 4 * (2 * NF * fs + 3 * np_ + HX) + ZTAB * (nz + 2) + 64
    assert nw >= NF and GUARD % 128 == 0 and (4 * fs) % 128 == 0  # a warp issues a field; boxes land on 128 bytes
    assert smem <= 227 * 1024
    planes = 2 * NF * fs  # P0s, in floats from the staging area on; then Ws, P1s, HX of padding, the table
    tab = planes + 3 * np_ + HX
    assert (4 * tab + GUARD) % 16 == 0 and ZTAB % 8 == 0
    assert GUARD + 4 * tab + ZTAB * (nz + 2) + 2 * 8 <= smem  # the two barriers
    W, L = np.meshgrid(np.arange(nw), np.arange(32), indexing="ij")
    for sft in (0, 2):
        row0 = rpw * W * RS + sft + 2 * L
        assert row0.max() + (rpw - 1) * RS + 1 < fs
        for buf in (0, 1):
            for f in range(NF):
                base = (buf * NF + f) * fs + row0
                low = -1 if f == F["F_FY"] else 0
                for r in range(low, rpw):
                    idx = base + r * RS
                    assert idx.min() >= -GUARD // 4 and idx.max() + 1 < planes and np.all(idx % 2 == 0)
    for q in range(3):
        base = planes + q * np_ + rpw * W * HX + 2 * L
        for off in (-HX, 0, (rpw - 1) * HX, rpw * HX):  # a row above, the warp's, a row below
            idx = base + off
            assert idx.min() >= 0 and idx.max() + 1 < tab
