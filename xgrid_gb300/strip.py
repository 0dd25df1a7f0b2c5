"""Strips: a star-shaped sweep of 4-byte elements at memory bandwidth, 2-D and 3-D.

A 5- or 7-point FP32 sweep does a dozen or two operations per cell against eight or twelve
bytes, so it is bound by HBM where the loads keep enough bytes in flight and the instructions
around them are few.  In the tile kernel a CTA lives for a few dependent round trips to memory
(4096^2, five loads: 44 us against 20 us at the copy bandwidth), and the staged z-walk
(``codegen.zstage_frame``) spends two thirds of its instructions on staging and ring loads,
and needs rows aligned to 16 bytes.  Here every warp owns a strip of ``32 J`` columns (by ``R``
rows of 3-D grids) and walks a chunk of the slowest axis:

* lane l holds columns ``x0 + l + 32 j``: every load and store is 32 consecutive elements,
  whatever the alignment of the row;
* the planes (rows of 2-D grids) next to the current one stay in registers; the ``U`` planes
  after them are loaded while the current ``U`` are computed;
* a neighbour column comes from the next lane (or the next segment's first lane) by a shuffle
  (as loads one element to the side, from L1, the 4096^2 sweep takes 54 us instead of 29);
  the columns next to the strip -- wrapped, clamped or the flattened neighbour at the grid's
  first and last column -- are one predicated load per row and side; the rows next to a 3-D strip are loaded as the strip's own are (from L1
  where the CTA's next warp holds them).

Boundary cells: one bit per cell (``xg_mask_bits``) tells the cells that the sweep leaves
alone, and the group's boundary phases follow as launches over their cell lists.  A row's mask
words are loaded with the planes ahead, one word a lane, and handed round by shuffles (loaded by
every lane where its cells are stored, they cost an L1 or L2 latency per row: 256^3 walls 51 us
against 44; two bits per cell and the phases' constants stored by the sweep itself: 47).  The chunk
length comes from the SM count, so that the strips fill whole rounds of the resident warps.
Same arithmetic per cell as the other paths.
"""
from __future__ import annotations

from . import analysis

WARPS = 4              # warps per CTA
# (segments of 32 columns, rows, planes ahead, resident CTAs per SM asked of ptxas), by dimension
# and loaded buffers; wide strips first.  Measured: 4096^2 transport 29 us (2 rows ahead; with 4:
# 31, with 2 segments 39); 256^3 walls 51 us with 8 segments, 58 with 2 x 2 (before the mask
# words were loaded ahead; 44 since); 203 x 245 x 307
# diffusion 56 us (4 x 1: 64, 1 x 4: 66).
SHAPE = {(2, 1): [(4, 1, 2, 6)], (2, 2): [(2, 1, 2, 6)], (3, 1): [(8, 1, 1, 4), (2, 2, 1, 6)], (3, 2): [(2, 2, 1, 4)]}
FILL = 60  # a strip shape applies where the grid's columns fill at least this share (%) of its lanes
# Sweeps that compute in FP64 (a Python literal is a double) are bound by the FP64 pipe, which strips
# with idle lanes, or few of them, keep waiting.  2-D: narrow strips, but wide ones where they are full
# and no mask is read (us, 128 against 64 columns: heat with walls 4097^2 206 and 199, 8192^2 757 and 750,
# 1300^2 30.8 and 28.7; without 1500^2 34.9 and 30.8, 6000^2 406 and 411).  3-D, where the tile kernel
# is no z-walk: strips only for ragged rows on 64 planes and more (tiles and strips, us: 384^3 755 and 922,
# 256^3 232 and 246, 80 x 80 x 96 15.4 and 25.6, 24 x 1000 x 200 77 and 88, 9 x 60 x 1001 16.4 and 27.1;
# but 203 x 201 x 205 139 and 129, 100 x 101 x 103 30.8 and 27.9).
SHAPE_FP64_2D, FILL_FP64 = (2, 1, 2, 6), 99
MIN_PLANES_FP64 = 64
# smallest grids (cells), by dimension, without and with boundary phases (launches of their own
# then): 2-D transport 2048^2 11.0 against 13.8 us on tiles, 1000^2 10.3 against 9.3; 3-D
# diffusion 100^3 10.0 against 12.5; walls 2-D 1024^2 8.4 against 9.0, 3-D 80^3 13.6 against
# 14.5, 64^3 14.4 against 10.3
MIN_CELLS = {2: 1 << 21, 3: 1 << 17}
MIN_CELLS_PHASES = {2: 1 << 20, 3: 1 << 19}
# from three phases on their launches weigh more, on 2-D rows of whole 32-column tiles, which the fused
# launch takes best: four constant walls at 1024^2 12.3 against 10.2 us, 1024 x 1536 12.3 against 10.4,
# 2048^2 16.4 against 16.9; ragged rows 1150^2 12.3 against 14.4, 1500^2 14.3 against 17.9.  (3-D: four
# walls 80 x 80 x 96 14.4 both, six 16.6 against 16.4, 128^3 18.5 against 20.8)
MANY_PHASES, MIN_CELLS_MANY = 3, 1 << 21


def plan(em, j: int):
    """(dimension, loaded buffers) of sweep ``j`` when it can run on strips, else None: 2-D
    or 3-D, 4-byte elements, a store at the cell itself, loads at the cell and its
    neighbours along one axis."""
    s = em.g.sweeps[j]
    if any(s.store_offset):
        return None
    dims = set()
    for slot in em.slots_used([s]):
        t = em.gen.defn.signature.arguments[em.arg_index(slot)][1]
        dims.add(t.dimension)
        if t.dimension not in (2, 3) or em.elem(slot) not in ("float", "int32_t"):
            return None
    bufs = []
    for _, ld in s.loads:
        if sum(abs(o) for o in ld.offset) > 1:
            return None
        b = (ld.slot, ld.level, ld.version)
        if b not in bufs:
            bufs.append(b)
    key = (s.slot, s.level, s.read_version_of_target)
    if s.implicit and key not in bufs:
        bufs.append(key)
    if len(dims) != 1 or (min(dims), len(bufs)) not in SHAPE:
        return None
    return min(dims), bufs


def shapes(em, pl) -> list:
    """(strip shape, least fill) in the order of choice."""
    dim, bufs = pl
    out = [(s, FILL) for s in SHAPE[(dim, len(bufs))]]
    if dim == 2 and len(bufs) == 1 and em.fp64_ops():
        wide = [(out[0][0], FILL_FP64)] if len(em.g.sweeps) == 1 else []
        out = wide + [(SHAPE_FP64_2D, FILL)]
    return out


def kernels(em, tag: str, j: int, pl) -> list:
    """One kernel per strip shape."""
    return [_kernel(em, tag, j, pl, v, shape) for v, (shape, _) in enumerate(shapes(em, pl))]


def _kernel(em, tag: str, j: int, pl, variant: int, shape: tuple) -> str:
    from .codegen import SweepEnv
    n, gid, gen = em.name, em.gid, em.gen
    s = em.g.sweeps[j]
    dim, bufs = pl
    J, R, U, blocks = shape
    none = gen.cfg.overstep == "none"
    T = em.elem(s.slot)
    dst = em.bname((s.slot, s.level, s.write_version))
    walk = 0 if dim == 3 else 1  # the walked axis in a (z, y, x) offset
    offs = {b: {ld.offset for _, ld in s.loads if (ld.slot, ld.level, ld.version) == b} for b in bufs}
    lo = {b: min([0] + [o[walk] for o in offs[b]]) for b in bufs}
    hi = {b: max([0] + [o[walk] for o in offs[b]]) for b in bufs}
    rows = {b: [d for d in (-1, 1) if dim == 3 and (0, d, 0) in offs[b]] for b in bufs}
    side = {b: [d for d in (-1, 1) if (0, 0, d) in offs[b]] for b in bufs}
    P = f"struct xgp_{n}_{gid}_{tag}"
    K = [f"template <typename I, bool MASKED> __global__ void __launch_bounds__({WARPS * 32}, {blocks}) "
         f"xgk_{n}_{gid}_{tag}_rs{variant}(const __grid_constant__ {P} p, const int alen, const int nsx, const int nsy, "
         "const int nwarps, const uint32_t* __restrict__ bits) {",
         f"  constexpr int J = {J}, R = {R}, U = {U};",
         "  constexpr unsigned FULL = 0xffffffffu;",
         "  const int lane = threadIdx.x & 31;",
         f"  const int wid = blockIdx.x * {WARPS} + (threadIdx.x >> 5);",
         "  if (wid >= nwarps) return;",
         "  const xg_fp64 xg_f = xg_fp64_units();",
         "  (void)xg_f;",
         f"  const int X = (int)p.X, NY = {'(int)p.Y' if dim == 3 else '1'}, A = (int)p.{'Z' if dim == 3 else 'Y'};",
         "  // warps of a CTA are neighbours along y (3-D) or x (2-D)",
         "  const int y0 = wid % nsy * R, x0 = wid / nsy % nsx * (32 * J), aa = wid / (nsy * nsx) * alen;",
         "  const int ab = aa + alen < A ? aa + alen : A;",
         "  bool in[J];  // the lane's columns inside the grid",
         "#pragma unroll",
         "  for (int j = 0; j < J; ++j) in[j] = x0 + lane + 32 * j < X;",
         "  // the side columns: x0 - 1 for lane 0, the one after the strip's last cell for the lane that holds it",
         "  const int xl = x0 + 32 * J < X ? x0 + 32 * J - 1 : X - 1, js = (xl - x0) >> 5;",
         "  const bool first = lane == 0, last = lane == ((xl - x0) & 31);"]
    k0, k1 = (-1, R) if dim == 3 else (0, 0)
    K += ["  // offsets of the rows y0 - 1 .. y0 + R in a plane",
          f"  I yo[{k1 - k0 + 1}];", "#pragma unroll", f"  for (int k = 0; k < {k1 - k0 + 1}; ++k)"]
    if none:
        K += [f"    yo[k] = (I)(y0 + k + ({k0})) * X;",
              "  // neighbours are flattened offsets; what lies outside the allocation reads 0",
              "  const I plane = (I)NY * X, total = plane * A;",
              "  const int xw = x0 - 1, xe = xl + 1;",
              "  auto base = [&](int a) { return (I)a * plane; };",
              "  auto ok_row = [&](I q) { return q >= 0 && q < total; };"]
    else:
        K += [f"    yo[k] = (I)xg_near(xg_overstep, y0 + k + ({k0}), NY) * X;",
              "  const I plane = (I)NY * X;",
              "  const int xw = xg_near(xg_overstep, x0 - 1, X), xe = xg_near(xg_overstep, xl + 1, X);",
              "  auto base = [&](int a) { return (I)xg_near(xg_overstep, a, A) * plane; };",
              "  auto ok_row = [&](I) { return true; };"]
    for b in bufs:
        t, v, np_ = em.elem(b[0]), em.bname(b), hi[b] - lo[b]
        K += [f"  const {t}* __restrict__ {v} = p.{v} + x0 + lane;",
              f"  const {t}* __restrict__ {v}_s = p.{v};",
              f"  {t} c{v}[U + {np_}][R][J], n{v}[U][R][J];  // planes a {lo[b]:+d} .. , the U planes after them"]
        if rows[b]:
            K.append(f"  {t} h{v}[U][2][J], hn{v}[U][2][J];  // the rows next to the strip, of planes a .. and of the next")
        if side[b]:
            K.append(f"  {t} s{v}[U][R][2], sn{v}[U][R][2];  // the columns next to the strip")
    K.append(f"  {T}* __restrict__ out = p.{dst} + x0 + lane;")

    def load_plane(b, dest, a, cond):
        t, v = em.elem(b[0]), em.bname(b)
        return ["      {", f"        const bool oka = {cond};", f"        const I pl = base({a});",
                "#pragma unroll", "        for (int r = 0; r < R; ++r) {",
                f"          const I q = pl + yo[r - ({k0})];", "          const bool ok = oka && ok_row(q);",
                "#pragma unroll",
                f"          for (int j = 0; j < J; ++j) {dest}[r][j] = ok && in[j] ? {v}[q + 32 * j] : ({t})0;",
                "        }", "      }"]

    def load_rim(b, hd, sd, a, cond):
        t, v = em.elem(b[0]), em.bname(b)
        out = ["      {", f"        const bool oka = {cond};", f"        const I pl = base({a});"]
        for d in rows[b]:
            k = 0 if d < 0 else 1
            out += ["        {", f"          const I q = pl + yo[{0 if d < 0 else R - k0}];",
                    "          const bool ok = oka && ok_row(q);", "#pragma unroll",
                    f"          for (int j = 0; j < J; ++j) {hd}[{k}][j] = ok && in[j] ? {v}[q + 32 * j] : ({t})0;",
                    "        }"]
        if side[b]:
            out += ["#pragma unroll", "        for (int r = 0; r < R; ++r) {", f"          const I q = pl + yo[r - ({k0})];"]
            for d in side[b]:
                k, who, x = (0, "first", "xw") if d < 0 else (1, "last", "xe")
                out.append(f"          {sd}[r][{k}] = {who} && oka && ok_row(q + {x}) ? {v}_s[q + {x}] : ({t})0;")
            out.append("        }")
        return out + ["      }"]
    K += ["  // mask words of the strip's rows, lane j holding those of columns 32 j: loaded with the planes ahead",
          "  const int W = (X + 31) / 32, wx = x0 / 32 + lane;",
          "  uint32_t wc[U][R], wn[U][R];",
          "  auto words = [&](uint32_t (&w)[R], int a) {",
          "#pragma unroll", "    for (int r = 0; r < R; ++r)",
          "      w[r] = MASKED && a < ab && y0 + r < NY && lane < J && wx < W ? bits[((I)a * NY + y0 + r) * W + wx] : 0u;",
          "  };",
          "#pragma unroll", "  for (int u = 0; u < U; ++u) words(wc[u], aa + u);"]
    for b in bufs:
        v, np_ = em.bname(b), hi[b] - lo[b]
        K += ["#pragma unroll", f"  for (int k = 0; k < U + {np_}; ++k) {{"]
        K += load_plane(b, f"c{v}[k]", f"aa + k + ({lo[b]})", f"aa + k + ({lo[b]}) <= ab") + ["  }"]
        if rows[b] or side[b]:
            K += ["#pragma unroll", "  for (int u = 0; u < U; ++u) {"]
            K += load_rim(b, f"h{v}[u]", f"s{v}[u]", "aa + u", "aa + u < ab") + ["  }"]
    K += ["#pragma unroll 1", "  for (int a = aa; a < ab; a += U) {",
          "    // the next planes and their rim",
          "#pragma unroll", "    for (int u = 0; u < U; ++u) {", "      words(wn[u], a + U + u);"]
    for b in bufs:
        v = em.bname(b)
        K += load_plane(b, f"n{v}[u]", f"a + U + u + ({hi[b]})", f"a + U + u + ({hi[b]}) <= ab")
        K += load_rim(b, f"hn{v}[u]", f"sn{v}[u]", "a + U + u", "a + U + u < ab")
    K += ["    }", "#pragma unroll", "    for (int u = 0; u < U; ++u)", "#pragma unroll", "      for (int r = 0; r < R; ++r) {"]
    cond = " && ".join((["a + u < ab"] if U > 1 else []) + (["y0 + r < NY"] if dim == 3 else []))
    K += [f"        if ({cond or 'true'}) {{", "        const I q = ((I)(a + u) * NY + y0 + r) * X;  // the cell itself"]
    for b in bufs:
        t, v = em.elem(b[0]), em.bname(b)
        cur = f"c{v}[u + {-lo[b]}][r]"
        for d in side[b]:
            K += [f"        {t} {'W' if d < 0 else 'E'}{v}[J];", "#pragma unroll", "        for (int j = 0; j < J; ++j) {"]
            if d < 0:
                K += [f"          W{v}[j] = __shfl_sync(FULL, lane == 31 && j ? {cur}[j ? j - 1 : 0] : {cur}[j], "
                      "(lane + 31) & 31);",
                      f"          if (j == 0 && first) W{v}[j] = s{v}[u][r][0];"]
            else:
                K += [f"          E{v}[j] = __shfl_sync(FULL, lane == 0 && j < J - 1 ? {cur}[j < J - 1 ? j + 1 : j] : "
                      f"{cur}[j], (lane + 1) & 31);",
                      f"          if (last && j == js) E{v}[j] = s{v}[u][r][1];"]
            K.append("        }")
    K += ["#pragma unroll", "        for (int j = 0; j < J; ++j) {"]
    names, local = {}, {}
    for st, ld in s.loads:
        if ld not in local:
            local[ld] = f"l{len(local)}"
            b = (ld.slot, ld.level, ld.version)
            v, o = em.bname(b), ld.offset
            z = f"u + {o[walk] - lo[b]}"
            if o[2]:
                src = f"{'W' if o[2] < 0 else 'E'}{v}[j]"
            elif dim == 3 and o[1] < 0:
                src = f"r > 0 ? c{v}[{z}][r > 0 ? r - 1 : 0][j] : h{v}[u][0][j]"
            elif dim == 3 and o[1] > 0:
                src = f"r < R - 1 ? c{v}[{z}][r < R - 1 ? r + 1 : r][j] : h{v}[u][1][j]"
            else:
                src = f"c{v}[{z}][r][j]"
            K.append(f"          const {em.elem(ld.slot)} {local[ld]} = {src};")
        names[id(st)] = local[ld]
    env = SweepEnv(gen, em.hoist_map, names, em.div_map, em.mul_map)
    val = gen.expr(s.stmt.value, env)
    K += ["          bool live = in[j];",
          "          if (MASKED) {  // bit set: the sweep leaves the cell alone",
          "            const uint32_t word = __shfl_sync(FULL, wc[u][r], j);"]
    if s.implicit:
        b = (s.slot, s.level, s.read_version_of_target)
        K.append(f"            if (live && (word >> lane & 1u)) out[q + 32 * j] = c{em.bname(b)}[u + {-lo[b]}][r][j];")
    K += ["            live = live && !(word >> lane & 1u);", "          }",
          f"          if (live) out[q + 32 * j] = {val};", "        }", "        }", "      }"]
    for b in bufs:
        v, np_ = em.bname(b), hi[b] - lo[b]
        K += ["#pragma unroll", "    for (int r = 0; r < R; ++r)", "#pragma unroll", "      for (int j = 0; j < J; ++j) {"]
        if np_:
            K += ["#pragma unroll", f"        for (int k = 0; k < {np_}; ++k) c{v}[k][r][j] = c{v}[k + U][r][j];"]
        K += ["#pragma unroll", f"        for (int u = 0; u < U; ++u) c{v}[u + {np_}][r][j] = n{v}[u][r][j];", "      }"]
        if rows[b]:
            K += ["#pragma unroll", "    for (int u = 0; u < U; ++u)", "#pragma unroll",
                  f"      for (int j = 0; j < J; ++j) {{ h{v}[u][0][j] = hn{v}[u][0][j]; h{v}[u][1][j] = hn{v}[u][1][j]; }}"]
        if side[b]:
            K += ["#pragma unroll", "    for (int u = 0; u < U; ++u)", "#pragma unroll",
                  f"      for (int r = 0; r < R; ++r) {{ s{v}[u][r][0] = sn{v}[u][r][0]; s{v}[u][r][1] = sn{v}[u][r][1]; }}"]
    K += ["#pragma unroll", "    for (int u = 0; u < U; ++u)", "#pragma unroll",
          "      for (int r = 0; r < R; ++r) wc[u][r] = wn[u][r];", "  }", "}"]
    return "\n".join(K)


def apply_lines(em, pl) -> list:
    """``xgl_<name>_<gid>_strips(G)``: 1 + the strip shape that the main sweep runs on, or 0:
    untuned grids of one shape, large enough, wide enough for a shape."""
    n, gid = em.name, em.gid
    dim, bufs = pl
    s = em.g.sweeps[0]
    phases = len(em.g.sweeps) - 1
    floor = (MIN_CELLS_PHASES if phases else MIN_CELLS)[dim]
    if dim == 2 and phases >= MANY_PHASES:
        floor = f"(dom.x % 32 == 0 ? {MIN_CELLS_MANY} : {floor})"
    L = [f"static int xgl_{n}_{gid}_strips(const xg_grid* G) {{",
         f"  const xg_ext dom = xg_extent(&G[{s.slot}]);",
         f"  if (!xg_zstage_{n} || xg_tiling_set_{n}[{gid}] || dom.z * dom.y * dom.x < {floor}) return 0;",
         "  if (dom.x > 0x3fffffffLL) return 0;  // a strip's columns and their neighbours are int"]
    L += [f"  if (!xg_same_ext(xg_extent(&G[{slot}]), dom)) return 0;"
          for slot in em.slots_used(em.g.sweeps) if slot != s.slot]
    if dim == 3 and em.fp64_ops() and not em.walks():
        L.append(f"  if (dom.x % 32 == 0 || dom.z < {MIN_PLANES_FP64}) return 0;")
    for v, ((J, R, _, _), fill) in enumerate(shapes(em, pl)):
        rows = f" && dom.y > {R}" if dim == 3 else ""  # a strip's rows reach at most one period beyond the grid
        L.append(f"  if (100 * dom.x >= {fill} * {32 * J} * ((dom.x + {32 * J - 1}) / {32 * J}){rows}) return {v + 1};")
    return L + ["  return 0;", "}"]


def launch(em, tag: str, pl, site: int, mask: str, ind: str) -> list:
    """Host lines (parameters ``p``, stream ``s``, ``shape`` from ``xgl_<name>_<gid>_strips``):
    run the sweep on strips; the caller closes the two blocks that stay open."""
    n, gid = em.name, em.gid
    dim, bufs = pl
    kinds = [shape for shape, _ in shapes(em, pl)]
    kname = f"xgk_{n}_{gid}_{tag}_rs"
    a, y = ("p.Z", "p.Y") if dim == 3 else ("p.Y", "1")
    pick = lambda xs: " : ".join(f"shape == {v + 1} ? {x}" for v, x in enumerate(xs)) + " : 0"
    L = ["{",
         "  int alen = 0;",
         "  int64_t nsx = 0, nsy = 0, nw = 0, nz = 0;",
         "  const uint32_t* bits = NULL;",
         f"  XG_TRY(xg_strip_chunks({a}, {y}, p.X, {pick([32 * v[0] for v in kinds])}, {pick([v[1] for v in kinds])}, "
         f"{pick([WARPS * v[3] for v in kinds])}, &alen, &nsx, &nsy, &nw));",
         f"  XG_TRY(xg_mask_nonzero({mask}, &nz));",
         f"  if (nz != 0) XG_TRY(xg_mask_bits({mask}, &bits));",
         "  if (nw <= 0x3fffffffLL) {",
         f"    if (xg_hook_{n}) XG_TRY(xg_hook_{n}(xg_hook_ctx_{n}, {site}, G, {len(em.gen.slots)}, s));",
         f"    xg_prof_launch({site}, s);",
         f"    const unsigned nb = (unsigned)((nw + {WARPS - 1}) / {WARPS});",
         "    const bool small = xg_small_index(p.Z, p.Y, p.X);"]
    first = True
    for v in range(len(kinds)):
        for it, c in (("int", "small"), ("int64_t", "!small")):
            for m, cm in (("false", "nz == 0"), ("true", "nz != 0")):
                L.append(f"    {'' if first else 'else '}if (shape == {v + 1} && {c} && {cm}) {kname}{v}<{it}, {m}>"
                         f"<<<nb, {WARPS * 32}, 0, s>>>(p, alen, (int)nsx, (int)nsy, (int)nw, bits);")
                first = False
    L += ["    XG_CUDA(cudaGetLastError());", f"    xg_prof_end({site}, s);"]
    return [ind + line for line in L]
