// k2b.cu -- the 2D block-step kernel: one launch takes Ez, Hx, Hy (TM) or Ex,
// Ey, Hz (TE) of the whole grid several steps on (the loop body of
// 2D/.../program.f90:320-471).
//
// A block owns a tile of the grid and holds it, widened by a halo of one cell
// per step on each side, in registers: a warp owns R rows of 32 vectors of V
// cells, a thread the R vectors of its column.  A half step reads the cell to
// the left (E) or right (H) from the neighbouring lane by a shuffle, the row
// below (E) or above (H) from the thread's own registers or, at the edge of
// the warp's rows, from the row the warp beside it left in shared memory: one
// row written and one read per warp and half step.  The halo's outermost valid
// cell falls away with every half step; what is left after the last one is the
// tile, which is stored.  The halo belongs to the neighbouring tiles, which
// compute the same values themselves, so tiles are independent of one another.
// That works because a launch reads one set of buffers and stores to the
// other (a ping-pong pair).
//
// Why this shape.  One launch per half step is bound at 2048^2 and below by
// the latency of its launches and loads, and above by the traffic of a pass
// per half step.  Here a launch moves each field once in and once out for all
// its steps, and the arithmetic in between runs from registers.
//
// Every cell is handled here: the split-PML shell, the edges of the main
// range, source rows, monitored rows (each step stages its samples) and the
// dispersive cells.  Those of a tile are listed at commit; their state is held
// in shared memory between the steps (beyond its capacity in a scratch
// buffer), their curl is handed over by the thread that owns the cell, and the
// new E handed back.  The arithmetic of every cell is that of the half-step
// kernels (k2d.cu), term for term, so the results equal theirs bit for bit.
#include <cuda_runtime.h>

#include "fdtd_internal.h"
#include "kcommon.cuh"

namespace fdtd {

namespace {

typedef float T;

template <int M>
struct Mode {
  static constexpr int value = M;
};

__device__ __forceinline__ int wrap_i(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

// whether the cells lo..hi of row j hold a probe, or a sample of any kind
__device__ __forceinline__ bool row_probed(const StepParams<T> &p, int j, int lo, int hi) {
  for (int q = 0; q < p.nprobe; ++q)
    if (p.probe[q].cell[1] == j && p.probe[q].cell[0] >= lo && p.probe[q].cell[0] <= hi) return true;
  return false;
}
__device__ __forceinline__ bool row_sampled(const StepParams<T> &p, int j, int lo, int hi) {
  for (int q = 0; q < p.nmon; ++q) {
    const Monitor &m = p.mon[q];
    if (j >= m.lo[1] && j <= m.hi[1] && hi >= m.lo[0] && lo <= m.hi[0]) return true;
  }
  return row_probed(p, j, lo, hi);
}

// Flags (SF_*) of the warp strips of the plan's tiles, from the material ids and
// the set-up's ranges, with the id of a strip's main cells where they have one.
// Sources count where one of the strip's cells is driven, samples where an owned
// cell is: by rows alone a vertical line of either would make every tile of the
// grid a general one (2048^2 with a square of line monitors: 43.9 us a step, 13.9
// like this; the half-step kernels 27.7).
__global__ void tile_flags_kernel(const __grid_constant__ StepParams<T> p, const Tile2 *tiles, int ntiles, int R, int NW,
                                  int W, BlockGeom g, uint32_t *out) {
  const int strip = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (strip >= ntiles * NW) return;
  const int t = strip / NW, w = strip % NW;
  const int x0 = tiles[t].tx * g.ox - g.hx, y0 = tiles[t].y0 - g.hy + w * R;
  unsigned f = 0;
  int lo = 256, hi = -1;  // of the main cells' ids
  for (int r = 0; r < R; ++r) {
    int j = y0 + r;
    if (g.per[1]) j = wrap_i(j, g.ny);
    const bool jin = j >= 0 && j < g.ny;
    const int rf = jin ? p.rowflag[j] : 0, xo = tiles[t].tx * g.ox;
    if ((rf & ROW_SAMPLE) && row_sampled(p, j, xo, min(xo + g.ox, g.nx) - 1)) f |= SF_SMP | 0x10000u << r;
    for (int x = lane; x < W; x += 32) {
      int i = x0 + x;
      if (g.per[0]) i = wrap_i(i, g.nx);
      const bool in = jin && i >= 0 && i < g.nx;
      const bool shell = in && g.split && (i < g.slo[0] || i > g.shi[0] || j < g.slo[1] || j > g.shi[1]);
      const bool main = in && !shell && i >= g.mlo[0] && i <= g.mhi[0] && j >= g.mlo[1] && j <= g.mhi[1];
      if (!main) f |= SF_GEN;
      if (shell) f |= SF_SHELL;
      if (in && (rf & ROW_SRC))
        for (int q = 0; q < p.nsrc; ++q)
          if (i >= p.src[q].lo[0] && i <= p.src[q].hi[0] && j >= p.src[q].lo[1] && j <= p.src[q].hi[1]) f |= SF_SRC;
      if (main) {
        const int id = p.mat[(long long)j * g.nx + i];
        lo = min(lo, id);
        hi = max(hi, id);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    f |= __shfl_xor_sync(0xffffffffu, f, o);
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (hi >= 0 && (lo != hi || hi >= kAdeId)) f |= SF_MIX;
  if (lane == 0) out[strip] = f | (unsigned)(hi < 0 || (f & SF_MIX) ? g.id0 : hi) << 8;
}

// One tile.  GEN: any cells, sources and samples; else every cell is a main cell
// and each strip has one material, and only fields, halo and arithmetic remain.
// The rows of a strip are unrolled (their fields are registers), so R bounds the
// code, and a general row's is five times a plain one's: the code of a step has
// to fit the instruction cache, or its fetch bounds the step (of a tile in the
// PML: 14 us with 6 general rows a warp, 2 us with 4, 1.2 us with 2).  So general
// tiles spread the same rows over twice the warps, in a launch of their own
// beside the plain tiles', which then need neither its registers nor its shared
// memory.
template <int L, int V, int R, int NW, int KIND, bool GEN>
__device__ __forceinline__ void block_tile(const StepParams<T> &p, const BlockPlan &pl, const Tile2 &tl) {
  constexpr int W = 32 * V, H = R * NW, NT = 32 * NW;
  constexpr int NC = L == 3 ? 1 : 2;            // E components
  constexpr bool TM = L == 3;
  static_assert(R * V <= 32 && (!GEN || R * (V + 1) <= 32), "a thread's cells are bits of one word");
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T *const topH = (T *)sm_raw, *const botE = topH + NW * W;
  T *const xsm = botE + NW * W, *const ysm = xsm + 4 * W;  // PML profiles f1 f2 g1 g2 along the tile's x and y
  T *const srcv = ysm + 4 * H;                   // source values, [step][source]
  int *const rowcnt = (int *)(srcv + kBlockSteps * kMaxSrc), *const rowj = rowcnt + 32;  // rows with samples
  T *const spS = (T *)(rowj + 4);                // the stored split part, [H][W]
  // per cell, [H][W] each: Ku/eps, or a dispersive cell's E (TE: Ex); TE: a
  // dispersive cell's Ey; H of the strips around dispersive cells (TM: Hx, Hy;
  // TE: Hz)
  T *const crv = (T *)(sm_raw + pl.off_crv), *const eyv = crv + H * W;
  T *const hav = crv + NC * H * W, *const hbv = TM ? hav + H * W : hav;  // with the y and the x derivative
  const int cap = tl.smp ? pl.cap_smp : pl.cap;  // dispersive cells with their state here
  int *const rst = (int *)(sm_raw + pl.off_st);  // first entry per row
  T *const st = (T *)(rst + (H + 4) / 4 * 4);    // state, [field][comp][cap], and places in the tile
  uint16_t *const ado = (uint16_t *)(st + pl.nf * NC * cap);
  // samples of the launch's steps, [step][row][field][W]: at most kBlockRows rows
  T *const smp = (T *)(sm_raw + pl.off_smp);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t *const sflags = pl.sflags[GEN] + blockIdx.x * NW;
  const unsigned sf = sflags[w];  // flags, the id of the strip's main cells << 8, rows with samples << 16
  const int nx = p.nx, ny = p.ny;
  const int xr = tl.tx * pl.g.ox - pl.g.hx + lane * V;  // the thread's first cell and first row, unwrapped
  const int yr = tl.y0 - pl.g.hy + w * R;
  const bool split = p.pml_mode == 2;
  const bool vecok = V == 1 || p.vec == V;
  auto row_j = [&](int r) { return p.per[1] ? wrap_i(yr + r, ny) : yr + r; };
  auto cell_i = [&](int q) { return p.per[0] ? wrap_i(xr + q, nx) : xr + q; };
  // per cell of a row of the thread: in the grid; owned by the tile.  Per cell
  // of the thread (bit r V + q): split-PML cells, main cells
  unsigned xin = 0, xow = 0, shm = 0, mnm = 0, adem = 0;
  {
    unsigned xsh = 0, xmn = 0;
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const int i = cell_i(q);
      const unsigned b = 1u << q;
      if (i >= 0 && i < nx) xin |= b;
      if (split && (i < p.slo[0] || i > p.shi[0])) xsh |= b;
      if (i >= p.mlo[0] && i <= p.mhi[0]) xmn |= b;
      const int lx = lane * V + q;
      if (lx >= pl.g.hx && lx < pl.g.hx + pl.g.ox && xr + q < nx) xow |= b;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = row_j(r);
      const bool jin = j >= 0 && j < ny, jsh = split && (j < p.slo[1] || j > p.shi[1]);
      const unsigned sh = jin ? (jsh ? xin : xsh & xin) : 0u;
      const unsigned mn = j >= p.mlo[1] && j <= p.mhi[1] ? xmn & ~sh : 0u;
      shm |= sh << (r * V);
      mnm |= mn << (r * V);
    }
  }
  const int i0 = cell_i(0);  // of aligned vectors
  auto row_own = [&](int r) {
    const int ly = w * R + r;
    return ly >= pl.g.hy && ly < pl.g.hy + tl.oy && yr + r < ny;
  };
  const T cas = __ldg(p.mca + (sf >> 8 & 0xffu));  // Ku/eps of a strip of one material
  // this strip or the one above it may hold dispersive cells
  const bool near = GEN && tl.nade > 0 && ((sf | (w + 1 < NW ? sflags[w + 1] : 0u)) & SF_MIX);
  // rows with a source, and owned rows with samples
  unsigned srow = 0, grow = 0;
  if (GEN && (sf & (SF_SRC | SF_SMP)))
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = row_j(r);
      if ((sf & SF_SRC) && j >= 0 && j < ny && (__ldg(p.rowflag + j) & ROW_SRC)) srow |= 1u << r;
      if ((sf >> (16 + r) & 1u) && p.gather && row_own(r)) grow |= 1u << r;
    }
  // a strip of one material driven by the job's one source
  unsigned srcm = 0;
  T css = T(0);
  if (GEN && p.nsrc == 1 && srow && !(sf & SF_MIX)) {
    css = __ldg(p.mcs + (sf >> 8 & 0xffu));
    const Source &sr = p.src[0];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const int i = cell_i(q), j = row_j(r);
        const unsigned bit = 1u << (r * V + q);
        if ((mnm & bit) && i >= sr.lo[0] && i <= sr.hi[0] && j >= sr.lo[1] && j <= sr.hi[1] && sr.lo[2] <= 0 &&
            sr.hi[2] >= 0 && (TM ? sr.comp == 2 : sr.comp == 0 || sr.comp == 1))
          srcm |= bit;
      }
    srow = 0;
  }
  if (GEN && split) {
    const T *const px[4] = {p.cf1[0], p.cf2[0], p.cg1[0], p.cg2[0]}, *const py[4] = {p.cf1[1], p.cf2[1], p.cg1[1], p.cg2[1]};
    for (int x = threadIdx.x; x < W + H; x += NT) {
      const bool ix = x < W;
      const int g = ix ? tl.tx * pl.g.ox - pl.g.hx + x : tl.y0 - pl.g.hy + x - W;
      const int n = ix ? nx : ny, i = p.per[ix ? 0 : 1] ? wrap_i(g, n) : g;
      T v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = i >= 0 && i < n ? __ldg((ix ? px[u] : py[u]) + i) : T(0);
#pragma unroll
      for (int u = 0; u < 4; ++u) (ix ? xsm + u * W : ysm + u * H - W)[x] = v[u];
    }
  }
  if (GEN && (sf & (SF_MIX | SF_GEN))) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = row_j(r);
      T cv[V];
#pragma unroll
      for (int q = 0; q < V; ++q) cv[q] = cas;
      if (sf & SF_MIX) {
        uint8_t id[V];
#pragma unroll
        for (int q = 0; q < V; ++q) id[q] = 0;
        if (j >= 0 && j < ny) {
          if (vecok) {
            if (xin) vld_ids<V>(p.mat + (long long)j * nx + i0, id);
          } else {
#pragma unroll
            for (int q = 0; q < V; ++q)
              if ((xin >> q) & 1u) id[q] = __ldg(p.mat + (long long)j * nx + cell_i(q));
          }
        }
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const unsigned b = 1u << (r * V + q);
          if ((mnm & b) && id[q] >= kAdeId) adem |= b;
          cv[q] = (mnm & b) && id[q] < kAdeId ? __ldg(p.mca + id[q]) : T(0);
        }
      }
      vst<T, V>(crv + (w * R + r) * W + lane * V, cv);
    }
  }

  pdl_wait();
  pdl_release();

  const int n0 = step_n(p);
  // TM: a = Ez, b = Hx, c = Hy; TE: a = Ex, b = Ey, c = Hz
  T a[R][V], b[R][V], c[R][V];
  {
    const T *const fa = TM ? p.ez : p.ex, *const fb = TM ? p.hx : p.ey, *const fc = TM ? p.hy : p.hz;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = row_j(r);
      const bool jin = j >= 0 && j < ny;
#pragma unroll
      for (int q = 0; q < V; ++q) a[r][q] = b[r][q] = c[r][q] = T(0);
      if (vecok) {
        if (jin && xin) {
          const long long o = (long long)j * nx + i0;
          vld<T, V>(fa + o, a[r]);
          vld<T, V>(fb + o, b[r]);
          vld<T, V>(fc + o, c[r]);
        }
      } else if (jin) {
#pragma unroll
        for (int q = 0; q < V; ++q)
          if ((xin >> q) & 1u) {
            const long long o = (long long)j * nx + cell_i(q);
            a[r][q] = fa[o];
            b[r][q] = fb[o];
            c[r][q] = fc[o];
          }
      }
    }
  }
  if (GEN && (sf & SF_SHELL)) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = row_j(r);
      const bool jin = j >= 0 && j < ny;
      T v[V] = {};
      if (vecok) {
        if (jin && xin) vld<T, V>(p.sp[0] + (long long)j * nx + i0, v);
      } else if (jin) {
#pragma unroll
        for (int q = 0; q < V; ++q)
          if ((xin >> q) & 1u) v[q] = p.sp[0][(long long)j * nx + cell_i(q)];
      }
      vst<T, V>(spS + (w * R + r) * W + lane * V, v);
    }
  }
  // entry e's state: base, stride between fields, index
  auto st_of = [&](int e, T *&base, int &stride, int &idx) __attribute__((always_inline)) {
    if (e < cap) {
      base = st;
      stride = cap;
      idx = e;
    } else {
      base = pl.scratch;
      stride = pl.scr_stride;
      idx = tl.scr0 + e - cap;
    }
  };
  for (int e = threadIdx.x; GEN && e < tl.nade; e += NT) {
    const uint2 en = __ldg(pl.ade + tl.ade0 + e);
    const int slot = (int)(en.x & 0x7fffffffu);
    const int o = (int)(en.y & 0xffffu);
    if (e < cap) ado[e] = (uint16_t)o;
    // rst[y]: the first entry of row y or above (the list is in the order of rows)
    const int y0 = e > 0 ? (int)(__ldg(&pl.ade[tl.ade0 + e - 1].y) & 0xffffu) / W + 1 : 0;
    for (int y = y0; y <= o / W; ++y) rst[y] = e;
    if (e == tl.nade - 1)
      for (int y = o / W + 1; y <= H; ++y) rst[y] = tl.nade;
    T *base;
    int stride, idx;
    st_of(e, base, stride, idx);
    for (int f = 0; f < pl.nf; ++f)
#pragma unroll
      for (int u = 0; u < NC; ++u)
        base[(long long)(f * NC + u) * stride + idx] = p.ade_state[(long long)(f * 3 + u) * p.ade_stride + slot];
  }
  for (int t = threadIdx.x; GEN && t < pl.ks * p.nsrc; t += NT)
    srcv[t] = T(p.srcval_tab[(long long)(n0 - 1) * p.nsrc + t]);
  // the owned rows with samples: their number in the tile, in the order of
  // warps; more than kBlockRows of them go straight to the stage ring
  int srow0 = 0, nsrow = 0;
  if (GEN && tl.smp) {
    if (lane == 0) rowcnt[w] = __popc(grow);
    __syncthreads();
    for (int u = 0; u < NW; ++u) {
      if (u < w) srow0 += rowcnt[u];
      nsrow += rowcnt[u];
    }
    if (nsrow <= kBlockRows && lane == 0)
      for (unsigned m = grow, k = srow0; m; m &= m - 1, ++k) rowj[k] = yr + __ffs(m) - 1;
  }
  // the thread's cells with a probe (bits of grow above its rows': the loop over
  // the steps has no register to spare)
  if (GEN && grow && p.nprobe > 0)
#pragma unroll 1
    for (unsigned m = grow; m; m &= m - 1) {
      const int rr = __ffs(m) - 1;
#pragma unroll 1
      for (int q = 0; q < V; ++q)
        if (((xow >> q) & 1u) && row_probed(p, yr + rr, xr + q, xr + q)) grow |= 1u << (R + rr * V + q);
    }
  if (GEN && KIND != MK_GOLD && adem) {  // their E before the first step
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int q = 0; q < V; ++q)
        if (adem & (1u << (r * V + q))) {
          crv[(w * R + r) * W + lane * V + q] = a[r][q];
          if (!TM) eyv[(w * R + r) * W + lane * V + q] = b[r][q];
        }
  }
  const bool tsrc = __syncthreads_or(GEN && (sf & SF_SRC));  // the tile has rows with a source

  // sum of step s's source values that drive component comp at cell (i, j)
  auto src_at = [&](int s, int comp, int i, int j) __attribute__((always_inline)) {
    T v = T(0);
    for (int q = 0; q < p.nsrc; ++q) {
      const Source &sr = p.src[q];
      if (sr.comp == comp && i >= sr.lo[0] && i <= sr.hi[0] && j >= sr.lo[1] && j <= sr.hi[1] && sr.lo[2] <= 0 &&
          sr.hi[2] >= 0)
        v += srcv[s * p.nsrc + q];
    }
    return v;
  };

#pragma unroll 1
  for (int s = 0; s < pl.ks; ++s) {
    const int n = n0 + s;
    // strips whose rows no owned cell needs any more take no part
    const bool need_e = w * R + R - 1 >= s + 1 && w * R <= H - 1 - s;
    const bool need_h = w * R + R - 1 >= s + 1 && w * R <= H - 2 - s;

    // E of row r; below: the row below of the H component with a y
    // derivative.  MODE 0: main cells of one material; 1: main cells of any
    // material; 2: any cells.  Nothing branches inside a row, so that the loads
    // and chains of a strip's rows overlap.
    auto erow = [&](auto mode, int r, const T (&below)[V]) __attribute__((always_inline)) {
      constexpr int MODE = decltype(mode)::value;
      const T left = __shfl_up_sync(0xffffffffu, c[r][V - 1], 1);
      T f1x[V], f2x[V], ox[V], cv[V], f1y = T(0), f2y = T(0);
      const int o = (w * R + r) * W + lane * V;
#pragma unroll
      for (int q = 0; q < V; ++q) cv[q] = cas;
      if (MODE >= 1) vld<T, V>(crv + o, cv);  // a dispersive cell's is its old E: its result is replaced below
      if (MODE == 2) {
        vld<T, V>(xsm + lane * V, f1x);
        vld<T, V>(xsm + W + lane * V, f2x);
        f1y = ysm[w * R + r];
        f2y = ysm[H + w * R + r];
        if (TM) {
          vld<T, V>(spS + o, ox);
        }
      }
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const T lft = q ? c[r][q - 1] : left;
        const T dxp = c[r][q] - lft, dyp = TM ? -b[r][q] + below[q] : c[r][q] - below[q];
        const unsigned bit = 1u << (r * V + q);
        T na, nb = T(0);
        if (TM) na = a[r][q] + cv[q] * (dxp + dyp);
        else {
          na = a[r][q] + cv[q] * dyp;
          nb = b[r][q] - cv[q] * dxp;
        }
        bool up = true;  // an updated cell
        if (MODE == 2) {
          const bool sh = shm & bit;
          up = (shm | mnm) & bit;
          if (TM) {
            const T py = a[r][q] - ox[q];
            const T nezx = lin2(f1x[q], ox[q], f2x[q], dxp);
            const T nezy = lin2(f1y, py, f2y, dyp);
            ox[q] = sh ? nezx : ox[q];
            na = sh ? nezx + nezy : na;
          } else {
            na = sh ? lin2(f1y, a[r][q], f2y, dyp) : na;
            nb = sh ? lin2(f1x[q], b[r][q], f2x[q], -c[r][q] + lft) : nb;
          }
        }
        a[r][q] = up ? na : a[r][q];
        if (!TM) b[r][q] = up ? nb : b[r][q];
      }
      if (MODE == 2 && TM) vst<T, V>(spS + o, ox);
    };
    // H of row r; up: the row above of the E component with a y derivative
    auto hrow = [&](auto mode, int r, const T (&up)[V]) __attribute__((always_inline)) {
      constexpr int MODE = decltype(mode)::value;
      const T right = __shfl_down_sync(0xffffffffu, TM ? a[r][0] : b[r][0], 1);
      T g1x[V], g2x[V], ox[V], g1y = T(0), g2y = T(0);
      const int o = (w * R + r) * W + lane * V;
      if (MODE == 2) {
        vld<T, V>(xsm + 2 * W + lane * V, g1x);
        vld<T, V>(xsm + 3 * W + lane * V, g2x);
        g1y = ysm[2 * H + w * R + r];
        g2y = ysm[3 * H + w * R + r];
        if (!TM) {
          vld<T, V>(spS + o, ox);
        }
      }
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const T rgt = q < V - 1 ? (TM ? a[r][q + 1] : b[r][q + 1]) : right;
        const unsigned bit = 1u << (r * V + q);
        T nb = T(0), nc;
        if (TM) {
          nb = b[r][q] + p.ku * (-up[q] + a[r][q]);
          nc = c[r][q] + p.ku * (rgt - a[r][q]);
        } else {
          const T curlE = ((rgt - b[r][q]) - up[q]) + a[r][q];
          nc = c[r][q] - p.ku * curlE;
        }
        bool upd = true;
        if (MODE == 2) {
          const bool sh = shm & bit;
          upd = (shm | mnm) & bit;
          if (TM) {
            nb = sh ? lin2(g1y, b[r][q], g2y, -up[q] + a[r][q]) : nb;
            nc = sh ? lin2(g1x[q], c[r][q], g2x[q], rgt - a[r][q]) : nc;
          } else {
            const T py = c[r][q] - ox[q];
            // each as the half-step kernels of this vector width round it
            const T dy = up[q] - a[r][q], dx = -rgt + b[r][q];
            const T nhzy = vecok ? lin2(g1y, py, g2y, dy) : lin2(g2y, dy, g1y, py);
            const T nhzx = vecok ? lin2(g1x[q], ox[q], g2x[q], dx) : lin2(g2x[q], dx, g1x[q], ox[q]);
            ox[q] = sh ? nhzx : ox[q];
            nc = sh ? nhzy + nhzx : nc;
          }
        }
        if (TM) b[r][q] = upd ? nb : b[r][q];
        c[r][q] = upd ? nc : c[r][q];
      }
      if (MODE == 2 && !TM) vst<T, V>(spS + o, ox);
    };
    // all rows of a strip but the one that needs another warp's row
    auto e_rows = [&](auto mode) __attribute__((always_inline)) {
#pragma unroll
      for (int r = R - 1; r >= 1; --r) erow(mode, r, TM ? b[r - 1] : c[r - 1]);
    };
    auto h_rows = [&](auto mode) __attribute__((always_inline)) {
#pragma unroll
      for (int r = 0; r < R - 1; ++r) hrow(mode, r, a[r + 1]);
    };
    const bool gen = GEN && (sf & SF_GEN), mix = GEN && (sf & SF_MIX);

    // ---- E half.  topH is read between this half's barrier and the next one,
    // botE between that one and the next step's first, so each is written and
    // read once between barriers.
    vst<T, V>(topH + w * W + lane * V, TM ? b[R - 1] : c[R - 1]);
    if (GEN && near) {  // H around dispersive cells
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int o = (w * R + r) * W + lane * V;
        vst<T, V>(hav + o, TM ? b[r] : c[r]);
        if (TM) vst<T, V>(hbv + o, c[r]);
      }
    }
    if (need_e) {
      if constexpr (GEN) {
        if (gen) e_rows(Mode<2>());
        else if (mix) e_rows(Mode<1>());
        else e_rows(Mode<0>());
      } else e_rows(Mode<0>());
    }
    __syncthreads();
    if (need_e) {
      T below[V];
#pragma unroll
      for (int q = 0; q < V; ++q) below[q] = T(0);
      if (w > 0) vld<T, V>(topH + (w - 1) * W + lane * V, below);
      if constexpr (GEN) {
        if (gen) erow(Mode<2>(), 0, below);
        else if (mix) erow(Mode<1>(), 0, below);
        else erow(Mode<0>(), 0, below);
      } else erow(Mode<0>(), 0, below);
    }
    // ---- sources of the main cells.  One source over a strip of one material:
    // its cells are bits of srcm.  Else (rare) a row at a time, its cells picked
    // out of the registers, so that the code stands here once.
    if (GEN && need_e && srcm) {
      const T sv = srcv[s];
      if (sv != T(0)) {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int q = 0; q < V; ++q)
            if (srcm & (1u << (r * V + q))) {
              if (TM || p.src[0].comp == 0) a[r][q] = fma1(css, sv, a[r][q]);
              else b[r][q] = fma1(css, sv, b[r][q]);
            }
      }
    } else if (GEN && need_e && srow) {
#pragma unroll 1
      for (unsigned m = srow; m; m &= m - 1) {
        const int rr = __ffs(m) - 1, j = row_j(rr);
        T va[V] = {}, vb[V] = {}, cs[V] = {};
#pragma unroll 1
        for (int q = 0; q < V; ++q) {
          T xa = src_at(s, TM ? 2 : 0, cell_i(q), j), xb = TM ? T(0) : src_at(s, 1, cell_i(q), j), xc = T(0);
          const bool on = ((mnm & ~adem) >> (rr * V + q)) & 1u;  // the dispersive update adds its own
          if (on) xc = __ldg(p.mcs + __ldg(p.mat + (long long)j * nx + cell_i(q)));
          else xa = xb = T(0);
#pragma unroll
          for (int u = 0; u < V; ++u)
            if (u == q) {
              va[u] = xa;
              vb[u] = xb;
              cs[u] = xc;
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int q = 0; q < V; ++q)
            if (r == rr) {
              if (va[q] != T(0)) a[r][q] = fma1(cs[q], va[q], a[r][q]);
              if (!TM && vb[q] != T(0)) b[r][q] = fma1(cs[q], vb[q], b[r][q]);
            }
      }
    }
    // ---- dispersive cells, by the threads of the tile's list: from the H (and
    // old E) of the strips around them in shared memory, the new E back through it
    if (GEN && tl.nade > 0) {  // uniform over the block
      __syncthreads();
      // the entries of the rows that owned cells still need
      const int eb = rst[s + 1], ee = rst[H - s];
      auto ade_pass = [&](auto one, int e0, int e1, T *base, int stride, int shift) __attribute__((always_inline)) {
        constexpr bool ONE = decltype(one)::value;  // one material: its coefficients are constant operands
#pragma unroll 1
        for (int e = e0 + threadIdx.x; e < e1; e += NT) {
          int o, id = kAdeId;
          if (ONE) o = ado[e];
          else {
            const uint2 en = __ldg(pl.ade + tl.ade0 + e);
            o = (int)(en.y & 0xffffu);
            id = (int)(en.y >> 16);
          }
          const int idx = e + shift;
          T sa = T(0), sb = T(0);
          if (tsrc) {
            const int xg = tl.tx * pl.g.ox - pl.g.hx + o % W, yg = tl.y0 - pl.g.hy + o / W;
            const int i = p.per[0] ? wrap_i(xg, nx) : xg, j = p.per[1] ? wrap_i(yg, ny) : yg;
            sa = src_at(s, TM ? 2 : 0, i, j);
            if (!TM) sb = src_at(s, 1, i, j);
          }
          const AdeCoef<T> &ac = ONE ? p.acp[0] : ade_coef(p, id);
          const AdeCoef<T> *am = p.ac + (id - kAdeId);
          // rows s+1.. only, so the cells below and to the left are the tile's
          const T dxp = hbv[o] - hbv[o - 1], dyp = TM ? -hav[o] + hav[o - W] : hav[o] - hav[o - W];
          const T inc = fma1(p.ku, TM ? dxp + dyp : dyp, sa);
          crv[o] = ade_update_fixed<T, KIND, NC>(base, stride, idx, 0, ac, am, inc, KIND != MK_GOLD ? crv[o] : T(0));
          if (!TM) {
            const T incy = fma1(-p.ku, dxp, sb);
            eyv[o] = ade_update_fixed<T, KIND, NC>(base, stride, idx, 1, ac, am, incy, KIND != MK_GOLD ? eyv[o] : T(0));
          }
        }
      };
      const int em = min(ee, cap);  // entries whose state is in shared memory, and the others
      if (KIND == MK_GOLD && pl.one_ade) ade_pass(Mode<1>(), eb, em, st, cap, 0);
      else ade_pass(Mode<0>(), eb, em, st, cap, 0);
      if (ee > cap) ade_pass(Mode<0>(), eb > cap ? eb : cap, ee, pl.scratch, pl.scr_stride, tl.scr0 - cap);
      __syncthreads();
      if (need_e && (sf & SF_MIX)) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          T ev[V], fv[V];
          vld<T, V>(crv + (w * R + r) * W + lane * V, ev);
          if (!TM) vld<T, V>(eyv + (w * R + r) * W + lane * V, fv);
#pragma unroll
          for (int q = 0; q < V; ++q) {
            const bool d = adem & (1u << (r * V + q));
            a[r][q] = d ? ev[q] : a[r][q];
            if (!TM) b[r][q] = d ? fv[q] : b[r][q];
          }
        }
      }
    }
    // ---- H half
    vst<T, V>(botE + w * W + lane * V, a[0]);
    if (need_h) {
      if constexpr (GEN) {
        if (gen) h_rows(Mode<2>());
        else h_rows(Mode<0>());
      } else h_rows(Mode<0>());
    }
    __syncthreads();
    if (need_h) {
      T up[V];
#pragma unroll
      for (int q = 0; q < V; ++q) up[q] = T(0);
      if (w < NW - 1) vld<T, V>(botE + (w + 1) * W + lane * V, up);
      if constexpr (GEN) {
        if (gen) hrow(Mode<2>(), R - 1, up);
        else hrow(Mode<0>(), R - 1, up);
      } else hrow(Mode<0>(), R - 1, up);
    }
    // ---- samples of the owned cells: the row's fields to shared memory
    if (GEN && grow) {
      if (nsrow <= kBlockRows) {
        T *d = smp + ((s * kBlockRows + srow0) * 3) * W + lane * V;
#pragma unroll
        for (int r = 0; r < R; ++r)
          if ((grow >> r) & 1u) {
            vst<T, V>(d, a[r]);
            vst<T, V>(d + W, b[r]);
            vst<T, V>(d + 2 * W, c[r]);
            d += 3 * W;
          }
      } else {
        // many rows (a line along y, an area): straight to the stage ring, every
        // cell of a monitor's component by a store of its own register
        T *const stg = stage_ring(p) + (long long)(p.slot + s) * p.stage_row;
        const int x0 = tl.tx * pl.g.ox, x1 = min(x0 + pl.g.ox, nx) - 1;
#pragma unroll 1
        for (int t = 0; t < p.nmon; ++t) {
          const Monitor &mo = p.mon[t];
          if (x1 < mo.lo[0] || x0 > mo.hi[0] || yr + R - 1 < mo.lo[1] || yr > mo.hi[1]) continue;
          const int wx = mo.hi[0] - mo.lo[0] + 1;
#pragma unroll 1
          for (int u = 0; u < mo.ncomp; ++u) {
            const int cc = mo.comps[u];
            T *const to = stg + mo.base + (long long)u * mo.ncell + (xr - mo.lo[0]);
            auto put = [&](auto value) __attribute__((always_inline)) {
#pragma unroll
              for (int r = 0; r < R; ++r) {
                const int j = yr + r;
                if (!((grow >> r) & 1u) || j < mo.lo[1] || j > mo.hi[1]) continue;
                T *const row = to + (long long)wx * (j - mo.lo[1]);
#pragma unroll
                for (int q = 0; q < V; ++q)
                  if (((xow >> q) & 1u) && xr + q >= mo.lo[0] && xr + q <= mo.hi[0]) row[q] = value(r, q);
              }
            };
            if (cc == (TM ? 2 : 0)) put([&](int r, int q) { return a[r][q]; });
            else if (cc == (TM ? 3 : 1)) put([&](int r, int q) { return b[r][q]; });
            else if (cc == (TM ? 4 : 5)) put([&](int r, int q) { return c[r][q]; });
            else put([&](int, int) { return T(0); });
          }
        }
      }
#pragma unroll 1
      for (unsigned m = __reduce_or_sync(0xffffffffu, grow >> R); m; m &= m - 1) {
        const int at = __ffs(m) - 1;
        if (!((grow >> (R + at)) & 1u)) continue;
        T va = T(0), vb = T(0), vc = T(0);
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int u = 0; u < V; ++u)
            if (r * V + u == at) {
              va = a[r][u];
              vb = b[r][u];
              vc = c[r][u];
            }
        const T vals[6] = {TM ? T(0) : va, TM ? T(0) : vb, TM ? va : T(0), TM ? vb : T(0), TM ? vc : T(0), TM ? T(0) : vc};
        gather_cell<T>(p, n, xr + at % V, yr + at / V, 0, vals, p.slot + s, false);
      }
    }
  }

  // ---- the samples to the stage ring: a warp copies a row of one component
  // and step
  if (GEN && nsrow > 0 && nsrow <= kBlockRows) {
    __syncthreads();
    T *const stg = stage_ring(p);
    const int x0 = tl.tx * pl.g.ox, x1 = min(x0 + pl.g.ox, nx);
    for (int k = 0; k < nsrow; ++k) {
      const int j = rowj[k];
      for (int t = 0; t < p.nmon; ++t) {
        const Monitor &mo = p.mon[t];
        if (j < mo.lo[1] || j > mo.hi[1]) continue;
        const int lo = max(x0, mo.lo[0]), hi = min(x1 - 1, mo.hi[0]), wx = mo.hi[0] - mo.lo[0] + 1;
        for (int v = w; v < mo.ncomp * pl.ks; v += NW) {
          const int u = v % mo.ncomp, s = v / mo.ncomp, cc = mo.comps[u];
          const int f = cc == (TM ? 2 : 0) ? 0 : cc == (TM ? 3 : 1) ? 1 : cc == (TM ? 4 : 5) ? 2 : -1;
          T *const row = stg + (long long)(p.slot + s) * p.stage_row + mo.base + (long long)u * mo.ncell +
                         (long long)wx * (j - mo.lo[1]) - mo.lo[0];
          const T *const from = smp + ((s * kBlockRows + k) * 3 + (f < 0 ? 0 : f)) * W + pl.g.hx - x0;
          for (int i = lo + lane; i <= hi; i += 32) row[i] = f < 0 ? T(0) : from[i];
        }
      }
    }
  }

  // ---- the tile's cells and states to the other set
  T *const oa = TM ? p.ezo : p.exo, *const ob = TM ? p.hxo : p.eyo, *const oc = TM ? p.hyo : p.hzo;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (!row_own(r)) continue;
    const long long o = (long long)(yr + r) * nx + xr;
    if (vecok) {
      if (xow) {
        vst<T, V>(oa + o, a[r]);
        vst<T, V>(ob + o, b[r]);
        vst<T, V>(oc + o, c[r]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < V; ++q)
        if ((xow >> q) & 1u) {
          oa[o + q] = a[r][q];
          ob[o + q] = b[r][q];
          oc[o + q] = c[r][q];
        }
    }
    if (GEN && (sf & SF_SHELL)) {
      T v[V];
      vld<T, V>(spS + (w * R + r) * W + lane * V, v);
      if (vecok) {
        if (xow) vst<T, V>(p.spo + o, v);
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q)
          if ((xow >> q) & 1u) p.spo[o + q] = v[q];
      }
    }
  }
  for (int e = threadIdx.x; GEN && e < tl.nade; e += NT) {
    const uint2 en = __ldg(pl.ade + tl.ade0 + e);
    if (!(en.x >> 31)) continue;
    const int slot = (int)(en.x & 0x7fffffffu);
    T *base;
    int stride, idx;
    st_of(e, base, stride, idx);
    for (int f = 0; f < pl.nf; ++f)
#pragma unroll
      for (int u = 0; u < NC; ++u)
        pl.ade_out[(long long)(f * 3 + u) * p.ade_stride + slot] = base[(long long)(f * NC + u) * stride + idx];
  }
}

// MB: blocks per SM the registers are bounded for
template <int L, int V, int R, int NW, int MB, int KIND, bool GEN>
__global__ void __launch_bounds__(32 * NW, MB) step2d_block(const __grid_constant__ StepParams<T> p,
                                                           const __grid_constant__ BlockPlan pl) {
  block_tile<L, V, R, NW, KIND, GEN>(p, pl, pl.tiles[(GEN ? 0 : pl.ngen) + blockIdx.x]);
}

}  // namespace

// rows per warp and warps of plain tiles (two blocks per SM) and of general ones
// (one), which hold the same rows
struct Shapes {
  static constexpr int V = 4, RA[kBlockShapes] = {8, 4}, NA[kBlockShapes] = {8, 8}, RB[kBlockShapes] = {4, 2},
                       NB[kBlockShapes] = {16, 16};
};

BlockShape block_shape(int s) { return {Shapes::V, Shapes::RA[s], Shapes::NA[s], Shapes::RB[s], Shapes::NB[s]}; }

void block_smem(BlockPlan &pl, int layout, int max_ade, bool split, bool smp_rows) {
  constexpr int kTop = 224 * 1024;  // one block per SM
  const BlockShape s = block_shape(pl.shape);
  const int W = 32 * s.V, H = s.RB * s.NB;
  int b = (2 * s.NB * W + 4 * (W + H) + kBlockSteps * kMaxSrc) * (int)sizeof(T) + 36 * (int)sizeof(int);
  if (split) b += H * W * (int)sizeof(T);
  pl.off_crv = b;
  b += (max_ade > 0 ? 3 : 1) * H * W * (int)sizeof(T);
  pl.off_st = b;
  if (max_ade > 0) b += (H + 4) / 4 * 4 * (int)sizeof(int);
  // the state of a tile's dispersive cells, and in a tile with samples their
  // buffer behind it (with less room for state)
  const int each = pl.nf * (layout == 3 ? 1 : 2) * (int)sizeof(T) + (int)sizeof(uint16_t);
  const int smp = smp_rows ? kBlockSteps * kBlockRows * 3 * W * (int)sizeof(T) : 0;
  const int top = kTop - 16;
  auto entries = [&](int room) { return max_ade <= 0 || room < 0 ? 0 : room / each < max_ade ? room / each : max_ade; };
  pl.cap = entries(top - b);
  pl.cap_smp = entries(top - b - smp);
  const int e0 = b + (pl.cap * each + 15) / 16 * 16, e1 = b + (pl.cap_smp * each + 15) / 16 * 16;
  pl.off_smp = e1;
  b = e0 > e1 + smp ? e0 : e1 + smp;
  pl.smem = b;
}

template <int L, int S, int KIND, bool GEN>
int launch_block_k(const StepParams<T> &p, const BlockPlan &pl, cudaStream_t s) {
  constexpr int R = GEN ? Shapes::RB[S] : Shapes::RA[S], NW = GEN ? Shapes::NB[S] : Shapes::NA[S];
  constexpr int V = Shapes::V;
  auto kern = step2d_block<L, V, R, NW, GEN ? 1 : 2, KIND, GEN>;
  static std::atomic<unsigned long long> done{0};
  if (!smem_limit(kern, 227 * 1024, done)) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(GEN ? pl.ngen : pl.ntiles - pl.ngen);
  cfg.blockDim = dim3(32 * NW);
  cfg.dynamicSmemBytes = GEN ? pl.smem : 2 * NW * 32 * V * sizeof(T);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p, pl) == cudaSuccess ? 1 : -1;
}

template <int L, int S>
int launch_block_s(const StepParams<T> &p, const BlockPlan &pl, bool gen, cudaStream_t s) {
  if (!gen) return launch_block_k<L, S, MK_GOLD, false>(p, pl, s);
  return p.nade == 0 || p.ade_kind == MK_GOLD ? launch_block_k<L, S, MK_GOLD, true>(p, pl, s)
                                              : launch_block_k<L, S, -1, true>(p, pl, s);
}

int launch_step2d_block(const StepParams<T> &p, const BlockPlan &pl, bool gen, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if ((gen ? pl.ngen : pl.ntiles - pl.ngen) <= 0) return 0;
  if (p.layout == 3) return pl.shape == 0 ? launch_block_s<3, 0>(p, pl, gen, s) : launch_block_s<3, 1>(p, pl, gen, s);
  return pl.shape == 0 ? launch_block_s<2, 0>(p, pl, gen, s) : launch_block_s<2, 1>(p, pl, gen, s);
}

void launch_tile_flags(const StepParams<T> &p, const Tile2 *tiles, int ntiles, int R, int NW, int V, const BlockGeom &g,
                       uint32_t *out, void *stream) {
  const int strips = ntiles * NW;
  if (strips <= 0) return;
  tile_flags_kernel<<<(strips + 7) / 8, 256, 0, (cudaStream_t)stream>>>(p, tiles, ntiles, R, NW, 32 * V, g, out);
}

}  // namespace fdtd
