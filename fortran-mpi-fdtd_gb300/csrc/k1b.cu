// k1b.cu -- the 1D line, a block of steps per launch (the loop body of
// 1D/.../program.f90:217-291).
//
// A block owns a stretch of the line and holds it, widened by a halo of one cell
// per step on each side, in registers, V cells per thread.  The cell to the left
// (E) or right (H) of a thread's cells comes from the next lane by a shuffle, or
// across warps through shared memory.  The halo's outermost valid cell falls away
// with every half step, so a launch of ks steps needs nothing from other blocks:
// it reads one set of buffers and stores its stretch to the other.  The halo
// belongs to the neighbours, which compute the same values themselves.
//
// Why this shape.  A step of the line is a few operations on a few thousand
// cells, so a step costs what its synchronisation costs: 3.7 us with two cluster
// barriers per step (k1d.cu), and FP64 adds the pipe's time of 1,600 cells per
// SM (11 us on the 13004-cell stack).  Here blocks of four warps meet at their
// own barrier only, and the line spreads over all SMs.  Four warps and not one
// of four times the cells per thread, because an SM's FP64 units are shared out
// to its four schedulers: one warp has a quarter of them.  Measured, us per step:
// the 4000-cell gold line FP32 0.31 (k1d.cu 3.2), FP64 1.35; the 13004-cell
// stack with its incident line FP32 0.55, FP64 1.38 (k1d.cu 11).  One warp of 4
// and 8 cells per thread: 0.37, 2.75; 1.0, 4.4.
//
// The PML slabs at the ends continue the line: their cells hold the slab arrays'
// values and take the slab's update, and the coupling rows are what the
// neighbouring cell holds.  The arithmetic of every cell is that of
// line1d_cluster_kernel, term for term, with the same roundings.
#include <cuda_runtime.h>

#include "fdtd_internal.h"
#include "kcommon.cuh"

namespace fdtd {

namespace {

constexpr int kLineWarps = 4;
constexpr int kLineRecords = 16;  // sampled cells of a stretch whose samples are staged in shared memory

// which of a cell's four values (Ex, Hz, incident Ex, Hz) a component code is
__device__ __forceinline__ int line_field(int comp, bool inc) {
  return comp == FDTD_EX ? 0 : comp == FDTD_HZ ? 1 : !inc ? -1 : comp == FDTD_EX_INC ? 2 : comp == FDTD_HZ_INC ? 3 : -1;
}

// the samples of one cell and step, straight to the stage and the probes
template <typename T>
__device__ __noinline__ void line_sample(const LineParams<T> &p, const LineBlock<T> &b, int j, int s, const T *v, bool inc) {
  for (int m = 0; m < p.nmon; ++m) {
    const Monitor &mo = p.mon[m];
    if (j < mo.lo[1] || j > mo.hi[1]) continue;
    for (int c = 0; c < mo.ncomp; ++c) {
      const int f = line_field(mo.comps[c], inc);
      b.stage[(long long)(b.s0 + s) * b.stage_row + mo.base + (long long)c * mo.ncell + (j - mo.lo[1])] = f < 0 ? T(0) : v[f];
    }
  }
  const int n = p.n_first + b.s0 + s;
  for (int m = 0; m < p.nprobe; ++m) {
    const Probe &pr = p.probe[m];
    if (j != pr.cell[1] || n < pr.n_first || n > pr.n_last || n - pr.n_first >= pr.cap) continue;
    for (int c = 0; c < pr.ncomp; ++c) {
      const int f = line_field(pr.comps[c], inc);
      pr.buf[(long long)(n - pr.n_first) * pr.ncomp + c] = f < 0 ? 0.0 : (double)v[f];
    }
  }
}

// KIND: MK_NONE no dispersive cells, MK_GOLD all of one gold material (its state
// in registers), -1 any (state in shared memory)
template <typename T, int V, bool INC, int KIND>
__global__ void __launch_bounds__(32 * kLineWarps) line1d_block(const __grid_constant__ LineParams<T> p,
                                                   const __grid_constant__ LineBlock<T> b) {
  constexpr int W = 32 * V * kLineWarps, NT = 32 * kLineWarps;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T *const srcv = (T *)sm_raw;                     // [step][source]
  T *const rec = srcv + kLineSteps * kMaxSrc;      // samples [step][cell][ex hz ex_inc hz_inc]
  T *const inc_s = rec + kLineSteps * kLineRecords * 4, *const e_s = inc_s + W, *const st = e_s + W;  // KIND -1
  __shared__ uint16_t place[W];                    // a sampled cell's record
  __shared__ int wcount[kLineWarps];
  __shared__ T hs[kLineWarps][2], es[kLineWarps][2];  // a warp's last H and first E, of both lines
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c00 = threadIdx.x * V;
  const int own0 = blockIdx.x * b.own, own1 = min(own0 + b.own, p.N);
  const int j0 = own0 - b.ks + c00;
  const int lo = p.slab_on[0] ? p.ja + 1 : 0, hi = p.slab_on[1] ? p.jb : p.N;  // the cells between the slabs
  const T ku = p.ku;
  const int bd = INC ? p.tfsf_bd : -1;
  // per cell (bit q): main range, constant dielectric, dispersive, slab cells,
  // owned, driven by a grid or an incident source, sampled
  unsigned mnm = 0, dim = 0, adem = 0, slm = 0, owm = 0, sm0 = 0, sm6 = 0, smp = 0;
  T ca[V], cs[V], c0[4][V], c1[4][V];
  int slot[V], ade[V];
#pragma unroll
  for (int q = 0; q < V; ++q) {
    const int j = j0 + q;
    const unsigned bit = 1u << q;
    ca[q] = cs[q] = T(0);
    slot[q] = ade[q] = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) c0[u][q] = c1[u][q] = T(0);
    if (j < 0 || j >= p.N) continue;
    if (j >= own0 && j < own1) owm |= bit;
    if (j < lo || j >= hi) {
      slm |= bit;
      const int side = j < lo ? 0 : 1, r = side == 0 ? j + 1 : j - hi + 1;
      c0[0][q] = p.f1[0][side][r]; c0[1][q] = p.f2[0][side][r]; c0[2][q] = p.g1[0][side][r]; c0[3][q] = p.g2[0][side][r];
      if (INC) {
        c1[0][q] = p.f1[1][side][r]; c1[1][q] = p.f2[1][side][r]; c1[2][q] = p.g1[1][side][r]; c1[3][q] = p.g2[1][side][r];
      }
    } else if (j >= p.mlo && j <= p.mhi) {
      mnm |= bit;
      const MatCoef<T> &m = p.mc[p.mat[j]];
      if (m.kind == MK_DIEL) {
        dim |= bit;
        ca[q] = m.ca;
        cs[q] = m.cs;
      } else if (KIND != MK_NONE && is_ade_kind(m.kind)) {
        adem |= bit;
        slot[q] = b.slot[j];
        ade[q] = m.ade;
      }
      for (int s = 0; s < p.nsrc; ++s)
        if (j >= p.src[s].lo[1] && j <= p.src[s].hi[1]) {
          if (p.src[s].comp == 0) sm0 |= bit;
          if (p.src[s].comp == 6) sm6 |= bit;
        }
    }
    if ((owm & bit)) {
      for (int m = 0; m < p.nmon; ++m)
        if (j >= p.mon[m].lo[1] && j <= p.mon[m].hi[1]) smp |= bit;
      for (int m = 0; m < p.nprobe; ++m)
        if (j == p.probe[m].cell[1]) smp |= bit;
    }
  }
  const bool any_slab = __any_sync(0xffffffffu, slm), any_ade = __any_sync(0xffffffffu, adem);
  // a cell with a source, or beside the total-field boundary, in this warp
  bool tf = false;
#pragma unroll
  for (int q = 0; q < V; ++q) tf |= INC && (j0 + q == bd || j0 + q == bd - 1);
  const bool any_tf = __any_sync(0xffffffffu, tf), any_src = __any_sync(0xffffffffu, sm0 | sm6);
  // records of the sampled cells, in the order of the line
  int first = __popc(smp), nrec = 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, first, o);
    if (lane >= o) first += t;
  }
  if (lane == 31) wcount[w] = first;
  __syncthreads();
  for (int u = 0; u < kLineWarps; ++u) {
    if (u < w) first += wcount[u];
    nrec += wcount[u];
  }
  first -= __popc(smp);
#pragma unroll
  for (int q = 0; q < V; ++q) place[c00 + q] = (uint16_t)(first + __popc(smp & ((1u << q) - 1u)));

  pdl_wait();
  pdl_release();

  T e[V], h[V], ei[V], hv[V];  // Ex, Hz, and of the incident line
#pragma unroll
  for (int q = 0; q < V; ++q) {
    const int j = j0 + q;
    e[q] = h[q] = ei[q] = hv[q] = T(0);
    if (j < 0 || j >= p.N) continue;
    if (slm & (1u << q)) {
      const int side = j < lo ? 0 : 1, r = side == 0 ? j + 1 : j - hi + 1;
      e[q] = p.pex[0][side][r];
      h[q] = p.phz[0][side][r];
      if (INC) {
        ei[q] = p.pex[1][side][r];
        hv[q] = p.phz[1][side][r];
      }
    } else {
      e[q] = p.ex[j];
      h[q] = p.hz[j];
      if (INC) {
        ei[q] = p.exi[j];
        hv[q] = p.hzi[j];
      }
    }
  }
  T gs[6][V];  // gold state
  if (KIND == MK_GOLD) {
#pragma unroll
    for (int f = 0; f < 6; ++f)
#pragma unroll
      for (int q = 0; q < V; ++q)
        gs[f][q] = (adem >> q) & 1u ? p.ade_state[(long long)(f * 3) * p.ade_stride + slot[q]] : T(0);
  } else if (KIND == -1 && any_ade) {
    for (int f = 0; f < p.ade_nf; ++f)
#pragma unroll
      for (int q = 0; q < V; ++q)
        if ((adem >> q) & 1u) st[f * W + c00 + q] = p.ade_state[(long long)(f * 3) * p.ade_stride + slot[q]];
  }
  for (int t = threadIdx.x; t < b.ks * p.nsrc; t += NT) srcv[t] = T(p.srcval[(long long)b.s0 * p.nsrc + t]);
  if (lane == 31) {
    hs[w][0] = h[V - 1];
    hs[w][1] = hv[V - 1];
  }
  __syncthreads();

#pragma unroll 1
  for (int s = 0; s < b.ks; ++s) {
    // ---- E half ----
    T hl = __shfl_up_sync(0xffffffffu, h[V - 1], 1);
    T hil = INC ? __shfl_up_sync(0xffffffffu, hv[V - 1], 1) : T(0);
    if (lane == 0 && w > 0) {
      hl = hs[w - 1][0];
      if (INC) hil = hs[w - 1][1];
    }
    T sx[V], si[V];  // sources and the total-field boundary's term
    bool drive = any_tf;
#pragma unroll
    for (int q = 0; q < V; ++q) sx[q] = si[q] = T(0);
    if (any_src) {
      for (int t = 0; t < p.nsrc; ++t) {
        const T v = srcv[s * p.nsrc + t];
        if (v == T(0)) continue;  // (an added zero changes no sum)
        drive = true;
        const int l = p.src[t].lo[1], u = p.src[t].hi[1], c = p.src[t].comp;
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (j0 + q >= l && j0 + q <= u) {
            if (c == 0) sx[q] += v;
            if (c == 6) si[q] += v;
          }
      }
    }
    if (INC && any_tf) {
#pragma unroll
      for (int q = 0; q < V; ++q)
        if (j0 + q == bd) sx[q] = fma1(-ku, q ? hv[q - 1] : hil, sx[q]);
    }
    T cu[V];
    // a cell's new value: main ca d + x, slab f1 x + (f2 d); one product and sum
    // for both, their factors chosen before it
    auto next = [&](unsigned bit, T x, T d, T k, unsigned on, T f1, T f2) {
      if (!any_slab) return on & bit ? fma1(k, d, x) : x;
      const bool sl = slm & bit;
      const T t = mul1(f2, d);
      const T r = fma1(sl ? f1 : k, sl ? x : d, sl ? t : x);
      return (on | slm) & bit ? r : x;
    };
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const unsigned bit = 1u << q;
      cu[q] = h[q] - (q ? h[q - 1] : hl);
      e[q] = next(bit, e[q], cu[q], ca[q], dim, c0[0][q], c0[1][q]);
      if (INC) ei[q] = next(bit, ei[q], hv[q] - (q ? hv[q - 1] : hil), ku, mnm, c1[0][q], c1[1][q]);
    }
    if (drive) {
#pragma unroll
      for (int q = 0; q < V; ++q) {
        if (((dim >> q) & 1u) && sx[q] != T(0)) e[q] = fma1(cs[q], sx[q], e[q]);
        if (INC && ((mnm >> q) & 1u) && si[q] != T(0)) ei[q] = ei[q] + si[q];
      }
    }
    if (KIND == MK_GOLD && any_ade) {  // ade_update_fixed's gold update on the threads' own state
      const AdeCoef<T> &a = b.gold;
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const T Q = gs[0][q] + fma1(ku, cu[q], sx[q]), S = gs[1][q];
        const T g1r = gs[2][q], g1i = gs[3][q], g2r = gs[4][q], g2i = gs[5][q];
        const T p1r = g1r + lin2(a.dr[0], g1r, -a.di[0], g1i), p1i = g1i + lin2(a.di[0], g1r, a.dr[0], g1i);
        const T p2r = g2r + lin2(a.dr[1], g2r, -a.di[1], g2i), p2i = g2i + lin2(a.di[1], g2r, a.dr[1], g2i);
        const T nre = (fma1(a.ha, S, Q) + p1r) + p2r, nim = p1i + p2i;
        const T ne = lin2(nre, a.wr, -nim, a.wi);
        gs[0][q] = fma1(-a.hb, ne, Q);
        gs[1][q] = S + lin2(a.hb, ne, -a.dha, S);
        gs[2][q] = fma1(a.gcr[0], ne, p1r);
        gs[3][q] = fma1(a.gci[0], ne, p1i);
        gs[4][q] = fma1(a.gcr[1], ne, p2r);
        gs[5][q] = fma1(a.gci[1], ne, p2i);
        e[q] = (adem >> q) & 1u ? ne : e[q];
      }
    } else if (KIND == -1 && any_ade) {
#pragma unroll
      for (int q = 0; q < V; ++q) {
        inc_s[c00 + q] = fma1(ku, cu[q], sx[q]);
        e_s[c00 + q] = e[q];
      }
#pragma unroll 1
      for (int q = 0; q < V; ++q) {
        if (!((adem >> q) & 1u)) continue;
        int ai = ade[0];
#pragma unroll
        for (int u = 1; u < V; ++u) ai = u == q ? ade[u] : ai;
        const int c = c00 + q;
        e_s[c] = ade_update_fixed<T, -1, 1>(st, W, c, 0, p.ac[ai], p.ac + ai, inc_s[c], e_s[c]);
      }
#pragma unroll
      for (int q = 0; q < V; ++q) e[q] = e_s[c00 + q];
    }
    // ---- H half ----
    if (lane == 0) {
      es[w][0] = e[0];
      es[w][1] = ei[0];
    }
    __syncthreads();
    T er = __shfl_down_sync(0xffffffffu, e[0], 1);
    T eir = INC ? __shfl_down_sync(0xffffffffu, ei[0], 1) : T(0);
    if (lane == 31 && w < kLineWarps - 1) {
      er = es[w + 1][0];
      if (INC) eir = es[w + 1][1];
    }
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const unsigned bit = 1u << q;
      h[q] = next(bit, h[q], (q < V - 1 ? e[q + 1] : er) - e[q], ku, mnm, c0[2][q], c0[3][q]);
      if (INC) {
        const T r = q < V - 1 ? ei[q + 1] : eir;
        hv[q] = next(bit, hv[q], r - ei[q], ku, mnm, c1[2][q], c1[3][q]);
        if (any_tf && bd > 0 && j0 + q == bd - 1) h[q] = fma1(-ku, r, h[q]);
      }
    }
    if (lane == 31) {
      hs[w][0] = h[V - 1];
      hs[w][1] = hv[V - 1];
    }
    __syncthreads();
    // ---- samples ----
    if (nrec > 0 && smp) {
      if (nrec <= kLineRecords) {
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (smp & (1u << q)) {
            T *const r = rec + ((s * kLineRecords) + place[c00 + q]) * 4;
            r[0] = e[q];
            r[1] = h[q];
            r[2] = ei[q];
            r[3] = hv[q];
          }
      } else {
        for (int q = 0; q < V; ++q) {
          if (!((smp >> q) & 1u)) continue;
          T v[4] = {e[0], h[0], ei[0], hv[0]};
#pragma unroll
          for (int u = 1; u < V; ++u)
            if (u == q) {
              v[0] = e[u];
              v[1] = h[u];
              v[2] = ei[u];
              v[3] = hv[u];
            }
          line_sample(p, b, j0 + q, s, v, INC);
        }
      }
    }
  }

  // ---- the staged samples, a thread per step ----
  if (nrec > 0 && nrec <= kLineRecords) {
    __syncthreads();
    for (int m = 0; m < p.nmon + p.nprobe; ++m) {
      const int l = m < p.nmon ? p.mon[m].lo[1] : p.probe[m - p.nmon].cell[1];
      const int u = m < p.nmon ? p.mon[m].hi[1] : l;
      for (int j = max(l, own0); j <= min(u, own1 - 1); ++j) {
        const int k = place[j - own0 + b.ks];
        for (int s = threadIdx.x; s < b.ks; s += NT) {
          const T *const r = rec + ((s * kLineRecords) + k) * 4;
          if (m < p.nmon) {
            const Monitor &mo = p.mon[m];
            for (int c = 0; c < mo.ncomp; ++c) {
              const int f = line_field(mo.comps[c], INC);
              b.stage[(long long)(b.s0 + s) * b.stage_row + mo.base + (long long)c * mo.ncell + (j - l)] = f < 0 ? T(0) : r[f];
            }
          } else {
            const Probe &pr = p.probe[m - p.nmon];
            const int n = p.n_first + b.s0 + s;
            if (n < pr.n_first || n > pr.n_last || n - pr.n_first >= pr.cap) continue;
            for (int c = 0; c < pr.ncomp; ++c) {
              const int f = line_field(pr.comps[c], INC);
              pr.buf[(long long)(n - pr.n_first) * pr.ncomp + c] = f < 0 ? 0.0 : (double)r[f];
            }
          }
        }
      }
    }
  }

  // ---- the owned cells to the other set: the slab's own arrays and the line,
  // whose slab cells keep what they held but for the one beside the main range
#pragma unroll
  for (int q = 0; q < V; ++q) {
    if (!((owm >> q) & 1u)) continue;
    const int j = j0 + q;
    auto put = [&](int l, T ev, T hw, const T *ex, const T *hz, T *exo, T *hzo) {
      const bool low = j < lo, high = j >= hi;
      const bool edge = (low && j == lo - 1) || (high && j == hi);
      const bool line = !low && !high;
      exo[j] = line || edge ? ev : ex[j];
      hzo[j] = line || edge ? hw : hz[j];
      if (!line) {
        const int side = low ? 0 : 1, r = low ? j + 1 : j - hi + 1;
        b.pexo[l][side][r] = ev;
        b.phzo[l][side][r] = hw;
        // the conducting row beyond the slab's last cell
        if (j == 0 || j == p.N - 1) {
          const int z = low ? 0 : r + 1;
          b.pexo[l][side][z] = p.pex[l][side][z];
          b.phzo[l][side][z] = p.phz[l][side][z];
        }
      }
      // the slabs' copies of the main cells beside them
      if (p.slab_on[0] && j == lo) {
        b.pexo[l][0][lo + 1] = ev;
        b.phzo[l][0][lo + 1] = hw;
      }
      if (p.slab_on[1] && j == hi - 1) {
        b.pexo[l][1][0] = ev;
        b.phzo[l][1][0] = hw;
      }
    };
    put(0, e[q], h[q], p.ex, p.hz, b.exo, b.hzo);
    if (INC) put(1, ei[q], hv[q], p.exi, p.hzi, b.exio, b.hzio);
    if (KIND != MK_NONE && ((adem >> q) & 1u)) {
      if (KIND == MK_GOLD) {
#pragma unroll
        for (int f = 0; f < 6; ++f) b.ade_out[(long long)(f * 3) * p.ade_stride + slot[q]] = gs[f][q];
      } else {
        for (int f = 0; f < p.ade_nf; ++f) b.ade_out[(long long)(f * 3) * p.ade_stride + slot[q]] = st[f * W + c00 + q];
      }
    }
  }
}

template <typename T, int V, bool INC, int KIND>
int launch_v(const LineParams<T> &p, const LineBlock<T> &b, cudaStream_t s) {
  auto kern = line1d_block<T, V, INC, KIND>;
  static std::atomic<unsigned long long> done{0};
  if (!smem_limit(kern, 96 * 1024, done)) return -1;
  const size_t sm = (size_t)(kLineSteps * (kMaxSrc + kLineRecords * 4) + (KIND == -1 ? (2 + p.ade_nf) * 32 * kLineWarps * V : 0)) * sizeof(T);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + b.own - 1) / b.own);
  cfg.blockDim = dim3(32 * kLineWarps);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p, b) == cudaSuccess ? 1 : -1;
}

template <typename T, int V, bool INC>
int launch_i(const LineParams<T> &p, const LineBlock<T> &b, cudaStream_t s) {
  if (p.nade == 0) return launch_v<T, V, INC, MK_NONE>(p, b, s);
  if (b.one_gold) return launch_v<T, V, INC, MK_GOLD>(p, b, s);
  return launch_v<T, V, INC, -1>(p, b, s);
}

}  // namespace

template <typename T>
int launch_line1d_block(const LineParams<T> &p, const LineBlock<T> &b, int V, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const bool inc = p.exi != nullptr;
  if (V == 1) return inc ? launch_i<T, 1, true>(p, b, s) : launch_i<T, 1, false>(p, b, s);
  return inc ? launch_i<T, 2, true>(p, b, s) : launch_i<T, 2, false>(p, b, s);
}
template int launch_line1d_block<float>(const LineParams<float> &, const LineBlock<float> &, int, void *);
template int launch_line1d_block<double>(const LineParams<double> &, const LineBlock<double> &, int, void *);

}  // namespace fdtd
