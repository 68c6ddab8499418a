// k3b.cu -- the 3D block-step kernel (FP32): two steps of the whole grid per
// launch (updateD, updateH and the split PML of
// 3D/.../include/myfdtd_func.f90:19-64, 3D/BERpmly_mod.f90:117-195, twice).
//
// A block owns a tile of the grid and marches it along z.  A warp holds a row
// of 64 cells, two per lane.  When plane k arrives it computes E of the first
// new step there, H of that step on plane k-1, E of the second step on plane
// k-2 and H of the second step on plane k-3, so a cell's fields are read once
// and written once in two steps.  The tile is widened by what the two steps
// reach: a cell pair on each side in x, a row below and two above, and planes
// at both ends; the widened cells belong to the neighbouring tiles, which
// compute the same values themselves.  Tiles read one set of buffers and store
// to the other (a ping-pong pair), so they are independent of one another.
//
// The cell left or right of a lane's pair comes from the next lane by a
// shuffle, the row below or above through shared memory; every stage reads
// only rows that the round before stored, so a round has one barrier.  Planes
// are loaded a round ahead into registers.
//
// A warp whose row holds only main cells of the one most common material takes
// the plain update; others choose per cell: the split update in the PML shell,
// other materials, dispersive cells, sources.  The split parts of the first
// step wait in shared memory for the second, dispersive state in a buffer of
// its own (ade_mid: tiles that share a cell store the same values there; the
// second step's state goes only from the owner to the other state set).
// Rows with samples go to a buffer after the first step, from which the gather
// kernel takes that step's samples.
//
// A chunk of four planes whose rows are plain runs with its planes' registers in
// fixed places, and so does one of rows of x and y shell cells between the z
// shells, whose coefficients are the same on every plane; every other plane
// takes a general round, which moves its registers on.  Tiles with dispersive
// cells run in a kernel of their own, so that its registers do not spill the
// others'.
//
// What bounds it: the latency of its loads and of the shared-memory exchange
// with 16 warps on an SM (issue 35% busy, DRAM 40%); without any loads or stores
// a step of 480 x 480 x 384 plain cells takes 260 us, with them 443 (the memory
// traffic alone 311).  16 warps of 128 registers: 20 of 96 spill (605 us), two
// blocks of 10 waste more on the halo (562); planes prefetched to L2 two rounds
// before their loads, not at all: 582 us; streaming stores, not: 462.  Per step:
// 512^3 with a gold sphere and 16 PML cells 1160 us against 1500 of the fused
// kernel, the 256 x 256 x 384 column 212 against 285 of the split ones.
#include <cuda_runtime.h>
#include <type_traits>

#include "fdtd_internal.h"
#include "kcommon.cuh"

namespace fdtd {

namespace {

typedef unsigned long long f2;  // two floats, the lower cell in the low half

__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void un(f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ float lo2(f2 v) { float a, b; un(v, a, b); return a; }
__device__ __forceinline__ float hi2(f2 v) { float a, b; un(v, a, b); return b; }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// the pair one cell to the left or to the right (the warp's ends: any value)
__device__ __forceinline__ f2 left2(f2 v) {
  float a, b;
  un(v, a, b);
  return pk(__shfl_up_sync(0xffffffffu, b, 1), a);
}
__device__ __forceinline__ f2 right2(f2 v) {
  float a, b;
  un(v, a, b);
  return pk(b, __shfl_down_sync(0xffffffffu, a, 1));
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// the halves of a where the masks say so, else of b
__device__ __forceinline__ f2 sel2(bool lo, bool hi, f2 a, f2 b) {
  float a0, a1, b0, b1;
  un(a, a0, a1);
  un(b, b0, b1);
  return pk(lo ? a0 : b0, hi ? a1 : b1);
}
__device__ __forceinline__ f2 ldg2(const float *a) { return __ldg(reinterpret_cast<const f2 *>(a)); }
// at a 32-bit byte offset from a base that is the same in all threads (one
// register of address per thread)
__device__ __forceinline__ f2 ldg2(const float *base, unsigned at) {
  return __ldg(reinterpret_cast<const f2 *>(reinterpret_cast<const char *>(base) + at));
}
// (streaming stores: nothing reads the new fields before the next launch)
__device__ __forceinline__ void stg2(float *base, unsigned at, f2 v) {
  __stcs(reinterpret_cast<f2 *>(reinterpret_cast<char *>(base) + at), v);
}

// start a line on its way to L2
__device__ __forceinline__ void prefetch(const float *base, unsigned at) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(base) + at));
}

// ade_update_fixed's gold update of one component with the state in registers
// (f: Q S g1r g1i g2r g2i)
__device__ __forceinline__ float gold_update(float (&f)[6], const AdeCoef<float> &a, float inc) {
  const float Q = f[0] + inc, S = f[1];
  const float p1r = f[2] + lin2(a.dr[0], f[2], -a.di[0], f[3]), p2r = f[4] + lin2(a.dr[1], f[4], -a.di[1], f[5]);
  const float p1i = f[3] + lin2(a.di[0], f[2], a.dr[0], f[3]), p2i = f[5] + lin2(a.di[1], f[4], a.dr[1], f[5]);
  const float nre = (fma1(a.ha, S, Q) + p1r) + p2r, nim = p1i + p2i;
  const float e = lin2(nre, a.wr, -nim, a.wi);
  f[0] = fma1(-a.hb, e, Q);
  f[1] = S + lin2(a.hb, e, -a.dha, S);
  f[2] = fma1(a.gcr[0], e, p1r);
  f[3] = fma1(a.gci[0], e, p1i);
  f[4] = fma1(a.gcr[1], e, p2r);
  f[5] = fma1(a.gci[1], e, p2i);
  return e;
}

// E of a pair with gold cells (bits 0 and 1 of `which`): their states' loads go
// out together.  bits 2 and 3: the cell's new state is stored
__device__ __forceinline__ void gold_pair(const StepParams<float> &p, const float *from, float *to, const int *slots, int which,
                                          f2 (&e)[3], f2 i0, f2 i1, f2 i2) {
  const f2 inc[3] = {i0, i1, i2};
  int slot[2] = {0, 0};
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (which >> q & 1) slot[q] = __ldg(slots + q);
  float f[3][2][6];
#pragma unroll
  for (int u = 0; u < 3; ++u)
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int w = 0; w < 6; ++w) f[u][q][w] = which >> q & 1 ? from[(long long)(3 * w + u) * p.ade_stride + slot[q]] : 0.0f;
#pragma unroll
  for (int u = 0; u < 3; ++u) {
    float x[2], in[2];
    un(e[u], x[0], x[1]);
    un(inc[u], in[0], in[1]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const float r = gold_update(f[u][q], p.acp[0], in[q]);
      if (!(which >> q & 1)) continue;
      x[q] = r;
      if (which >> (2 + q) & 1)
#pragma unroll
        for (int w = 0; w < 6; ++w) to[(long long)(3 * w + u) * p.ade_stride + slot[q]] = f[u][q][w];
    }
    e[u] = pk(x[0], x[1]);
  }
}

// E of a dispersive cell, its state from `from`, to `to` if not null; every load
// of the state is issued before the first of it is used
__device__ __noinline__ float3 ade_cell(const StepParams<float> &p, const float *from, float *to, int slot, int id, float3 inc,
                                        float3 e) {
  const AdeCoef<float> *am = p.ac + (id - kAdeId);
  const int nf = ade_fields(am->kind, am->npoles, am->nl, 0);
  float st[3][kAdeFields + 2];  // field f of component u at f + u
  const long long fs = 3ll * p.ade_stride;
#pragma unroll
  for (int f = 0; f < kAdeFields; ++f)
    if (f < nf) {
#pragma unroll
      for (int u = 0; u < 3; ++u) st[u][f + u] = from[f * fs + (long long)u * p.ade_stride + slot];
    }
  e.x = ade_update_fixed<float, -1, 1>(st[0], 1, 0, 0, *am, am, inc.x, e.x);
  e.y = ade_update_fixed<float, -1, 1>(st[1], 1, 0, 1, *am, am, inc.y, e.y);
  e.z = ade_update_fixed<float, -1, 1>(st[2], 1, 0, 2, *am, am, inc.z, e.z);
  if (to) {
#pragma unroll
    for (int f = 0; f < kAdeFields; ++f)
      if (f < nf) {
#pragma unroll
        for (int u = 0; u < 3; ++u) to[f * fs + (long long)u * p.ade_stride + slot] = st[u][f + u];
      }
  }
  return e;
}

enum { B3_SRC = ROW_SRC, B3_SMP = ROW_SAMPLE, B3_MIX = 4, B3_DEAD = 8, B3_GEN = 16, B3_GENZ = 32, B3_ADE = 64 };  // flags of a row

// NS: steps of the launch (1 or 2); NW: warps, rows of the widened tile
template <int NS, int NW, bool ADE>
__global__ void __launch_bounds__(32 * NW, 1) step3d_block(const __grid_constant__ StepParams<float> p,
                                                           const __grid_constant__ Block3 b) {
  extern __shared__ __align__(16) f2 sm3[];
  constexpr int NT = 32 * NW;
  // rows of this and of the last round: [parity][E1x E1z H1x H1z E2x E2z][thread]
  f2 *const xr = sm3 + threadIdx.x;
  // split parts of the first step: [parity][6][thread]
  f2 *const part = sm3 + 12 * NT + threadIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  f2 *const xb = xr + (w > 0 ? -32 : 0), *const xa = xr + (w < NW - 1 ? 32 : 0);  // of the row below, above
  int t = __ldg(b.order + (ADE ? 0 : b.nade) + blockIdx.x);
  const int tx = t % b.ntx;
  t /= b.ntx;
  const int ty = t % b.nty, tz = t / b.nty;
  const int i0 = tx * b.ox - 2 + 2 * lane, j0 = ty * b.oy - 1 + w;
  const int za = tz * b.oz, zb = min(za + b.oz, p.nz);
  const bool split = p.pml_mode == 2;
  // this thread's column of cell pairs: its place in the grid (wrapped on a
  // periodic axis), or no cells of it
  int i = i0, j = j0, jb = j0 - 1;
  if (p.per[0]) i = ((i0 % p.nx) + p.nx) % p.nx;
  if (p.per[1]) {
    j = ((j0 % p.ny) + p.ny) % p.ny;
    jb = (((j0 - 1) % p.ny) + p.ny) % p.ny;
  }
  const bool live_x = i >= 0 && i < p.nx, live = live_x && j >= 0 && j < p.ny;
  const bool live_b = live_x && jb >= 0 && jb < p.ny;
  const bool own = live && lane >= 1 && 2 * lane < 2 + b.ox && w >= 1 && w <= b.oy && i0 < p.nx && j0 < p.ny;
  const unsigned ro = live ? 4u * (unsigned)(j * p.nx + i) : 0u, rb = live_b ? 4u * (unsigned)(jb * p.nx + i) : 0u;  // bytes
  const unsigned plane = 4u * (unsigned)(p.nx * p.ny);  // bytes; a field has fewer than 2^32
  // shell and main cells of the pair (without the plane's part)
  const bool iny = split && (j < p.slo[1] || j > p.shi[1]);
  bool inx[2], mxy[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    inx[q] = split && (i + q < p.slo[0] || i + q > p.shi[0]);
    mxy[q] = live && i + q >= p.mlo[0] && i + q <= p.mhi[0] && j >= p.mlo[1] && j <= p.mhi[1];
  }
  const bool anyx = inx[0] || inx[1];
  // a row that is not all main cells, or at the grid's end
  const bool gen_xy = __any_sync(0xffffffffu, !(mxy[0] && mxy[1] && !inx[0] && !inx[1] && !iny && live_b));
  const f2 ku2 = pk(p.ku, p.ku), ca2 = pk(p.ca0, p.ca0);
  // A row with cells of the x and y shells, on the planes between the z shells,
  // has the same coefficients on every plane: in shared memory, per thread, the x
  // and y profiles (E 1 2, H 1 2) and the factors of the plain update
  f2 *const co = sm3 + 24 * NT + threadIdx.x;
  enum { CX = 0, CY = 4, CZ = 8, CM = 12 };
  const bool sh0 = inx[0] || iny, sh1 = inx[1] || iny;
  const bool has_dead = __any_sync(0xffffffffu, !live);
  const bool mid_ok = __all_sync(0xffffffffu, !live || ((sh0 || mxy[0]) && (sh1 || mxy[1])));
  const bool wx = __any_sync(0xffffffffu, anyx);
  if (split) {
    auto two = [](float x) { return pk(x, x); };
    const int ic = live ? i : 0, jc = live ? j : 0, kc = p.slo[2];
    co[(CX + 0) * NT] = ldg2(p.cf1[0] + ic);
    co[(CX + 1) * NT] = ldg2(p.cf2[0] + ic);
    co[(CX + 2) * NT] = ldg2(p.cg1[0] + ic);
    co[(CX + 3) * NT] = ldg2(p.cg2[0] + ic);
    co[(CY + 0) * NT] = two(__ldg(p.cf1[1] + jc));
    co[(CY + 1) * NT] = two(__ldg(p.cf2[1] + jc));
    co[(CY + 2) * NT] = two(__ldg(p.cg1[1] + jc));
    co[(CY + 3) * NT] = two(__ldg(p.cg2[1] + jc));
    co[(CZ + 0) * NT] = two(__ldg(p.cf1[2] + kc));
    co[(CZ + 1) * NT] = two(__ldg(p.cf2[2] + kc));
    co[(CZ + 2) * NT] = two(__ldg(p.cg1[2] + kc));
    co[(CZ + 3) * NT] = two(__ldg(p.cg2[2] + kc));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const f2 m = h ? ku2 : ca2;
      co[(CM + 3 * h + 0) * NT] = sel2(sh0, sh1, co[(CY + 1 + 2 * h) * NT], m);
      co[(CM + 3 * h + 1) * NT] = sel2(sh0, sh1, co[(CZ + 1 + 2 * h) * NT], m);
      co[(CM + 3 * h + 2) * NT] = sel2(sh0, sh1, co[(CX + 1 + 2 * h) * NT], m);
    }
  } else {
#pragma unroll
    for (int u = 0; u < 6; ++u) co[(CM + u) * NT] = u < 3 ? ca2 : ku2;
  }

  // (a tile reaches two planes past either end, and a periodic axis has as many)
  auto wrap_z = [&](int k) { return !p.per[2] ? k : k < 0 ? k + p.nz : k >= p.nz ? k - p.nz : k; };
  auto flags_of = [&](int k) -> unsigned {
    const int kw = wrap_z(k);
    if (kw < 0 || kw >= p.nz || j < 0 || j >= p.ny) return B3_DEAD | B3_GEN;
    return __ldg(b.flags + ((long long)kw * p.ny + j) * b.ntx + tx);
  };
  pdl_wait();
  pdl_release();
  // the sources' values of the launch's steps, [step][source]: read from the table
  // per cell and component they made a line of sources along z, one row of one
  // column of tiles, hold up a launch (256^3: 760 us a step, 260 without it)
  __shared__ float srcv[2 * kMaxSrc];
  if (p.nsrc > 0) {
    const int n = step_n(p);
    if (threadIdx.x < NS * p.nsrc) srcv[threadIdx.x] = float(p.srcval_tab[(long long)(n - 1) * p.nsrc + threadIdx.x]);
    __syncthreads();
  }
  // their sum on component comp of a cell in step s
  auto src_at = [&](int s, int comp, int x, int y, int z) {
    float v = 0.0f;
    for (int q = 0; q < p.nsrc; ++q) {
      const Source &sr = p.src[q];
      if (sr.comp == comp && x >= sr.lo[0] && x <= sr.hi[0] && y >= sr.lo[1] && y <= sr.hi[1] && z >= sr.lo[2] && z <= sr.hi[2])
        v += srcv[s * p.nsrc + q];
    }
    return v;
  };

  // plane k's fields live in one of four slots from its load to its store
  f2 E[4][3] = {}, H[4][3] = {}, nxd = 0, nzd = 0;  // nxd, nzd: Hx, Hz of the row below on the next plane
  auto load = [&](int k, f2(&e)[3], f2(&h)[3]) {
    const int kw = wrap_z(k);
    const bool in = kw >= 0 && kw < p.nz;
    const unsigned c = (unsigned)kw * plane + ro, cb = (unsigned)kw * plane + rb;
    if (in && !gen_xy) {
      e[0] = ldg2(p.ex, c);
      e[1] = ldg2(p.ey, c);
      e[2] = ldg2(p.ez, c);
      h[0] = ldg2(p.hx, c);
      h[1] = ldg2(p.hy, c);
      h[2] = ldg2(p.hz, c);
      nxd = ldg2(p.hx, cb);
      nzd = ldg2(p.hz, cb);
    } else {
      e[0] = e[1] = e[2] = h[0] = h[1] = h[2] = nxd = nzd = 0;
      if (in && live) {
        e[0] = ldg2(p.ex, c);
        e[1] = ldg2(p.ey, c);
        e[2] = ldg2(p.ez, c);
        h[0] = ldg2(p.hx, c);
        h[1] = ldg2(p.hy, c);
        h[2] = ldg2(p.hz, c);
      }
      if (in && live_b) {
        nxd = ldg2(p.hx, cb);
        nzd = ldg2(p.hz, cb);
      }
    }
  };

  // Planes are on their way to L2 kAhead rounds before the registers ask for
  // them: a lane for each of the six fields and each of the three 128-byte lines
  // that a row of 256 bytes can touch.
  constexpr int kAhead = 2;
  const int pf = lane / 3, pl = pf < 6 ? lane % 3 * 16 - (lane % 3 == 2) : 0;  // (pairs 0, 16 and 31 of the row)
  const float *const pbase = pf == 0 ? p.ex : pf == 1 ? p.ey : pf == 2 ? p.ez : pf == 3 ? p.hx : pf == 4 ? p.hy : p.hz;
  const bool line = __shfl_sync(0xffffffffu, live, pl) && pf < 6;
  const unsigned pro = __shfl_sync(0xffffffffu, ro, pl);
  auto ahead = [&](int k) {
    const int kw = wrap_z(k);
    if (line && kw >= 0 && kw < p.nz && k <= zb + 1) prefetch(pbase, (unsigned)kw * plane + pro);
  };

  // The split parts of a pair on plane k, the three from o on, as the launch finds them
  auto load_parts = [&](f2(&st)[3], int k, int o) {
    const int kw = wrap_z(k);
    st[0] = st[1] = st[2] = 0;
    if (!split || !live || kw < 0 || kw >= p.nz) return;
    const bool inz = kw < p.slo[2] || kw > p.shi[2];
    const unsigned c = (unsigned)kw * plane + ro;
    if (iny || inz) st[0] = ldg2(p.sp[o], c);
    if (inz || anyx) st[1] = ldg2(p.sp[o + 1], c);
    if (anyx || iny) st[2] = ldg2(p.sp[o + 2], c);
  };

  // The update of three components v of a pair on plane kw: v += m (a + c) in
  // main cells (m: E Ku/eps, H Ku), the split update in shell cells, whose stored
  // part takes the curl term a with the profile of axis y, z, x and the rest of
  // the component c with that of z, x, y.  The roundings are those of edge_e3 and
  // edge_h3.  st: the stored parts before; s: step of the launch; o: the first of
  // the three parts.
  auto general = [&](f2(&v)[3], const f2(&a)[3], const f2(&c)[3], f2 m, int kw, int kp, f2(&st)[3], int s, int o,
                     const float *const *t1, const float *const *t2) {
    const bool inz = split && (kw < p.slo[2] || kw > p.shi[2]), mz = kw >= p.mlo[2] && kw <= p.mhi[2];
    const bool sh0 = inx[0] || iny || inz, sh1 = inx[1] || iny || inz;
    const bool on0 = live && (sh0 || (mxy[0] && mz)), on1 = live && (sh1 || (mxy[1] && mz));
    f2 f1[3] = {}, f2_[3] = {};
    if (sh0 || sh1) {
      f1[0] = ldg2(t1[0] + (live ? i : 0));
      f2_[0] = ldg2(t2[0] + (live ? i : 0));
      const float y1 = __ldg(t1[1] + (live ? j : 0)), y2 = __ldg(t2[1] + (live ? j : 0)), z1 = __ldg(t1[2] + kw),
                  z2 = __ldg(t2[2] + kw);
      f1[1] = pk(y1, y1);
      f2_[1] = pk(y2, y2);
      f1[2] = pk(z1, z1);
      f2_[2] = pk(z2, z2);
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const int A = u == 0 ? 1 : u == 1 ? 2 : 0, B = u == 0 ? 2 : u == 1 ? 0 : 1;
      const bool two0 = u == 0 ? iny || inz : u == 1 ? inz || inx[0] : inx[0] || iny;
      const bool two1 = u == 0 ? iny || inz : u == 1 ? inz || inx[1] : inx[1] || iny;
      f2 r = fma2(sel2(sh0, sh1, f2_[A], m), add2(a[u], c[u]), v[u]);
      if (two0 || two1) {
        const f2 d = sub2(v[u], st[u]), np = fma2(f2_[A], a[u], mul2(f1[A], st[u]));
        const f2 nb = B == 0 ? fma2(f1[B], d, mul2(f2_[B], c[u])) : fma2(f2_[B], c[u], mul2(f1[B], d));
        r = sel2(two0, two1, add2(np, nb), r);
        if (s + 1 < NS) part[((kp & 1) * 6 + o + u) * NT] = np;
        else if (own && kp >= za && kp < zb) stg2(b.spo[o + u], (unsigned)kw * plane + ro, np);
      }
      v[u] = sel2(on0, on1, r, v[u]);
    }
  };
  // the same for such a row: h 0 E, 1 H
  auto general_xy = [&](f2(&v)[3], const f2(&a)[3], const f2(&c)[3], int k, f2(&st)[3], int s, int h) {
    const f2 x1 = co[(CX + 2 * h) * NT], x2 = co[(CX + 2 * h + 1) * NT];
    const f2 y1 = co[(CY + 2 * h) * NT], y2 = co[(CY + 2 * h + 1) * NT];
    const f2 z1 = co[(CZ + 2 * h) * NT], z2 = co[(CZ + 2 * h + 1) * NT];
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const f2 A1 = u == 0 ? y1 : u == 1 ? z1 : x1, A2 = u == 0 ? y2 : u == 1 ? z2 : x2;
      const f2 B1 = u == 0 ? z1 : u == 1 ? x1 : y1, B2 = u == 0 ? z2 : u == 1 ? x2 : y2;
      f2 r = fma2(co[(CM + 3 * h + u) * NT], add2(a[u], c[u]), v[u]);
      if (u == 0 ? iny : u == 1 ? wx : wx || iny) {
        const f2 d = sub2(v[u], st[u]), np = fma2(A2, a[u], mul2(A1, st[u]));
        const f2 nb = u == 1 ? fma2(B1, d, mul2(B2, c[u])) : fma2(B2, c[u], mul2(B1, d));
        const bool two0 = u == 0 ? iny : u == 1 ? inx[0] : sh0, two1 = u == 0 ? iny : u == 1 ? inx[1] : sh1;
        r = sel2(two0, two1, add2(np, nb), r);
        if (two0 || two1) {
          if (s + 1 < NS) part[((k & 1) * 6 + 3 * h + u) * NT] = np;
          else if (own) stg2(b.spo[3 * h + u], (unsigned)wrap_z(k) * plane + ro, np);
        }
      }
      v[u] = r;
    }
    if (has_dead && !live) v[0] = v[1] = v[2] = 0;
  };
  // the second step's parts, left by the first
  auto kept_parts = [&](f2(&st)[3], int kp, int o) {
#pragma unroll
    for (int u = 0; u < 3; ++u) st[u] = part[((kp & 1) * 6 + o + u) * NT];
  };

  // the two curl terms of each E component: own H, Hx and Hy of the plane below,
  // Hx and Hz of the row below; and of each H component: own E, Ex and Ey of the
  // plane above, Ex and Ez of the row above
  auto curl_h = [&](f2(&a)[3], f2(&c)[3], const f2(&h)[3], f2 hxb, f2 hyb, f2 hxd, f2 hzd) {
    a[0] = sub2(h[2], hzd);
    a[1] = sub2(h[0], hxb);
    a[2] = sub2(h[1], left2(h[1]));
    c[0] = sub2(hyb, h[1]);
    c[1] = sub2(left2(h[2]), h[2]);
    c[2] = sub2(hxd, h[0]);
  };
  auto curl_e = [&](f2(&a)[3], f2(&c)[3], const f2(&e)[3], f2 exa, f2 eya, f2 exu, f2 ezu) {
    a[0] = sub2(e[2], ezu);
    a[1] = sub2(e[0], exa);
    a[2] = sub2(e[1], right2(e[1]));
    c[0] = sub2(eya, e[1]);
    c[1] = sub2(right2(e[2]), e[2]);
    c[2] = sub2(exu, e[0]);
  };
  auto plain = [&](f2(&v)[3], const f2(&a)[3], const f2(&c)[3], f2 m) {
#pragma unroll
    for (int u = 0; u < 3; ++u) v[u] = fma2(m, add2(a[u], c[u]), v[u]);
  };

  // E of step s on plane k; fl: the row's flags
  auto e_update = [&](f2(&e)[3], const f2(&a)[3], const f2(&c)[3], int k, unsigned fl, f2(&st)[3], int s) {
    if (!(fl & ~B3_SMP)) {
      plain(e, a, c, ca2);
      return;
    }
    if (fl & B3_DEAD) return;
    const int kw = wrap_z(k);
    f2 m = ca2;
    int id[2] = {p.id0, p.id0};
    bool ade[2] = {false, false};
    const bool mz = kw >= p.mlo[2] && kw <= p.mhi[2] && !(split && (kw < p.slo[2] || kw > p.shi[2]));
    const unsigned cell = ((unsigned)kw * plane + ro) >> 2;
    if (fl & B3_MIX && live) {
      const uchar2 d = __ldg(reinterpret_cast<const uchar2 *>(p.mat + cell));
      id[0] = d.x;
      id[1] = d.y;
      float mv[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        mv[q] = id[q] == p.id0 ? p.ca0 : __ldg(p.mca + id[q]);
        if (ADE) ade[q] = id[q] >= kAdeId && mxy[q] && mz && !inx[q] && !iny;
      }
      m = pk(mv[0], mv[1]);
    }
    const f2 old[3] = {e[0], e[1], e[2]};
    if (fl & B3_GEN) general(e, a, c, m, kw, k, st, s, 0, p.cf1, p.cf2);
    else plain(e, a, c, m);
    const bool src = fl & B3_SRC;
    if (!src && !ade[0] && !ade[1]) return;
    if (ADE && b.one_gold && !src) {  // both cells' loads together, the state in registers
      const long long at = ((long long)(kw - b.alo[2]) * b.an[1] + (j - b.alo[1])) * b.an[0] + (i - b.alo[0]);
      const bool keep = s + 1 < NS || (own && k >= za && k < zb);
      gold_pair(p, s == 0 ? p.ade_state : b.ade_mid, s + 1 < NS ? b.ade_mid : b.ade_out, b.slot + at,
                (ade[0] ? 1 : 0) | (ade[1] ? 2 : 0) | (keep && (s + 1 == NS || lane > 0) ? 4 : 0) | (keep ? 8 : 0), e,
                mul2(ku2, add2(a[0], c[0])), mul2(ku2, add2(a[1], c[1])), mul2(ku2, add2(a[2], c[2])));
      return;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (!mxy[q] || !mz || inx[q] || iny || !(src || ade[q])) continue;
      float x[3], inc[3];
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        const float sv = src ? src_at(s, u, i + q, j, kw) : 0.0f;
        x[u] = q ? hi2(e[u]) : lo2(e[u]);
        const f2 sum = add2(a[u], c[u]);
        inc[u] = fma1(p.ku, q ? hi2(sum) : lo2(sum), sv);
        if (sv != 0.0f) x[u] = fma1(__ldg(p.mcs + id[q]), sv, x[u]);
      }
      if (ADE && ade[q]) {
        const int slot = __ldg(b.slot + ((long long)(kw - b.alo[2]) * b.an[1] + (j - b.alo[1])) * b.an[0] + (i + q - b.alo[0]));
        // the first step's state of a cell that holds: all but the halo's outermost
        const bool keep = s + 1 < NS ? lane > 0 || q > 0 : own && k >= za && k < zb;
        float ov[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) ov[u] = q ? hi2(old[u]) : lo2(old[u]);
        const float3 r = ade_cell(p, s == 0 ? p.ade_state : b.ade_mid, !keep ? nullptr : s + 1 < NS ? b.ade_mid : b.ade_out,
                                  slot, id[q], make_float3(inc[0], inc[1], inc[2]), make_float3(ov[0], ov[1], ov[2]));
        x[0] = r.x;
        x[1] = r.y;
        x[2] = r.z;
      }
#pragma unroll
      for (int u = 0; u < 3; ++u) e[u] = q ? pk(lo2(e[u]), x[u]) : pk(x[u], hi2(e[u]));
    }
  };

  auto h_update = [&](f2(&h)[3], const f2(&a)[3], const f2(&c)[3], int k, unsigned fl, f2(&st)[3], int s) {
    if (!(fl & B3_GEN)) {
      plain(h, a, c, ku2);
      return;
    }
    if (fl & B3_DEAD) return;
    general(h, a, c, ku2, wrap_z(k), k, st, s, 3, p.cg1, p.cg2);
  };
  auto store = [&](const f2(&e)[3], const f2(&h)[3], int k) {
    const unsigned c = (unsigned)k * plane + ro;
    if (!own) return;
    stg2(p.exo, c, e[0]);
    stg2(p.eyo, c, e[1]);
    stg2(p.ezo, c, e[2]);
    stg2(p.hxo, c, h[0]);
    stg2(p.hyo, c, h[1]);
    stg2(p.hzo, c, h[2]);
  };
  f2 sE[3], sH[3];  // split parts: E's of the next plane, H's of the one below it
  bool parts = false;
  // a row with samples after the first step, for the gather kernel
  auto keep_first = [&](const f2(&e)[3], const f2(&h)[3], int k) {
    if (!own) return;
    float *const to = b.first + (long long)__ldg(b.seg + ((long long)k * p.ny + j) * b.ntx + tx) * (6 * b.ox) + (2 * lane - 2);
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      *reinterpret_cast<f2 *>(to + u * b.ox) = e[u];
      *reinterpret_cast<f2 *>(to + (3 + u) * b.ox) = h[u];
    }
  };
  // one plane of any kind: the planes k, k-1, k-2, k-3 in slots u0, u3, u2, u1;
  // plane k+1 is loaded into slot u1
  const int k0 = za - (NS - 1), klast = zb + NS - 1, kend = NS == 2 ? zb + 2 : zb;
  auto round = [&](int k, int par, f2(&e0)[3], f2(&e1)[3], f2(&e2)[3], f2(&e3)[3], f2(&h0)[3], f2(&h1)[3], f2(&h2)[3],
                   f2(&h3)[3], unsigned f0, unsigned f1, unsigned f2_, unsigned f3) {
    f2 *const now = xr + par * 6 * NT;
    const f2 *const wb = xb + (par ^ 1) * 6 * NT, *const wa = xa + (par ^ 1) * 6 * NT;
    f2 a[3], c[3], st[3];
    if (NS == 2 && k >= za + 2) {
      curl_h(a, c, h2, h1[0], h1[1], wb[2 * NT], wb[3 * NT]);
      if (f2_ & B3_GEN) kept_parts(st, k - 2, 0);
      e_update(e2, a, c, k - 2, f2_, st, 1);
      now[4 * NT] = e2[0];
      now[5 * NT] = e2[2];
      if (k >= za + 3) {
        curl_e(a, c, e1, e2[0], e2[1], wa[4 * NT], wa[5 * NT]);
        if (f3 & B3_GEN) kept_parts(st, k - 3, 3);
        h_update(h1, a, c, k - 3, f3, st, 1);
        store(e1, h1, k - 3);
      }
    }
    if (k <= klast) {
      curl_h(a, c, h0, h3[0], h3[1], nxd, nzd);
      e_update(e0, a, c, k, f0, sE, 0);
      now[0] = e0[0];
      now[NT] = e0[2];
      if (k < klast) load(k + 1, e1, h1);
      ahead(k + 1 + kAhead);
      if (k > k0) {
        curl_e(a, c, e3, e0[0], e0[1], wa[0], wa[NT]);
        h_update(h3, a, c, k - 1, f1, sH, 0);
        now[2 * NT] = h3[0];
        now[3 * NT] = h3[2];
        if (k - 1 >= za && k - 1 < zb) {
          if (NS == 1) store(e3, h3, k - 1);
          if (NS == 2 && f1 & B3_SMP) keep_first(e3, h3, k - 1);
        }
      }
    }
    load_parts(sE, k + 1, 0);  // for the next round
    load_parts(sH, k, 3);
    __syncthreads();
  };

  for (int u = 1; u <= kAhead; ++u) ahead(k0 + u);
  load(k0 - 1, E[3], H[3]);
  load(k0, E[0], H[0]);
  unsigned cf = lane < 8 ? flags_of(k0 - 3 + lane) : 0u, nf = 0;  // flags of the planes k-3 .. k+4
#pragma unroll 1
  for (int k = k0; k <= kend; k += 4, cf = nf) {
    if (lane < 8) nf = flags_of(k + 1 + lane);
    const bool inside = k >= za + (NS == 2 ? 3 : 1) && k + 3 < klast;
    const bool fast = inside && !__any_sync(0xffffffffu, lane < 7 && cf & ~B3_SMP);
    const bool mid = inside && mid_ok && k + 2 < zb && !__any_sync(0xffffffffu, lane < 7 && cf & ~(B3_SMP | B3_GEN));
    // four planes of plain rows, or of rows with x and y shell cells: the slots fixed
    auto chunk = [&](auto kind) {
      constexpr bool XY = decltype(kind)::value;
      const unsigned smp = __ballot_sync(0xffffffffu, lane < 7 && cf & B3_SMP);  // bit q: plane k-3+q
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        f2 *const now = xr + (u & 1) * 6 * NT;
        const f2 *const wb = xb + (u & 1 ^ 1) * 6 * NT, *const wa = xa + (u & 1 ^ 1) * 6 * NT;
        f2(&e0)[3] = E[u], (&e3)[3] = E[(u + 3) & 3], (&e2)[3] = E[(u + 2) & 3], (&e1)[3] = E[(u + 1) & 3];
        f2(&h0)[3] = H[u], (&h3)[3] = H[(u + 3) & 3], (&h2)[3] = H[(u + 2) & 3], (&h1)[3] = H[(u + 1) & 3];
        f2 a[3], c[3], st[3];
        if constexpr (NS == 2) {
          curl_h(a, c, h2, h1[0], h1[1], wb[2 * NT], wb[3 * NT]);
          if constexpr (XY) {
            kept_parts(st, k + u - 2, 0);
            general_xy(e2, a, c, k + u - 2, st, 1, 0);
          } else {
            plain(e2, a, c, ca2);
          }
          now[4 * NT] = e2[0];
          now[5 * NT] = e2[2];
          curl_e(a, c, e1, e2[0], e2[1], wa[4 * NT], wa[5 * NT]);
          if constexpr (XY) {
            kept_parts(st, k + u - 3, 3);
            general_xy(h1, a, c, k + u - 3, st, 1, 1);
          } else {
            plain(h1, a, c, ku2);
          }
          store(e1, h1, k + u - 3);
        }
        curl_h(a, c, h0, h3[0], h3[1], nxd, nzd);
        if constexpr (XY) general_xy(e0, a, c, k + u, sE, 0, 0);
        else plain(e0, a, c, ca2);
        now[0] = e0[0];
        now[NT] = e0[2];
        load(k + u + 1, e1, h1);
        ahead(k + u + 1 + kAhead);
        curl_e(a, c, e3, e0[0], e0[1], wa[0], wa[NT]);
        if constexpr (XY) general_xy(h3, a, c, k + u - 1, sH, 0, 1);
        else plain(h3, a, c, ku2);
        now[2 * NT] = h3[0];
        now[3 * NT] = h3[2];
        if constexpr (NS == 1) store(e3, h3, k + u - 1);
        else if (smp >> (u + 2) & 1 && k + u - 1 < zb) keep_first(e3, h3, k + u - 1);
        if constexpr (XY) {
          load_parts(sE, k + u + 1, 0);
          load_parts(sH, k + u, 3);
        }
        __syncthreads();
      }
    };
    if (fast) {
      parts = false;
      chunk(std::false_type());
      continue;
    }
    if (!parts) {
      load_parts(sE, k, 0);
      load_parts(sH, k - 1, 3);
      parts = true;
    }
    if (mid) {
      chunk(std::true_type());
      continue;
    }
#pragma unroll 1
    for (int u = 0; u < 4 && k + u <= kend; ++u) {
      round(k + u, u & 1, E[0], E[1], E[2], E[3], H[0], H[1], H[2], H[3], __shfl_sync(0xffffffffu, cf, u + 3),
            __shfl_sync(0xffffffffu, cf, u + 2), __shfl_sync(0xffffffffu, cf, u + 1), __shfl_sync(0xffffffffu, cf, u));
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const f2 e = E[0][q], h = H[0][q];
        E[0][q] = E[1][q]; E[1][q] = E[2][q]; E[2][q] = E[3][q]; E[3][q] = e;
        H[0][q] = H[1][q]; H[1][q] = H[2][q]; H[2][q] = H[3][q]; H[3][q] = h;
      }
    }
  }
}

// the flags of the rows of every column of tiles; a warp each
__global__ void row_flags3_kernel(const __grid_constant__ StepParams<float> p, const __grid_constant__ Block3 b, uint8_t *out) {
  const long long t = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= (long long)p.ny * p.nz * b.ntx) return;
  const int tx = (int)(t % b.ntx), lane = threadIdx.x & 31;
  const long long row = t / b.ntx;
  const int j = (int)(row % p.ny), k = (int)(row / p.ny);
  const bool split = p.pml_mode == 2;
  const bool genz = k < p.mlo[2] || k > p.mhi[2] || (split && (k < p.slo[2] || k > p.shi[2]));
  const bool rsrc = p.rowflag[row] & ROW_SRC;
  bool mix = false, ade = false, src = false, gen = genz || j < p.mlo[1] || j > p.mhi[1] || (j == 0 && !p.per[1]) ||
                          (split && (j < p.slo[1] || j > p.shi[1]));
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    int i = tx * b.ox - 2 + 2 * lane + q;
    if (p.per[0]) i = ((i % p.nx) + p.nx) % p.nx;
    if (i < p.mlo[0] || i > p.mhi[0] || (split && (i < p.slo[0] || i > p.shi[0]))) gen = true;
    if (rsrc && i >= 0 && i < p.nx)
      for (int s = 0; s < p.nsrc; ++s)
        src |= i >= p.src[s].lo[0] && i <= p.src[s].hi[0] && j >= p.src[s].lo[1] && j <= p.src[s].hi[1] &&
               k >= p.src[s].lo[2] && k <= p.src[s].hi[2];
    if (i >= 0 && i < p.nx) {
      const int id = p.mat[row * p.nx + i];
      mix |= id != p.id0;
      ade |= id >= kAdeId;
    }
  }
  bool smp = false;
  const int x0 = tx * b.ox, x1 = min(x0 + b.ox, p.nx) - 1;
  for (int m = lane; m < p.nmon; m += 32) {
    const Monitor &mo = p.mon[m];
    smp |= j >= mo.lo[1] && j <= mo.hi[1] && k >= mo.lo[2] && k <= mo.hi[2] && x0 <= mo.hi[0] && x1 >= mo.lo[0];
  }
  for (int m = lane; m < p.nprobe; m += 32)
    smp |= j == p.probe[m].cell[1] && k == p.probe[m].cell[2] && p.probe[m].cell[0] >= x0 && p.probe[m].cell[0] <= x1;
  mix = __any_sync(0xffffffffu, mix);
  src = __any_sync(0xffffffffu, src);
  ade = __any_sync(0xffffffffu, ade);
  gen = __any_sync(0xffffffffu, gen);
  smp = __any_sync(0xffffffffu, smp);
  if (lane == 0)
    out[t] = (uint8_t)((smp ? B3_SMP : 0) | (src ? B3_SRC : 0) | (mix ? B3_MIX : 0) | (gen ? B3_GEN : 0) | (genz ? B3_GENZ : 0) | (ade ? B3_ADE : 0));
}

constexpr int kB3Warps = 16;

template <int NS, bool ADE>
int launch3b(const StepParams<float> &p, const Block3 &b, cudaStream_t s) {
  const int blocks = ADE ? b.nade : b.ntx * b.nty * b.ntz - b.nade;
  if (blocks == 0) return 0;
  const int smem = 42 * 32 * kB3Warps * (int)sizeof(f2);
  static std::atomic<unsigned long long> done{0};
  if (!smem_limit(step3d_block<NS, kB3Warps, ADE>, smem, done)) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(32 * kB3Warps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, step3d_block<NS, kB3Warps, ADE>, p, b) == cudaSuccess ? 1 : -1;
}
}  // namespace

void launch_row_flags3(const StepParams<float> &p, const Block3 &b, uint8_t *out, void *stream) {
  const long long n = (long long)p.ny * p.nz * b.ntx;
  row_flags3_kernel<<<(unsigned)((n + 7) / 8), 256, 0, (cudaStream_t)stream>>>(p, b, out);
}

// Tiles: 60 of a row's 64 cells, 13 of 16 rows; along z as many chunks as make
// the rounds of the SMs' longest queue shortest.
void block3_tiles(Block3 &b, int nx, int ny, int nz, int num_sms) {
  b.ox = 60;
  b.oy = kB3Warps - 3;
  b.ntx = (nx + b.ox - 1) / b.ox;
  b.nty = (ny + b.oy - 1) / b.oy;
  const long long col = (long long)b.ntx * b.nty;
  long long best = -1;
  for (int c = 1; c <= nz; ++c) {
    const int oz = (nz + c - 1) / c, ntz = (nz + oz - 1) / oz;
    if (c > 1 && oz < 8) break;
    const long long cost = (col * ntz + num_sms - 1) / num_sms * (oz + 6);
    if (best < 0 || cost < best) {
      best = cost;
      b.oz = oz;
      b.ntz = ntz;
    }
  }
}

int launch_step3d_block(const StepParams<float> &p, const Block3 &b, int steps, bool ade, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (steps == 2) return ade ? launch3b<2, true>(p, b, s) : launch3b<2, false>(p, b, s);
  return ade ? launch3b<1, true>(p, b, s) : launch3b<1, false>(p, b, s);
}

}  // namespace fdtd
