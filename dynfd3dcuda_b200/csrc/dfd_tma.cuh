// Device helpers of the TMA-staged volume kernels (dfd_tile.cu: interior box,
// dfd_pml.cu: PML slabs): tile geometry, mbarrier and bulk-copy primitives, the
// one-sided operators on shared-memory lines, the per-node metric and the RK4 store.
//
// A tile is 32 (y) x 8 (z) nodes; a CTA owns one tile column and marches along x.  Every
// tile starts on a 16-byte boundary in y (the volume rows start one element early, so
// node j = 0 sits at a 16-byte boundary), as TMA requires for the innermost coordinate.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include "dfd_stencil.cuh"

namespace dfd {

namespace {
constexpr int TJ = TILE_J, TK = TILE_K;
constexpr int HW = TJ + 8;           // halo box width (y): 4 nodes each side (16-byte aligned)
constexpr int HH = TK + 4;           // halo box height (z): 1 + 3 rows, side set by the z operator
constexpr int HBOX = HW * HH;        // floats per field of a halo box
constexpr int HSLOT = 9 * HBOX;      // floats per stencil plane slot
constexpr int PB = TJ * TK;          // floats per field of a pointwise box
constexpr int QSLOT = 12 * PB;       // metric / media planes of a unit: U V ety etz zty ztz, 2 x (lam mu rho)
constexpr long long WAIT_LIMIT = 1LL << 22;  // polls of one mbarrier before giving up
constexpr long long DRILL_LIMIT = 1LL << 12; // the same in the test drill of the bounded waits
static_assert((HSLOT * 4) % 128 == 0 && (QSLOT * 4) % 128 == 0 && (PB * 4) % 128 == 0, "slot alignment");
static_assert(sizeof(TileUnit) % 16 == 0 && offsetof(TileScen, u) % 16 == 0, "bulk copy of the scenario values");
}  // namespace

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait for the completion of phase `parity`; false if it did not complete
__device__ __forceinline__ bool mbar_wait_n(uint64_t* b, unsigned parity, long long limit) {
  for (long long n = 0; n < limit; n++)
    if (mbar_try(b, parity)) return true;
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity) { return mbar_wait_n(b, parity, WAIT_LIMIT); }
__device__ __forceinline__ void tma_load4(float* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                          uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(b))
      : "memory");
}

// plain bulk copy (no tensor map) of bytes (a multiple of 16, both addresses 16-byte
// aligned) from global to shared memory, completing on mbarrier b
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(b))
               : "memory");
}

__device__ __forceinline__ void tma_load3(float* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(b))
      : "memory");
}

// one-sided 5-point operators on values (v0..v4 = the five stencil points in order)
template <int F>
__device__ __forceinline__ float d5v(float v0, float v1, float v2, float v3, float v4) {
  if (F == 1) return -DFD_C1 * v0 - DFD_C2 * v1 + DFD_C3 * v2 - DFD_C4 * v3 + DFD_C5 * v4;
  else return -DFD_C5 * v0 + DFD_C4 * v1 - DFD_C3 * v2 + DFD_C2 * v3 + DFD_C1 * v4;
}
// on a shared-memory line through p with stride S (forward: p-S..p+3S, backward: p-3S..p+S)
template <int F, int S>
__device__ __forceinline__ float d5s(const float* p) {
  if (F == 1) return d5v<1>(p[-S], p[0], p[S], p[2 * S], p[3 * S]);
  else return d5v<-1>(p[-3 * S], p[-2 * S], p[-S], p[0], p[S]);
}



// slot / phase-parity cursor over a ring of N mbarrier-guarded slots
struct Ring {
  int slot = 0, phase = 0;
  template <int N>
  __device__ __forceinline__ void next() {
    if (++slot == N) { slot = 0; phase ^= 1; }
  }
};

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}

// RK4 register update of fields F0..F1-1 of node q with right-hand side hv, then the
// sponge factor (rk4.cu:20-33, cerjan.cu:166-200): step-start values from the stencil
// input at stage 0, from the pointwise slot P at stages 1 and 2; at stage 2 the slot's
// second box holds the stage-1 input, from which, with y0 and the stage input, the
// accumulator is formed (rk_sum, rk_acc); at stage 3 the slot holds the accumulator
// alone, first.  IRK: the
// stage (the kernels are compiled per stage).
template <int F0, int F1, int IRK>
__device__ __forceinline__ void rk_tile_store(const VolArgs& a, long long n, long long q, const float* cur,
                                              const float* P, const float* hv, float damp) {
  const float rd = IRK == 2 ? rk_rd(damp) : 1.0f;
#pragma unroll
  for (int f = F0; f < F1; f++) {
    const long long x = f * n + q;
    float w;
    if (IRK == 0) {
      w = fmaf(a.rka, hv[f], cur[f * HBOX]);
    } else if (IRK == 1) {
      w = fmaf(a.rka, hv[f], P[f * PB]);
    } else if (IRK == 2) {
      const float y0 = P[f * PB];
      a.T[x] = rk_acc(y0, rk_sum(y0, P[(9 + f) * PB], cur[f * HBOX], rd), a.rkb, hv[f]);
      w = fmaf(a.rka, hv[f], y0);
    } else {
      w = fmaf(a.rkb, hv[f], P[f * PB]);
    }
    a.Wout[x] = w * damp;
  }
}

// Metric and media of a node of the tiled box: x row (xi), y row (eta), z row (zeta) and
// the elastic constants (the separable factors of dfd_setup.cu's plane_metric_kernel; the
// x components of eta and zeta are exactly zero there and in the stored metric).
struct NodeMetric {
  float ex0, ex1, ex2, ey1, ey2, ez1, ez2, lam, mu, rrho;
};


// Lean right-hand side of a node outside every PML slab and below the free-surface rows
// (rB = 1, no ADE state): momentum (velocity rates, hv[0..2]) and constitutive law (stress
// rates, hv[3..8]) from the one-sided derivatives on the shared-memory stencil planes
// (xs0..xs4 the five x planes, cur the node's plane; 32 x 8 tiles, the PML kernel's).  The x
// row of the metric has three components; the y and z rows have no x component, so the terms
// with it (exact zeros) and the derivative of Txx along y and z drop out.  Reference
// wave.cu:8-204.  The interior kernel has its own form on pairs of nodes (below).
#define DFD_DERX(f) d5v<FX>(xs0[(f) * HBOX], xs1[(f) * HBOX], xs2[(f) * HBOX], xs3[(f) * HBOX], xs4[(f) * HBOX])
#define DFD_DERY(f) d5s<FY, 1>(cur + (f) * HBOX)
#define DFD_DERZ(f) d5s<FZ, HW>(cur + (f) * HBOX)
template <int FX, int FY, int FZ>
__device__ __forceinline__ void lean_velocity(const float* xs0, const float* xs1, const float* xs2, const float* xs3,
                                              const float* xs4, const float* cur, const NodeMetric& g, float r,
                                              float* hv) {
  const float rrho = g.rrho;
  // momentum: velocity rates from the six stress derivatives per axis
  float h0 = 0.f, h1 = 0.f, h2 = 0.f;
  {
    const float er0 = g.ex0 * rrho, er1 = g.ex1 * rrho, er2 = g.ex2 * rrho;
    float dv;
    dv = DFD_DERX(3) * r; h0 += dv * er0;
    dv = DFD_DERX(4) * r; h1 += dv * er1;
    dv = DFD_DERX(5) * r; h2 += dv * er2;
    dv = DFD_DERX(6) * r; h0 += dv * er1; h1 += dv * er0;
    dv = DFD_DERX(7) * r; h0 += dv * er2; h2 += dv * er0;
    dv = DFD_DERX(8) * r; h1 += dv * er2; h2 += dv * er1;
  }
#define DFD_VAXIS0(DER, E1, E2)                                                                     \
  {                                                                                                 \
    const float er1 = (E1) * rrho, er2 = (E2) * rrho;                                               \
    float dv;                                                                                       \
    dv = DER(4) * r; h1 += dv * er1;                                                                \
    dv = DER(5) * r; h2 += dv * er2;                                                                \
    dv = DER(6) * r; h0 += dv * er1;                                                                \
    dv = DER(7) * r; h0 += dv * er2;                                                                \
    dv = DER(8) * r; h1 += dv * er2; h2 += dv * er1;                                                \
  }
  DFD_VAXIS0(DFD_DERY, g.ey1, g.ey2)
  DFD_VAXIS0(DFD_DERZ, g.ez1, g.ez2)
#undef DFD_VAXIS0
  hv[0] = h0; hv[1] = h1; hv[2] = h2;
}
template <int FX, int FY, int FZ>
__device__ __forceinline__ void lean_stress(const float* xs0, const float* xs1, const float* xs2, const float* xs3,
                                            const float* xs4, const float* cur, const NodeMetric& g, float r,
                                            float* hv) {
  const float lam = g.lam, mu = g.mu;
  const float l2m = lam + 2.0f * mu;
  // constitutive law: stress rates from the three velocity derivatives per axis
  float h3 = 0.f, h4 = 0.f, h5 = 0.f, h6 = 0.f, h7 = 0.f, h8 = 0.f;
  {
    const float e0 = g.ex0, e1 = g.ex1, e2 = g.ex2;
    float dv;
    dv = DFD_DERX(0) * r;
    h3 += dv * e0 * l2m; h4 += dv * e0 * lam; h5 += dv * e0 * lam; h6 += dv * e1 * mu; h7 += dv * e2 * mu;
    dv = DFD_DERX(1) * r;
    h3 += dv * e1 * lam; h4 += dv * e1 * l2m; h5 += dv * e1 * lam; h6 += dv * e0 * mu; h8 += dv * e2 * mu;
    dv = DFD_DERX(2) * r;
    h3 += dv * e2 * lam; h4 += dv * e2 * lam; h5 += dv * e2 * l2m; h7 += dv * e0 * mu; h8 += dv * e1 * mu;
  }
#define DFD_SAXIS0(DER, E1, E2)                                                                     \
  {                                                                                                 \
    const float e1 = (E1), e2 = (E2);                                                               \
    float dv;                                                                                       \
    dv = DER(0) * r; h6 += dv * e1 * mu; h7 += dv * e2 * mu;                                        \
    dv = DER(1) * r;                                                                                \
    h3 += dv * e1 * lam; h4 += dv * e1 * l2m; h5 += dv * e1 * lam; h8 += dv * e2 * mu;              \
    dv = DER(2) * r;                                                                                \
    h3 += dv * e2 * lam; h4 += dv * e2 * lam; h5 += dv * e2 * l2m; h8 += dv * e1 * mu;              \
  }
  DFD_SAXIS0(DFD_DERY, g.ey1, g.ey2)
  DFD_SAXIS0(DFD_DERZ, g.ez1, g.ez2)
#undef DFD_SAXIS0
  hv[3] = h3; hv[4] = h4; hv[5] = h5; hv[6] = h6; hv[7] = h7; hv[8] = h8;
}
#undef DFD_DERX
#undef DFD_DERY
#undef DFD_DERZ

// ---------------- two nodes per thread (packed FP32 pairs, one instruction for both)
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 pk(float a) { return pk(a, a); }
__device__ __forceinline__ void upk(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 lds2(const float* p) { return *reinterpret_cast<const f2*>(p); }

// F times the one-sided derivative on five points in memory order: with the backward
// operator's points taken in reverse, both signs use the same five constants, and the sign
// goes into the metric factor of the axis.
template <int F>
__device__ __forceinline__ f2 d5p(f2 v0, f2 v1, f2 v2, f2 v3, f2 v4) {
  const f2 p0 = F == 1 ? v0 : v4, p1 = F == 1 ? v1 : v3, p3 = F == 1 ? v3 : v1, p4 = F == 1 ? v4 : v0;
  f2 r = mul2(p0, pk(-DFD_C1));
  r = fma2(p1, pk(-DFD_C2), r);
  r = fma2(v2, pk(DFD_C3), r);
  r = fma2(p3, pk(-DFD_C4), r);
  return fma2(p4, pk(DFD_C5), r);
}
template <int F>
__device__ __forceinline__ float d5n(float v0, float v1, float v2, float v3, float v4) {
  const float p0 = F == 1 ? v0 : v4, p1 = F == 1 ? v1 : v3, p3 = F == 1 ? v3 : v1, p4 = F == 1 ? v4 : v0;
  return fmaf(DFD_C5, p4, fmaf(-DFD_C4, p3, fmaf(DFD_C3, v2, fmaf(-DFD_C2, p1, -DFD_C1 * p0))));
}
// along y through the pair at p (its first node at an even column): the points of both nodes
// come as aligned pairs, each node's operator in scalar (the pairs of an odd shift would
// have to be put together first)
template <int F>
__device__ __forceinline__ f2 d5y(const float* p) {
  float a, b, c, d, e, f, g, h;
  if (F == 1) {  // nodes 0, 1 need -1 .. 4
    upk(lds2(p - 2), a, b);
    upk(lds2(p), c, d);
    upk(lds2(p + 2), e, f);
    g = p[4];
    return pk(d5n<1>(b, c, d, e, f), d5n<1>(c, d, e, f, g));
  }
  // nodes 0, 1 need -3 .. 2
  a = p[-3];
  upk(lds2(p - 2), b, c);
  upk(lds2(p), d, e);
  upk(lds2(p + 2), f, h);
  return pk(d5n<-1>(a, b, c, d, e), d5n<-1>(b, c, d, e, f));
}
template <int F, int S>
__device__ __forceinline__ f2 d5z(const float* p) {
  if (F == 1) return d5p<1>(lds2(p - S), lds2(p), lds2(p + S), lds2(p + 2 * S), lds2(p + 3 * S));
  return d5p<-1>(lds2(p - 3 * S), lds2(p - 2 * S), lds2(p - S), lds2(p), lds2(p + S));
}

// Metric of a pair in the interior box: the xi row is xr (1, U, V) with xr = FX / (DH a(x)),
// the eta and zeta rows (ey, ez) carry FY / DH and FZ / DH.
struct PairMetric {
  f2 xr, U, V, ey1, ey2, ez1, ez2;
};
#define DFD_PX(f) d5p<FX>(lds2(x0 + (f) * HB), lds2(x1 + (f) * HB), lds2(x2 + (f) * HB), lds2(x3 + (f) * HB), lds2(x4 + (f) * HB))
#define DFD_PY(f) d5y<FY>(cur + (f) * HB)
#define DFD_PZ(f) d5z<FZ, PW>(cur + (f) * HB)
// lean_velocity and lean_stress on a pair; the sums over the metric rows are formed before
// the media factors (21 products for the six strain rates instead of 36)
template <int FX, int FY, int FZ, int PW, int HB>
__device__ __forceinline__ void pair_velocity(const float* x0, const float* x1, const float* x2, const float* x3,
                                              const float* x4, const float* cur, const PairMetric& g, f2 rrho, f2* hv) {
  f2 h0, h1, h2, t;
  h0 = DFD_PX(3);
  t = DFD_PX(6); h0 = fma2(g.U, t, h0); h1 = t;
  t = DFD_PX(7); h0 = fma2(g.V, t, h0); h2 = t;
  t = DFD_PX(4); h1 = fma2(g.U, t, h1);
  t = DFD_PX(8); h1 = fma2(g.V, t, h1); h2 = fma2(g.U, t, h2);
  t = DFD_PX(5); h2 = fma2(g.V, t, h2);
  h0 = mul2(h0, g.xr); h1 = mul2(h1, g.xr); h2 = mul2(h2, g.xr);
  t = DFD_PY(4); h1 = fma2(g.ey1, t, h1);
  t = DFD_PY(5); h2 = fma2(g.ey2, t, h2);
  t = DFD_PY(6); h0 = fma2(g.ey1, t, h0);
  t = DFD_PY(7); h0 = fma2(g.ey2, t, h0);
  t = DFD_PY(8); h1 = fma2(g.ey2, t, h1); h2 = fma2(g.ey1, t, h2);
  t = DFD_PZ(4); h1 = fma2(g.ez1, t, h1);
  t = DFD_PZ(5); h2 = fma2(g.ez2, t, h2);
  t = DFD_PZ(6); h0 = fma2(g.ez1, t, h0);
  t = DFD_PZ(7); h0 = fma2(g.ez2, t, h0);
  t = DFD_PZ(8); h1 = fma2(g.ez2, t, h1); h2 = fma2(g.ez1, t, h2);
  hv[0] = mul2(h0, rrho); hv[1] = mul2(h1, rrho); hv[2] = mul2(h2, rrho);
}
template <int FX, int FY, int FZ, int PW, int HB>
__device__ __forceinline__ void pair_stress(const float* x0, const float* x1, const float* x2, const float* x3,
                                            const float* x4, const float* cur, const PairMetric& g, f2 lam, f2 mu,
                                            f2* hv) {
  f2 d0, d1, d2, s01, s02, s12, t;
  t = DFD_PX(0); d0 = t; s01 = mul2(g.U, t); s02 = mul2(g.V, t);
  t = DFD_PX(1); d1 = mul2(g.U, t); s01 = add2(s01, t); s12 = mul2(g.V, t);
  t = DFD_PX(2); d2 = mul2(g.V, t); s02 = add2(s02, t); s12 = fma2(g.U, t, s12);
  d0 = mul2(d0, g.xr); d1 = mul2(d1, g.xr); d2 = mul2(d2, g.xr);
  s01 = mul2(s01, g.xr); s02 = mul2(s02, g.xr); s12 = mul2(s12, g.xr);
  t = DFD_PY(0); s01 = fma2(g.ey1, t, s01); s02 = fma2(g.ey2, t, s02);
  t = DFD_PY(1); d1 = fma2(g.ey1, t, d1); s12 = fma2(g.ey2, t, s12);
  t = DFD_PY(2); d2 = fma2(g.ey2, t, d2); s12 = fma2(g.ey1, t, s12);
  t = DFD_PZ(0); s01 = fma2(g.ez1, t, s01); s02 = fma2(g.ez2, t, s02);
  t = DFD_PZ(1); d1 = fma2(g.ez1, t, d1); s12 = fma2(g.ez2, t, s12);
  t = DFD_PZ(2); d2 = fma2(g.ez2, t, d2); s12 = fma2(g.ez1, t, s12);
  const f2 m2 = add2(mu, mu), tr = mul2(lam, add2(add2(d0, d1), d2));
  hv[3] = fma2(m2, d0, tr); hv[4] = fma2(m2, d1, tr); hv[5] = fma2(m2, d2, tr);
  hv[6] = mul2(mu, s01); hv[7] = mul2(mu, s02); hv[8] = mul2(mu, s12);
}
#undef DFD_PX
#undef DFD_PY
#undef DFD_PZ

// rk_tile_store on a pair; n0, n1: which of the two nodes are updated
template <int F0, int F1, int IRK, int HB, int PBB>
__device__ __forceinline__ void rk_pair_store(const VolArgs& a, long long n, long long q, const float* cur,
                                              const float* P, const f2* hv, float damp0, float damp1, bool n0, bool n1) {
  const f2 damp = pk(damp0, damp1), rka = pk(a.rka), rkb = pk(a.rkb);
  f2 rd;
  if (IRK == 2) rd = pk(rk_rd(damp0), rk_rd(damp1));
  auto put = [&](float* x, f2 v) {
    if (n0 && n1) {
      *reinterpret_cast<f2*>(x) = v;
    } else {
      float v0, v1;
      upk(v, v0, v1);
      if (n0) x[0] = v0;
      if (n1) x[1] = v1;
    }
  };
#pragma unroll
  for (int f = F0; f < F1; f++) {
    const long long x = f * n + q;
    f2 w;
    if (IRK == 0) {
      w = fma2(rka, hv[f], lds2(cur + f * HB));
    } else if (IRK == 1) {
      w = fma2(rka, hv[f], lds2(P + f * PBB));
    } else if (IRK == 2) {
      const f2 y0 = lds2(P + f * PBB), ny0 = mul2(y0, pk(-1.0f));
      const f2 u = fma2(lds2(P + (9 + f) * PBB), rd, ny0), v = fma2(lds2(cur + f * HB), rd, ny0);
      const f2 s = fma2(pk(2.0f), v, u);
      put(a.T + x, fma2(rkb, hv[f], fma2(s, pk(1.0f / 3.0f), y0)));
      w = fma2(rka, hv[f], y0);
    } else {
      w = fma2(rkb, hv[f], lds2(P + f * PBB));
    }
    put(a.Wout + x, mul2(w, damp));
  }
}

// first scenario of a batched launch whose units include the global unit u
__device__ __forceinline__ int tile_scenario(const TileScen* tab, int n, int u) {
  int lo = 0, hi = n;  // tab[lo].unit0 <= u < tab[hi].unit0
  while (hi - lo > 1) {
    int m = (lo + hi) / 2;
    if (tab[m].u.unit0 <= u) lo = m; else hi = m;
  }
  return lo;
}

}  // namespace dfd
