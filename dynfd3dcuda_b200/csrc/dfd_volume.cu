// Fused volume stage: one pass per RK stage computes the velocity-stress right-hand
// side with the 5-point one-sided DRP operators and curvilinear metric terms
// (reference wave.cu:8-494), the free-surface rows and traction image (wave.cu:205-487),
// the ADE PML auxiliary equations of all six faces (pmlx.cu:8-214, pmly.cu, pmlz.cu),
// the classic RK4 register update (rk4.cu:20-33,154-257) and the Cerjan sponge
// (cerjan.cu:166-200).  The right-hand side never reaches HBM: each stage reads the
// stencil input (9 fields), the 12 metric/media fields and its RK registers, and writes
// its output and, at stage 2, the accumulator -- 30/39/57/39 floats per node for stages 0..3.
//
// Nodes of the seven x-layers around the fault whose (j,k) is not "united" are left
// to the band kernel (dfd_fault.cu), exactly the nodes whose right-hand side the
// reference overwrites in fault_dvelo / fault_dstrs.
#include <cstring>

#include "dfd_stencil.cuh"

namespace dfd {

template <int F>
__device__ __forceinline__ float d5(const float* __restrict__ v, long long q, long long s) {
  if (F == 1)
    return -DFD_C1 * __ldg(v + q - s) - DFD_C2 * __ldg(v + q) + DFD_C3 * __ldg(v + q + s) -
           DFD_C4 * __ldg(v + q + 2 * s) + DFD_C5 * __ldg(v + q + 3 * s);
  else
    return -DFD_C5 * __ldg(v + q - 3 * s) + DFD_C4 * __ldg(v + q - 2 * s) - DFD_C3 * __ldg(v + q - s) +
           DFD_C2 * __ldg(v + q) + DFD_C1 * __ldg(v + q + s);
}
template <int F>
__device__ __forceinline__ float d5w(const float* v) {  // on the five points of the operator's window
  if (F == 1) return -DFD_C1 * v[0] - DFD_C2 * v[1] + DFD_C3 * v[2] - DFD_C4 * v[3] + DFD_C5 * v[4];
  else return -DFD_C5 * v[0] + DFD_C4 * v[1] - DFD_C3 * v[2] + DFD_C2 * v[3] + DFD_C1 * v[4];
}

// traction vector jac * e_axis . sigma at node q
__device__ __forceinline__ void traction(const float* __restrict__ W, const float* __restrict__ M, long long n,
                                         long long q, int mo, float& t1, float& t2, float& t3) {
  float e0 = __ldg(M + mo * n + q), e1 = __ldg(M + (mo + 1) * n + q), e2 = __ldg(M + (mo + 2) * n + q);
  float jac = __ldg(M + 9 * n + q);
  float txx = __ldg(W + 3 * n + q), tyy = __ldg(W + 4 * n + q), tzz = __ldg(W + 5 * n + q);
  float txy = __ldg(W + 6 * n + q), txz = __ldg(W + 7 * n + q), tyz = __ldg(W + 8 * n + q);
  t1 = (e0 * txx + e1 * txy + e2 * txz) * jac;
  t2 = (e0 * txy + e1 * tyy + e2 * tyz) * jac;
  t3 = (e0 * txz + e1 * tyz + e2 * tzz) * jac;
}

// General node update below the free-surface rows: PML faces and sponge.  Used for the
// shell of the domain outside the plain interior kernel's box.
template <int FX, int FY, int FZ>
__device__ __forceinline__ void volume_point_general(const VolArgs& a, int i, int j, int k) {
  const Dims& d = a.d;
  int i1 = i + 3, j1 = j + 3, k1 = k + 3;
  if (a.united && i1 >= d.i0 - 3 && i1 <= d.i0 + 3 && !a.united[j + k * d.nj]) return;  // band node
  const long long n = d.nxyz;
  const long long q = idx3(d, i1, j1, k1);
  const float* __restrict__ W = a.Win;
  const float* __restrict__ M = a.M;

  float lam = __ldg(M + 10 * n + q), mu = __ldg(M + 11 * n + q);
  float rrho = 1.0f / __ldg(M + 12 * n + q);
  float rb1 = __ldg(a.rBx + i), rb2 = __ldg(a.rBy + j), rb3 = __ldg(a.rBz + k);
  float h[9], p[9], dv[9], D[9];
#pragma unroll
  for (int f = 0; f < 9; f++) p[f] = 0.0f;
  const bool px1 = a.aux[0] && i < d.N, px2 = a.aux[1] && i >= d.ni - d.N;
  const bool py1 = a.aux[2] && j < d.N, py2 = a.aux[3] && j >= d.nj - d.N;
  const bool pz1 = a.aux[4] && k < d.N, pz2 = a.aux[5] && k >= d.nk - d.N;
  float ez0 = __ldg(M + 6 * n + q), ez1 = __ldg(M + 7 * n + q), ez2 = __ldg(M + 8 * n + q);

  // ---- x ----
#pragma unroll
  for (int f = 0; f < 9; f++) dv[f] = d5<FX>(W + f * n, q, d.sx) * a.rDH;
  axis_terms(dv, __ldg(M + q), __ldg(M + n + q), __ldg(M + 2 * n + q), lam, mu, rrho, D);
#pragma unroll
  for (int f = 0; f < 9; f++) h[f] = D[f] * rb1;
  if (px1 || px2) {
    const int fc = px1 ? 0 : 1;
    const long long st = pml_fstride(d, fc), qa = pml_index(d, fc, i, j, k);
    pml_face<-1>(a, fc, qa, st, rb1, __ldg(a.Bx + i), __ldg(a.Dpx + i), __ldg(a.Apx + i), D,
             nullptr, ez0, ez1, ez2, lam, mu, p);
  }
  // ---- y ----
#pragma unroll
  for (int f = 0; f < 9; f++) dv[f] = d5<FY>(W + f * n, q, 1) * a.rDH;
  axis_terms(dv, __ldg(M + 3 * n + q), __ldg(M + 4 * n + q), __ldg(M + 5 * n + q), lam, mu, rrho, D);
#pragma unroll
  for (int f = 0; f < 9; f++) h[f] += D[f] * rb2;
  if (py1 || py2) {
    const int fc = py1 ? 2 : 3;
    const long long st = pml_fstride(d, fc), qa = pml_index(d, fc, i, j, k);
    pml_face<-1>(a, fc, qa, st, rb2, __ldg(a.By + j), __ldg(a.Dpy + j), __ldg(a.Apy + j), D,
             nullptr, ez0, ez1, ez2, lam, mu, p);
  }
  // ---- z ----
#pragma unroll
  for (int f = 0; f < 9; f++) dv[f] = d5<FZ>(W + f * n, q, d.py) * a.rDH;
  axis_terms(dv, ez0, ez1, ez2, lam, mu, rrho, D);
#pragma unroll
  for (int f = 0; f < 9; f++) h[f] += D[f] * rb3;
  if (pz1 || pz2) {
    const int fc = pz1 ? 4 : 5;
    const long long st = pml_fstride(d, fc), qa = pml_index(d, fc, i, j, k);
    pml_face<-1>(a, fc, qa, st, rb3, __ldg(a.Bz + k), __ldg(a.Dpz + k), __ldg(a.Apz + k), D, nullptr,
             ez0, ez1, ez2, lam, mu, p);
  }
  // ---- RK4 registers and Cerjan sponge
  float damp = 1.0f;
  if (a.dampx) damp = fminf(fminf(__ldg(a.dampx + i1), __ldg(a.dampy + j1)), __ldg(a.dampz + k1));
  rk_store<-1>(a, q, h, p, damp);
}


// The three free-surface rows.  Every node needs jac e . sigma (the traction of an axis) on
// the five points of each axis's operator: read point by point from memory that is 15 x 10
// loads a node, and the kernel waited on them (66 us per stage on the 400 x 300 x 200 job,
// 20.5 on 200 x 100 x 100; 47 and 17 now, still latency: 12 warps per SM, 0.3 instructions
// issued per cycle and scheduler, DRAM at 14 to 19 % of its peak).
// A block takes SJ columns x 3 rows x SI planes, evaluates the tractions once per node of
// its tile and halo into shared memory (per thread its own node, a node of the x halo, a
// quarter of one of the y halo and a third (forward z operator) or all of one of the z halo:
// 2.6 to 3.25) and applies the operators there.
constexpr int SJ = 16, SI = 4, SURF_THREADS = SJ * 3 * SI;
struct SurfTile {
  float t1[3][SI + 4][3][SJ];   // xi traction, halo in x
  float t2[3][SI][3][SJ + 4];   // eta traction, halo in y
  float t3[3][SI][6][SJ];       // zeta traction, rows nk - 6 .. nk - 1
};
static inline int surface_blocks(const Dims& d) { return ((d.nj + SJ - 1) / SJ) * ((d.ni + SI - 1) / SI); }

template <int FX, int FY, int FZ, int IRK>
__device__ __forceinline__ void surface_body(const VolArgs& a, int blk, SurfTile& st) {
  const Dims& d = a.d;
  constexpr int RX = FX == 1 ? 1 : 3, RY = FY == 1 ? 1 : 3, RZ = FZ == 1 ? 1 : 3;  // centre of each window
  const int gj = (d.nj + SJ - 1) / SJ;
  const int tx = threadIdx.x % SJ, zr = threadIdx.x / SJ % 3, xi = threadIdx.x / (3 * SJ);
  const int jb = (blk % gj) * SJ, ib = (blk / gj) * SI;
  const int i = ib + xi, j = jb + tx, k = d.nk - 3 + zr;
  const int i1 = i + 3, j1 = j + 3, k1 = k + 3;
  const long long n = d.nxyz;
  const long long q = idx3(d, i1, j1, k1);
  const float* __restrict__ W = a.Win;
  const float* __restrict__ M = a.M;
  float t[3], m[13];
  // own node (the halo columns and planes of the arrays hold what edge nodes read)
  if (i1 < d.nx && j1 < d.ny) {
#pragma unroll
    for (int e = 0; e < 13; e++) m[e] = __ldg(M + e * n + q);
    const float txx = __ldg(W + 3 * n + q), tyy = __ldg(W + 4 * n + q), tzz = __ldg(W + 5 * n + q);
    const float txy = __ldg(W + 6 * n + q), txz = __ldg(W + 7 * n + q), tyz = __ldg(W + 8 * n + q);
    st.t1[0][xi + RX][zr][tx] = (m[0] * txx + m[1] * txy + m[2] * txz) * m[9];
    st.t1[1][xi + RX][zr][tx] = (m[0] * txy + m[1] * tyy + m[2] * tyz) * m[9];
    st.t1[2][xi + RX][zr][tx] = (m[0] * txz + m[1] * tyz + m[2] * tzz) * m[9];
    st.t2[0][xi][zr][tx + RY] = (m[3] * txx + m[4] * txy + m[5] * txz) * m[9];
    st.t2[1][xi][zr][tx + RY] = (m[3] * txy + m[4] * tyy + m[5] * tyz) * m[9];
    st.t2[2][xi][zr][tx + RY] = (m[3] * txz + m[4] * tyz + m[5] * tzz) * m[9];
    st.t3[0][xi][3 + zr][tx] = (m[6] * txx + m[7] * txy + m[8] * txz) * m[9];
    st.t3[1][xi][3 + zr][tx] = (m[6] * txy + m[7] * tyy + m[8] * tyz) * m[9];
    st.t3[2][xi][3 + zr][tx] = (m[6] * txz + m[7] * tyz + m[8] * tzz) * m[9];
    // z halo: three rows below for the backward operator, one for the forward one
    if (FZ == -1 || zr == 2) {
      traction(W, M, n, q - 3LL * d.py, 6, t[0], t[1], t[2]);
#pragma unroll
      for (int c = 0; c < 3; c++) st.t3[c][xi][zr][tx] = t[c];
    }
  }
  {
    // x halo: one of its four planes per thread plane
    const int px = xi < RX ? xi : xi + SI, ih = ib + px - RX + 3;
    if (ih < d.nx && j1 < d.ny) {
      traction(W, M, n, idx3(d, ih, j1, k1), 0, t[0], t[1], t[2]);
#pragma unroll
      for (int c = 0; c < 3; c++) st.t1[c][px][zr][tx] = t[c];
    }
  }
  if (tx < 4) {
    const int col = tx < RY ? tx : tx + SJ, jh = jb + col - RY + 3;
    if (jh < d.ny && i1 < d.nx) {
      traction(W, M, n, idx3(d, i1, jh, k1), 3, t[0], t[1], t[2]);
#pragma unroll
      for (int c = 0; c < 3; c++) st.t2[c][xi][zr][col] = t[c];
    }
  }
  __syncthreads();
  if (i >= d.ni || j >= d.nj) return;
  if (a.united && i1 >= d.i0 - 3 && i1 <= d.i0 + 3 && !a.united[j + k * d.nj]) return;  // band node

  const float lam = m[10], mu = m[11], rrho = 1.0f / m[12];
  const float rb1 = __ldg(a.rBx + i), rb2 = __ldg(a.rBy + j), rb3 = __ldg(a.rBz + k);
  const float ez0 = m[6], ez1 = m[7], ez2 = m[8];
  float h[9], p[9], dv[9], D[9], dxv[3], dyv[3], dz[3];
#pragma unroll
  for (int f = 0; f < 9; f++) p[f] = 0.0f;
  const bool top = k == d.nk - 1;
  const bool px1 = a.aux[0] && i < d.N, px2 = a.aux[1] && i >= d.ni - d.N;
  const bool py1 = a.aux[2] && j < d.N, py2 = a.aux[3] && j >= d.nj - d.N;
  const bool pz1 = a.aux[4] && k < d.N, pz2 = a.aux[5] && k >= d.nk - d.N;
  // The momentum equation comes from the tractions below, so the stress derivatives are
  // formed only for the ADE state of a face (D[0..2]).
#pragma unroll
  for (int f = 0; f < 9; f++) dv[f] = 0.0f;
  // ---- x ----
#pragma unroll
  for (int f = 0; f < 3; f++) dxv[f] = dv[f] = d5<FX>(W + f * n, q, d.sx) * a.rDH;
  if (px1 || px2) {
#pragma unroll
    for (int f = 3; f < 9; f++) dv[f] = d5<FX>(W + f * n, q, d.sx) * a.rDH;
  }
  axis_terms(dv, m[0], m[1], m[2], lam, mu, rrho, D);
#pragma unroll
  for (int f = 3; f < 9; f++) h[f] = D[f] * rb1;
  if (px1 || px2) {
    if (top) {
      const float* mx = a.mVx2Vz + (j1 + (long long)i1 * d.ny) * 9;
#pragma unroll
      for (int r = 0; r < 3; r++) dz[r] = mx[3 * r] * dxv[0] + mx[3 * r + 1] * dxv[1] + mx[3 * r + 2] * dxv[2];
    }
    const int fc = px1 ? 0 : 1;
    pml_face<IRK>(a, fc, pml_index(d, fc, i, j, k), pml_fstride(d, fc), rb1, __ldg(a.Bx + i), __ldg(a.Dpx + i),
                  __ldg(a.Apx + i), D, top ? dz : nullptr, ez0, ez1, ez2, lam, mu, p);
  }
  // ---- y ----
#pragma unroll
  for (int f = 0; f < 3; f++) dyv[f] = dv[f] = d5<FY>(W + f * n, q, 1) * a.rDH;
  if (py1 || py2) {
#pragma unroll
    for (int f = 3; f < 9; f++) dv[f] = d5<FY>(W + f * n, q, 1) * a.rDH;
  }
  axis_terms(dv, m[3], m[4], m[5], lam, mu, rrho, D);
#pragma unroll
  for (int f = 3; f < 9; f++) h[f] += D[f] * rb2;
  if (py1 || py2) {
    if (top) {
      const float* my = a.mVy2Vz + (j1 + (long long)i1 * d.ny) * 9;
#pragma unroll
      for (int r = 0; r < 3; r++) dz[r] = my[3 * r] * dyv[0] + my[3 * r + 1] * dyv[1] + my[3 * r + 2] * dyv[2];
    }
    const int fc = py1 ? 2 : 3;
    pml_face<IRK>(a, fc, pml_index(d, fc, i, j, k), pml_fstride(d, fc), rb2, __ldg(a.By + j), __ldg(a.Dpy + j),
                  __ldg(a.Apy + j), D, top ? dz : nullptr, ez0, ez1, ez2, lam, mu, p);
  }
  // ---- z: a face's ADE state takes the plain derivatives, the stress rates the velocity
  // derivatives of the top rows (wave.cu:205-245)
  if (pz1 || pz2) {
#pragma unroll
    for (int f = 0; f < 9; f++) dv[f] = d5<FZ>(W + f * n, q, d.py) * a.rDH;
    axis_terms(dv, ez0, ez1, ez2, lam, mu, rrho, D);
    const int fc = pz1 ? 4 : 5;
    pml_face<IRK>(a, fc, pml_index(d, fc, i, j, k), pml_fstride(d, fc), rb3, __ldg(a.Bz + k), __ldg(a.Dpz + k),
                  __ldg(a.Apz + k), D, nullptr, ez0, ez1, ez2, lam, mu, p);
  }
  if (top) {
    const float* mx = a.mVx2Vz + (j1 + (long long)i1 * d.ny) * 9;
    const float* my = a.mVy2Vz + (j1 + (long long)i1 * d.ny) * 9;
#pragma unroll
    for (int r = 0; r < 3; r++)
      dv[r] = (mx[3 * r] * dxv[0] + mx[3 * r + 1] * dxv[1] + mx[3 * r + 2] * dxv[2]) +
              (my[3 * r] * dyv[0] + my[3 * r + 1] * dyv[1] + my[3 * r + 2] * dyv[2]);
  } else if (k == d.nk - 2) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const float* v = W + r * n;
      dv[r] = (FZ == 1 ? (__ldg(v + q + d.py) - __ldg(v + q)) : (__ldg(v + q) - __ldg(v + q - d.py))) * a.rDH;
    }
  } else {
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const float* v = W + r * n;
      dv[r] = (FZ == 1 ? (-DFD_C24_1 * __ldg(v + q) + DFD_C24_2 * __ldg(v + q + d.py) - DFD_C24_3 * __ldg(v + q + 2 * d.py))
                       : (DFD_C24_3 * __ldg(v + q - 2 * d.py) - DFD_C24_2 * __ldg(v + q - d.py) + DFD_C24_1 * __ldg(v + q))) *
              a.rDH;
    }
  }
  axis_terms(dv, ez0, ez1, ez2, lam, mu, rrho, D);
#pragma unroll
  for (int f = 3; f < 9; f++) h[f] += D[f] * rb3;
  // ---- traction image for the momentum equation (wave.cu:398-487): no traction on the top
  // row, its odd image above
  const float rrhojac = rrho / m[9];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    float vx[5], vy[5], vz[5];
#pragma unroll
    for (int s = 0; s < 5; s++) {
      vx[s] = st.t1[c][xi + s][zr][tx];
      vy[s] = st.t2[c][xi][zr][tx + s];
      const int row = 3 + zr + s - RZ;
      vz[s] = row == 5 ? 0.0f : row > 5 ? -st.t3[c][xi][10 - row][tx] : st.t3[c][xi][row][tx];
    }
    h[c] = (d5w<FX>(vx) * a.rDH * rb1 + d5w<FY>(vy) * a.rDH * rb2 + d5w<FZ>(vz) * a.rDH * rb3) * rrhojac;
  }
  // ---- RK4 registers and Cerjan sponge
  float damp = 1.0f;
  if (a.dampx) damp = fminf(fminf(__ldg(a.dampx + i1), __ldg(a.dampy + j1)), __ldg(a.dampz + k1));
  rk_store<IRK>(a, q, h, p, damp);
}
template <int FX, int FY, int FZ, int IRK>
__global__ void __launch_bounds__(SURF_THREADS, 2) volume_surface_kernel(const __grid_constant__ VolArgs a) {
  __shared__ SurfTile st;
  surface_body<FX, FY, FZ, IRK>(a, blockIdx.x, st);
}
// all scenarios of an ensemble in one launch: scenario s owns blocks [start[s], start[s+1])
template <int FX, int FY, int FZ, int IRK>
__global__ void __launch_bounds__(SURF_THREADS, 2)
    volume_surface_batch(const VolArgs* __restrict__ tab, const int* __restrict__ start, int n) {
  __shared__ __align__(16) unsigned char raw_a[sizeof(VolArgs)];
  __shared__ SurfTile st;
  VolArgs* sa = reinterpret_cast<VolArgs*>(raw_a);
  int loc;
  const int sc = scenario_of(start, n, blockIdx.x, &loc);
  stage_args(sa, tab + sc);
  __syncthreads();
  surface_body<FX, FY, FZ, IRK>(*sa, loc, st);
}

// Shell kernels: the general update on up to six boxes (PML slabs) that surround the plain
// interior kernel's box; one 1-D grid of 128-thread blocks is split over them.  At most 170
// registers (the PML path needs about 160), three blocks per SM.  A box at least 32 nodes
// wide in y and 4 in z is tiled (32 y, 4 z) per block; a thinner box (the y slabs of the
// PML) is flattened over (y, z) with y fastest, so that no thread idles and the y-face PML
// state (y fastest over N nodes, then z) is read contiguously.
constexpr int SHELL_THREADS = 128;

template <int FX, int FY, int FZ>
__device__ __forceinline__ void volume_shell_body(const VolArgs& a, const Boxes& bx, int blk) {
  int b = 0;
  while (b + 1 < bx.ntop && blk >= bx.start[b + 1]) b++;
  int loc = blk - bx.start[b];
  int ni = bx.hi[b][0] - bx.lo[b][0], nj = bx.hi[b][1] - bx.lo[b][1], nk = bx.hi[b][2] - bx.lo[b][2];
  int i, j, k;
  if (bx.thin[b]) {
    int gyz = (nj * nk + SHELL_THREADS - 1) / SHELL_THREADS;
    int t = (loc % gyz) * SHELL_THREADS + threadIdx.x;
    i = loc / gyz;
    j = t % nj;
    k = t / nj;
    if (k >= nk) return;
  } else {
    int gj = (nj + 31) / 32, gk = (nk + 3) / 4;
    int bj = loc % gj, bk = (loc / gj) % gk, bi = loc / (gj * gk);
    j = bj * 32 + (threadIdx.x & 31);
    k = bk * 4 + (threadIdx.x >> 5);
    i = bi;
    if (i >= ni || j >= nj || k >= nk) return;
  }
  volume_point_general<FX, FY, FZ>(a, bx.lo[b][0] + i, bx.lo[b][1] + j, bx.lo[b][2] + k);
}
template <int FX, int FY, int FZ>
__global__ void __launch_bounds__(SHELL_THREADS, 3)
    volume_shell_kernel(const __grid_constant__ VolArgs a, const __grid_constant__ Boxes bx) {
  volume_shell_body<FX, FY, FZ>(a, bx, blockIdx.x);
}
// all scenarios of an ensemble in one launch: scenario s owns blocks [start[s], start[s+1])
template <int FX, int FY, int FZ>
__global__ void __launch_bounds__(SHELL_THREADS, 3)
    volume_shell_batch(const VolArgs* __restrict__ tab, const Boxes* __restrict__ boxes,
                       const int* __restrict__ start, int n) {
  __shared__ __align__(16) unsigned char raw_a[sizeof(VolArgs)];
  __shared__ __align__(16) unsigned char raw_b[sizeof(Boxes)];
  VolArgs* sa = reinterpret_cast<VolArgs*>(raw_a);
  Boxes* sb = reinterpret_cast<Boxes*>(raw_b);
  int loc;
  const int sc = scenario_of(start, n, blockIdx.x, &loc);
  stage_args(sa, tab + sc);
  stage_args(sb, boxes + sc);
  __syncthreads();
  volume_shell_body<FX, FY, FZ>(*sa, *sb, loc);
}

// Interior kernel: no PML (beta = 1, no auxiliary state), no free-surface rows.  Each
// derivative is scattered into the nine right-hand sides as soon as it is formed, which
// keeps the register count low enough for three resident blocks per SM; each thread
// walks a chunk of x so that the x-stencil halo is reused from L1.
template <int FX, int FY, int FZ>
__device__ __forceinline__ void interior_point(const VolArgs& a, long long q, float damp) {
  const long long n = a.d.nxyz;
  const float* __restrict__ W = a.Win;
  const float* __restrict__ M = a.M;
  const float r = a.rDH;
  float lam = __ldg(M + 10 * n + q), mu = __ldg(M + 11 * n + q);
  float rrho = 1.0f / __ldg(M + 12 * n + q);
  float l2m = lam + 2.0f * mu;
  float h0 = 0.f, h1 = 0.f, h2 = 0.f, h3 = 0.f, h4 = 0.f, h5 = 0.f, h6 = 0.f, h7 = 0.f, h8 = 0.f;
#define DFD_AXIS(F, S, MO)                                                                         \
  {                                                                                                \
    float e0 = __ldg(M + (MO) * n + q), e1 = __ldg(M + ((MO) + 1) * n + q), e2 = __ldg(M + ((MO) + 2) * n + q); \
    float dv;                                                                                      \
    dv = d5<F>(W, q, S) * r;                                                                       \
    h3 += dv * e0 * l2m; h4 += dv * e0 * lam; h5 += dv * e0 * lam; h6 += dv * e1 * mu; h7 += dv * e2 * mu; \
    dv = d5<F>(W + n, q, S) * r;                                                                   \
    h3 += dv * e1 * lam; h4 += dv * e1 * l2m; h5 += dv * e1 * lam; h6 += dv * e0 * mu; h8 += dv * e2 * mu; \
    dv = d5<F>(W + 2 * n, q, S) * r;                                                               \
    h3 += dv * e2 * lam; h4 += dv * e2 * lam; h5 += dv * e2 * l2m; h7 += dv * e0 * mu; h8 += dv * e1 * mu; \
    float er0 = e0 * rrho, er1 = e1 * rrho, er2 = e2 * rrho;                                       \
    dv = d5<F>(W + 3 * n, q, S) * r; h0 += dv * er0;                                               \
    dv = d5<F>(W + 4 * n, q, S) * r; h1 += dv * er1;                                               \
    dv = d5<F>(W + 5 * n, q, S) * r; h2 += dv * er2;                                               \
    dv = d5<F>(W + 6 * n, q, S) * r; h0 += dv * er1; h1 += dv * er0;                               \
    dv = d5<F>(W + 7 * n, q, S) * r; h0 += dv * er2; h2 += dv * er0;                               \
    dv = d5<F>(W + 8 * n, q, S) * r; h1 += dv * er2; h2 += dv * er1;                               \
  }
  DFD_AXIS(FX, a.d.sx, 0)
  DFD_AXIS(FY, 1, 3)
  DFD_AXIS(FZ, a.d.py, 6)
#undef DFD_AXIS
  const float hv[9] = {h0, h1, h2, h3, h4, h5, h6, h7, h8};
  rk_store<-1>(a, q, hv, nullptr, damp);
}

template <int FX, int FY, int FZ>
__global__ void __launch_bounds__(256, 3) volume_interior_kernel(VolArgs a, int3 lo, int3 hi, int chunk) {
  const Dims& d = a.d;
  int j = lo.y + blockIdx.x * blockDim.x + threadIdx.x;
  int k = lo.z + blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= hi.y || k >= hi.z) return;
  int ib = lo.x + blockIdx.z * chunk, ie = min(ib + chunk, hi.x);
  bool band = a.united && !a.united[j + k * d.nj];
  float dyz = 1.0f;
  if (a.dampx) dyz = fminf(__ldg(a.dampy + j + 3), __ldg(a.dampz + k + 3));
  long long q = idx3(d, ib + 3, j + 3, k + 3);
  for (int i = ib; i < ie; i++, q += d.sx) {
    if (band && i + 3 >= d.i0 - 3 && i + 3 <= d.i0 + 3) continue;
    float damp = a.dampx ? fminf(__ldg(a.dampx + i + 3), dyz) : 1.0f;
    interior_point<FX, FY, FZ>(a, q, damp);
  }
}

// Volume work of one stage: which box the tiled (or plain) interior kernel takes, the
// units of the tiled PML kernel, the boxes of the general kernel and the free-surface rows.
VolPlan plan_volume(const VolArgs& a, const TileCtx* tc) {
  const Dims& d = a.d;
  VolPlan pl;
  pl.tiled = pl.plain = false;
  pl.nodes = 0;
  pl.pgrid = 0;
  memset(&pl.ps, 0, sizeof pl.ps);
  Boxes& bx = pl.bx;
  bx.n = bx.ntop = 0;
  auto add = [&](int i0, int i1, int j0, int j1, int k0, int k1) {
    if (i1 <= i0 || j1 <= j0 || k1 <= k0) return;
    bx.lo[bx.n][0] = i0; bx.lo[bx.n][1] = j0; bx.lo[bx.n][2] = k0;
    bx.hi[bx.n][0] = i1; bx.hi[bx.n][1] = j1; bx.hi[bx.n][2] = k1;
    bx.n++;
  };
  // interior box: outside every PML slab, below the free-surface rows
  int nx0 = a.aux[0] ? d.N : 0, nx1 = a.aux[1] ? d.N : 0;
  int ny0 = a.aux[2] ? d.N : 0, ny1 = a.aux[3] ? d.N : 0;
  int nz0 = a.aux[4] ? d.N : 0, nz1 = a.aux[5] ? d.N : (a.freenode ? 3 : 0);
  int3 lo = make_int3(nx0, ny0, nz0), hi = make_int3(d.ni - nx1, d.nj - ny1, d.nk - nz1);
  const int ktop = a.freenode ? d.nk - 3 : d.nk;
  bool done = false;
  if (tc && tc->ok) {
    // the interior kernel takes the box between the slabs (its y start a multiple of 16,
    // where the PML kernel's y1 strips end; its y end a multiple of 4, where the y2
    // strips start); the PML kernel every other node below the free-surface rows
    int ya = a.aux[2] ? (d.N + STRIP - 1) / STRIP * STRIP : 0;
    int yb = a.aux[3] ? (d.nj - d.N) / 4 * 4 : d.nj;
    if (a.aux[3] && yb > ya) {
      // A column of the interior kernel's 32-wide tiles and a column of the PML kernel's
      // 16-wide strips cost about the same (half the nodes at about twice the cost per
      // node), and a partial column costs nearly a full one.  Of the y ends up to 28
      // columns earlier, take the one with the fewest columns of both (ties: the latest):
      // with NY = 600 and PML 20 that is 576 (17 whole tiles, two strips), not 580 (an
      // 18th tile 4 columns wide, the same two strips).
      auto cols = [&](int y) { return (y - ya + TILE_J - 1) / TILE_J + (d.nj - y + STRIP - 1) / STRIP; };
      int best = yb;
      for (int y = yb - 4; y >= yb - 28 && y > ya; y -= 4)
        if (cols(y) < cols(best)) best = y;
      yb = best;
    }
    int za = a.aux[4] ? d.N : 0;
    int zb = a.aux[5] ? d.nk - d.N : ktop;
    if (yb <= ya) ya = yb = 0;     // no interior column: strips over every column
    // whole 8-row tiles in z: the rows left over go to the PML kernel's z tiles (whose
    // second tile row over a 12-row slab has room for them), not to a nearly empty row of
    // interior tiles
    const int zr = (zb - za) % TILE_K;
    if (zb - za >= TILE_K && zr) {
      if (a.aux[4]) za += zr;
      else zb -= zr;
    }
    // ... unless they then cost the z1 slab a row of z tiles of its own: a row of the PML
    // kernel's tiles costs about two of the interior kernel's, so with PML 20 and 297 rows
    // (25 rows: a fourth z-tile row holding one) the slab keeps its 20 rows in three tile
    // rows and the interior box ends in a partial tile row
    if (a.aux[4] && zb - za >= TILE_K) {
      auto rows = [&](int z) { return 2 * ((z + TILE_K - 1) / TILE_K) + (zb - z + TILE_K - 1) / TILE_K; };
      int best = za;
      for (int z = d.N; z < za; z++)
        if (rows(z) < rows(best)) best = z;
      za = best;
    }
    if (zb <= za || zb - za < TILE_K) za = zb = ktop;  // no interior row: z tiles over every row
    int grid = 0;
    TileSched ps = pml_plan(a, ya, yb, za, zb, ktop, tc->nsm, &grid);
    const int3 rlo = make_int3(lo.x, ya, za), rhi = make_int3(hi.x, yb, zb);
    const bool inner = rhi.x > rlo.x && rhi.y > rlo.y && rhi.z > rlo.z;
    if (ps.nunits >= 0 && (!inner || tile_feasible(tc, a, rlo, rhi))) {
      done = true;
      pl.ps = ps;
      pl.pgrid = grid;
      if (inner) {
        pl.tiled = true;
        pl.lo = rlo;
        pl.hi = rhi;
      }
      add(0, d.ni, 0, d.nj, ktop, d.nk);  // the free-surface rows
    }
  }
  if (!done) {
    // the plain interior kernel on the interior box, the general kernel on the slabs
    // around it, then on the free-surface rows
    const bool some = hi.x > lo.x && hi.y > lo.y && hi.z > lo.z;
    if (some) {
      pl.plain = true;
      pl.lo = lo;
      pl.hi = hi;
    } else {
      lo = hi = make_int3(0, 0, 0);
    }
    add(0, lo.x, 0, d.nj, 0, ktop);
    add(hi.x, d.ni, 0, d.nj, 0, ktop);
    add(lo.x, hi.x, 0, lo.y, 0, ktop);
    add(lo.x, hi.x, hi.y, d.nj, 0, ktop);
    add(lo.x, hi.x, lo.y, hi.y, 0, lo.z);
    add(lo.x, hi.x, lo.y, hi.y, hi.z, ktop);
    bx.ntop = bx.n;
    add(0, d.ni, 0, d.nj, ktop, d.nk);
  }
  if (pl.tiled || pl.plain) pl.nodes = (long long)(pl.hi.x - pl.lo.x) * (pl.hi.y - pl.lo.y) * (pl.hi.z - pl.lo.z);
  int tot = 0;
  for (int b = 0; b < bx.n; b++) {
    bx.start[b] = tot;
    int ni = bx.hi[b][0] - bx.lo[b][0], nj = bx.hi[b][1] - bx.lo[b][1], nk = bx.hi[b][2] - bx.lo[b][2];
    bx.thin[b] = nj < 32 || nk < 4;
    if (b >= bx.ntop) tot += surface_blocks(d);  // the free-surface rows
    else tot += bx.thin[b] ? ((nj * nk + SHELL_THREADS - 1) / SHELL_THREADS) * ni : ((nj + 31) / 32) * ((nk + 3) / 4) * ni;
  }
  bx.start[bx.n] = tot;
  pl.shell_blocks = tot;
  return pl;
}

template <int FX, int FY, int FZ>
static long long launch_flags(const VolArgs& a, cudaStream_t s, cudaStream_t s_shell, const TileCtx* tc, int bin,
                              cudaEvent_t* kb, cudaEvent_t* ke, VolPlan* out, cudaEvent_t* fork) {
  const VolPlan pl = plan_volume(a, tc);
  if (out) *out = pl;
  if (kb) cudaEventRecord(*kb, s);
  if (pl.tiled) {
    launch_tile(tc, a, FX, FY, FZ, bin, pl.lo, pl.hi, s);
  } else if (pl.plain) {
    const int chunk = 8;
    dim3 block(32, 8, 1);
    dim3 grid((pl.hi.y - pl.lo.y + 31) / 32, (pl.hi.z - pl.lo.z + 7) / 8, (pl.hi.x - pl.lo.x + chunk - 1) / chunk);
    volume_interior_kernel<FX, FY, FZ><<<grid, block, 0, s>>>(a, pl.lo, pl.hi, chunk);
  }
  if (ke) cudaEventRecord(*ke, s);
  // directly behind the interior kernel unless timing events separate them
  if (pl.ps.nunits > 0) launch_pml(tc, a, FX, FY, FZ, bin, pl.ps, pl.pgrid, pl.tiled && !ke, s);
  if (fork && s_shell != s) {
    // the kernels below on s_shell once the tiled ones are done
    cudaEventRecord(*fork, s);
    cudaStreamWaitEvent(s_shell, *fork, 0);
  }
  const int below = pl.bx.start[pl.bx.ntop], above = pl.bx.start[pl.bx.n] - below;
  if (below > 0) volume_shell_kernel<FX, FY, FZ><<<below, SHELL_THREADS, 0, s_shell>>>(a, pl.bx);
  if (above > 0) {
#define DFD_L(K) volume_surface_kernel<FX, FY, FZ, K><<<above, SURF_THREADS, 0, s_shell>>>(a)
    DFD_BY_STAGE(a.irk, DFD_L);
#undef DFD_L
  }
  return pl.nodes;
}

template <int FX, int FY, int FZ>
static void shell_batch_t(const VolArgs* tab, const Boxes* boxes, const int* start, int n, int blocks, bool top,
                          int irk, cudaStream_t s) {
  if (top) {
#define DFD_L(K) volume_surface_batch<FX, FY, FZ, K><<<blocks, SURF_THREADS, 0, s>>>(tab, start, n)
    DFD_BY_STAGE(irk, DFD_L);
#undef DFD_L
  } else {
    volume_shell_batch<FX, FY, FZ><<<blocks, SHELL_THREADS, 0, s>>>(tab, boxes, start, n);
  }
}
void launch_shell_batch(const VolArgs* tab, const Boxes* boxes, const int* start, int n, int blocks, int FX, int FY,
                        int FZ, bool top, int irk, cudaStream_t s) {
  if (blocks <= 0) return;
  int code = (FX > 0) * 4 + (FY > 0) * 2 + (FZ > 0);
  switch (code) {
    case 0: shell_batch_t<-1, -1, -1>(tab, boxes, start, n, blocks, top, irk, s); break;
    case 1: shell_batch_t<-1, -1, 1>(tab, boxes, start, n, blocks, top, irk, s); break;
    case 2: shell_batch_t<-1, 1, -1>(tab, boxes, start, n, blocks, top, irk, s); break;
    case 3: shell_batch_t<-1, 1, 1>(tab, boxes, start, n, blocks, top, irk, s); break;
    case 4: shell_batch_t<1, -1, -1>(tab, boxes, start, n, blocks, top, irk, s); break;
    case 5: shell_batch_t<1, -1, 1>(tab, boxes, start, n, blocks, top, irk, s); break;
    case 6: shell_batch_t<1, 1, -1>(tab, boxes, start, n, blocks, top, irk, s); break;
    default: shell_batch_t<1, 1, 1>(tab, boxes, start, n, blocks, top, irk, s); break;
  }
}

// Launches the volume kernels of one stage; kb/ke (optional) are recorded on s right
// before and after the interior (tiled) kernel; with fork (and s_shell != s) the general and
// free-surface kernels run on s_shell after the tiled kernels, else on s_shell right away.  Returns the
// nodes of the box the interior kernel covers.
long long launch_volume_stage(const VolArgs& a, int FX, int FY, int FZ, cudaStream_t s, cudaStream_t s_shell,
                              const TileCtx* tc, int bin, cudaEvent_t* kb, cudaEvent_t* ke, VolPlan* out,
                              cudaEvent_t* fork) {
  int code = (FX > 0) * 4 + (FY > 0) * 2 + (FZ > 0);
  switch (code) {
    case 0: return launch_flags<-1, -1, -1>(a, s, s_shell, tc, bin, kb, ke, out, fork);
    case 1: return launch_flags<-1, -1, 1>(a, s, s_shell, tc, bin, kb, ke, out, fork);
    case 2: return launch_flags<-1, 1, -1>(a, s, s_shell, tc, bin, kb, ke, out, fork);
    case 3: return launch_flags<-1, 1, 1>(a, s, s_shell, tc, bin, kb, ke, out, fork);
    case 4: return launch_flags<1, -1, -1>(a, s, s_shell, tc, bin, kb, ke, out, fork);
    case 5: return launch_flags<1, -1, 1>(a, s, s_shell, tc, bin, kb, ke, out, fork);
    case 6: return launch_flags<1, 1, -1>(a, s, s_shell, tc, bin, kb, ke, out, fork);
    default: return launch_flags<1, 1, 1>(a, s, s_shell, tc, bin, kb, ke, out, fork);
  }
}

}  // namespace dfd
