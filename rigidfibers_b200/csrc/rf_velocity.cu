// Velocity update (numerical inner integrals) and the fiber time integrator.
//
// Reference: fortran/update_velocities.incl:1-89 (and the CUDA kernels
// src/kernels/reset_velocities.cu:6-39, update_velocities_2D.cu:6-166):
//   U_i = (0.5/d) [ (d+2) F + (d-2)(t_i.F) t_i + sum_{j!=i} sum_qi w_qi GF_ij(qi) ]
//   W_i = (1.5/d) (I - t_i t_i^T) sum_{j!=i} sum_qi w_qi P_1(s_qi) GF_ij(qi)
//   GF_ij(qi) = sum_qj w_qj K(R_ij(qi,qj)) f_j(qj),  f_j = F/2 + sum_k a_{j,k} P_{k+1}
// fortran/update_fibers_firststep.incl:1-10 and update_fibers.incl:1-17 for
// the time step, here accumulated in FP64 on FP64 state.
// Reductions are deterministic: per-(j-chunk, fiber) partial sums, then a
// fixed-order sum; no atomics.
#include "rf_common.cuh"
#include "rf_kernels.cuh"
#include "rf_analytic.cuh"

namespace rf {

// Source densities of both quadrature rules, weight included:
// fw[j * (Q + FN) + q] = w_q f_j(s_q) = W[0][q] F/2 + sum_k a_{j,k} W[k+1][q] for
// the Q points of the full rule, then the FN points of the far rule.
__global__ void k_source_density(const Tables tab, int N, const float* __restrict__ x, float4* __restrict__ fw,
                                 int* __restrict__ vflag) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *vflag = 0;   // the stage's non-finite guard (k_velocity_finalize)
  const int Q = tab.Q, M = tab.M, P = Q + kFarNodes;
  const int64_t n = (int64_t)N * P;
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(u / P), q = (int)(u % P);
    auto weight = [&](int k) { return q < Q ? tab.W[k][q] : tab.far_W[k][q - Q]; };
    float f0 = 0.f, f1 = 0.f, f2 = weight(0) * tab.fz_half;
    const float* a = x + (int64_t)j * 3 * M;
    for (int k = 0; k < M; ++k) {
      const float w = weight(k + 1);
      f0 = fmaf(a[3 * k + 0], w, f0);
      f1 = fmaf(a[3 * k + 1], w, f1);
      f2 = fmaf(a[3 * k + 2], w, f2);
    }
    fw[u] = make_float4(f0, f1, f2, 0.f);
  }
}

// acc += K(p - s t) f for one point of fiber j (p relative to its centre).  NR: a
// Newton step on the reciprocal root (the far rule's 64 kernel values per pair
// average their roundings less than the full rule's 576).
template <bool NR>
__device__ __forceinline__ void stokeslet_apply(float px, float py, float pz, const float4& st, const float4& f,
                                                float e2, float e2x3, float (&acc)[3]) {
  const float rx = px - st.x, ry = py - st.y, rz = pz - st.z;
  const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
  float inv = rsqrtf(r2);
  if (NR) inv = fmaf(0.5f * inv, fmaf(-r2 * inv, inv, 1.f), inv);
  const float inv2 = inv * inv;
  const float inv3 = inv2 * inv;
  const float inv5 = inv3 * inv2;
  const float a = fmaf(e2, inv3, inv);
  const float bb = fmaf(e2x3, inv5, inv3);
  // K f = a f + bb R (R.f)
  const float rf = fmaf(rx, f.x, fmaf(ry, f.y, rz * f.z)) * bb;
  acc[0] = fmaf(a, f.x, fmaf(rf, rx, acc[0]));
  acc[1] = fmaf(a, f.y, fmaf(rf, ry, acc[1]));
  acc[2] = fmaf(a, f.z, fmaf(rf, rz, acc[2]));
}

// Velocity sums of one ordered pair set.  Sources at least sqrt(far_d2) away (the
// assembly's rule, see make_tables) take the far rule, 64 kernel values per pair
// instead of Q^2; the others the full rule.  One launch: the first near_blocks
// blocks are near ones, the rest far ones, so that the few near pairs run beside
// the far ones.  Bound: FP32 issue; below a few hundred fibers latency, so both
// parts split the sources into many partial rows (vpart[row][i][6]: far chunks,
// then near segments).  Sums over one source's points are formed before they are
// added to the fiber's: the roundings stay those of one pair.
constexpr int kVelFibers = 32;
constexpr int kVelThreads = kVelFibers * kFarNodes;

struct VelSplit {
  int segs, jseg, near_blocks;      // near: source segments, sources per segment, blocks
  int chunks, jchunk, far_blocks;   // far: source chunks, sources per chunk, blocks
};

// 32 fibers i x one chunk of sources, thread (fiber, far point of i); the
// sources pass through shared memory 32 at a time (broadcast reads: lane = fiber)
__device__ __forceinline__ void velocity_far_block(const Tables& tab, int N, const double4* __restrict__ pos64,
                                                   const float4* __restrict__ ori, const float4* __restrict__ fw,
                                                   int tile, int chunk, int jchunk, float* __restrict__ vpart) {
  constexpr int FN = kFarNodes, B = kVelFibers;
  __shared__ float4 sP[B][FN], sF[B][FN];    // s_q t_j, w_q f_j(s_q)
  __shared__ double sXj[B][3];
  __shared__ float sGs[3][FN][B];
  const int tid = threadIdx.x;
  const int il = tid % B, qi = tid / B;
  const int i = tile * B + il;
  const int P = tab.Q + FN;
  double xi[3];
  float si[3];
  {
    const double4 x = pos64[min(i, N - 1)];
    const float4 t = ori[min(i, N - 1)];
    const float s = tab.far_pts[qi];
    xi[0] = x.x; xi[1] = x.y; xi[2] = x.z;
    si[0] = s * t.x; si[1] = s * t.y; si[2] = s * t.z;
  }
  const float e2 = tab.e2, e2x3 = -3.f * tab.e2, far_d2 = tab.far_d2;
  float g[3] = {0.f, 0.f, 0.f};
  const int jbeg = chunk * jchunk, jend = min(N, jbeg + jchunk);
  for (int js = jbeg; js < jend; js += B) {
    __syncthreads();
    {
      const int jl = tid / FN, q = tid % FN;
      const int j = min(js + jl, N - 1);
      const float4 t = ori[j];
      const float s = tab.far_pts[q];
      sP[jl][q] = make_float4(s * t.x, s * t.y, s * t.z, 0.f);
      sF[jl][q] = fw[(int64_t)j * P + tab.Q + q];
      if (q == 0) {
        const double4 x = pos64[j];
        sXj[jl][0] = x.x; sXj[jl][1] = x.y; sXj[jl][2] = x.z;
      }
    }
    __syncthreads();
    const int jn = min(B, jend - js);
    for (int jl = 0; jl < jn; ++jl) {
      // the centre difference in FP64, rounded once (as in the assembly): the
      // error scales with the fibers' distance, not with their distance from the origin
      const float dx = (float)(xi[0] - sXj[jl][0]), dy = (float)(xi[1] - sXj[jl][1]), dz = (float)(xi[2] - sXj[jl][2]);
      if (!far_pair(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), far_d2)) continue;   // near, or i itself
      float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < FN; ++q)
        stokeslet_apply<true>(dx + si[0], dy + si[1], dz + si[2], sP[jl][q], sF[jl][q], e2, e2x3, acc);
      g[0] += acc[0]; g[1] += acc[1]; g[2] += acc[2];
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) sGs[a][qi][il] = g[a];
  __syncthreads();
  // per fiber: sum_qi w_qi gs(qi) and sum_qi w_qi P_1(s_qi) gs(qi)
  if (tid < B * 6) {
    const int fl = tid % B, comp = tid / B;
    const float* w = comp >= 3 ? tab.far_W[1] : tab.far_W[0];
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < FN; ++q) s = fmaf(w[q], sGs[comp % 3][q][fl], s);
    if (tile * B + fl < N) vpart[((int64_t)chunk * N + tile * B + fl) * 6 + comp] = s;
  }
}

// dst[0..5] = sum_q W[0][q] g(q), sum_q W[1][q] g(q) over a warp whose lane l holds
// the points l, l + 32 of one fiber
template <int Q>
__device__ __forceinline__ void near_row_sums(const Tables& tab, const float (&g)[(Q + 31) / 32][3],
                                              float* __restrict__ dst) {
  constexpr int NP = (Q + 31) / 32;
  const int lane = threadIdx.x & 31;
  float u[6] = {};
#pragma unroll
  for (int h = 0; h < NP; ++h) {
    const int q = lane + 32 * h;
    if (q < Q) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        u[a] = fmaf(tab.W[0][q], g[h][a], u[a]);
        u[3 + a] = fmaf(tab.W[1][q], g[h][a], u[3 + a]);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < 6; ++a) u[a] += __shfl_xor_sync(0xffffffffu, u[a], o);
  if (lane < 6) {
    float v = u[0];
#pragma unroll
    for (int a = 1; a < 6; ++a) v = lane == a ? u[a] : v;
    dst[lane] = v;
  }
}

// One warp: fiber i's near sources of one segment, found 32 centres at a time and
// taken in index order, lane = quadrature point of i (Q = 48: two passes).  A
// source's densities pass through the warp's Q float4 of shared memory, the next
// one's on their way meanwhile: read where they are used, each batch of a few was
// a trip to L2 of its own (100 fibers: the velocities 52.7 us, 40.7 so).
template <int Q>
__device__ __forceinline__ void velocity_near_warp(const Tables& tab, int N, const double4* __restrict__ pos64,
                                                   const float4* __restrict__ ori, const float4* __restrict__ fw,
                                                   int i, int jbeg, int jend, float4* __restrict__ sf,
                                                   float* __restrict__ row) {
  constexpr int NP = (Q + 31) / 32;   // points per lane
  const int lane = threadIdx.x & 31;
  const int P = Q + kFarNodes;
  const double4 xi = pos64[i];
  const float4 ti = ori[i];
  const float e2 = tab.e2, e2x3 = -3.f * tab.e2, far_d2 = tab.far_d2;
  float g[NP][3] = {};
  float4 f[NP], t = ti;
  auto fetch = [&](int j) {
#pragma unroll
    for (int h = 0; h < NP; ++h)
      if (lane + 32 * h < Q) f[h] = fw[(int64_t)j * P + lane + 32 * h];
    t = ori[j];
  };
  for (int js = jbeg; js < jend; js += 32) {
    const int j = js + lane;
    float d[3] = {0.f, 0.f, 0.f};
    bool near = false;
    if (j < jend) {
      const double4 xj = pos64[j];
      d[0] = (float)(xi.x - xj.x); d[1] = (float)(xi.y - xj.y); d[2] = (float)(xi.z - xj.z);
      near = j != i && !far_pair(fmaf(d[0], d[0], fmaf(d[1], d[1], d[2] * d[2])), far_d2);
    }
    unsigned m = __ballot_sync(0xffffffffu, near);
    if (m != 0) fetch(js + __ffs(m) - 1);
    while (m != 0) {
      const int src = __ffs(m) - 1;
      const float4 tj = t;
      __syncwarp();   // the source before this one is read
#pragma unroll
      for (int h = 0; h < NP; ++h)
        if (lane + 32 * h < Q) sf[lane + 32 * h] = f[h];
      __syncwarp();
      m &= m - 1;
      if (m != 0) fetch(js + __ffs(m) - 1);
      const float dx = __shfl_sync(0xffffffffu, d[0], src), dy = __shfl_sync(0xffffffffu, d[1], src),
                  dz = __shfl_sync(0xffffffffu, d[2], src);
#pragma unroll
      for (int h = 0; h < NP; ++h) {
        const int q = lane + 32 * h;
        if (q < Q) {
          const float s = tab.pts[q];
          const float px = dx + s * ti.x, py = dy + s * ti.y, pz = dz + s * ti.z;
          float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll 4
          for (int p = 0; p < Q; ++p) {
            const float sp = tab.pts[p];
            stokeslet_apply<false>(px, py, pz, make_float4(sp * tj.x, sp * tj.y, sp * tj.z, 0.f),
                                   sf[p], e2, e2x3, acc);
          }
#pragma unroll
          for (int a = 0; a < 3; ++a) g[h][a] += acc[a];
        }
      }
    }
  }
  near_row_sums<Q>(tab, g, row + (int64_t)i * 6);
}

template <int Q>
__global__ void __launch_bounds__(kVelThreads)
k_velocity_numerical(const Tables tab, int N, const double4* __restrict__ pos64, const float4* __restrict__ ori,
                     const float4* __restrict__ fw, VelSplit v, float* __restrict__ vpart) {
  const int b = (int)blockIdx.x - v.near_blocks;
  if (b >= 0) {
    velocity_far_block(tab, N, pos64, ori, fw, b / v.chunks, b % v.chunks, v.jchunk, vpart);
    return;
  }
  __shared__ float4 sf[kVelThreads / 32][Q];
  const int w = (int)blockIdx.x * (kVelThreads / 32) + (int)(threadIdx.x >> 5);
  const int i = w / v.segs, seg = w % v.segs;
  if (i < N)
    velocity_near_warp<Q>(tab, N, pos64, ori, fw, i, seg * v.jseg, min(N, (seg + 1) * v.jseg), sf[threadIdx.x >> 5],
                          vpart + (int64_t)(v.chunks + seg) * N * 6);
}

// Sum of the partial rows (velocity_rows_block), self term, projection, scaling
// and the non-finite guard; *vflag was cleared by an earlier kernel of the stage.
__global__ void __launch_bounds__(kVelSumThreads)
k_velocity_finalize(const Tables tab, int N, const float4* __restrict__ ori, const float* __restrict__ vpart,
                    int nrows, float4* __restrict__ tvel, float4* __restrict__ rvel, int* __restrict__ vflag) {
  __shared__ float sums[kVelSumFibers][7];
  velocity_rows_block(vpart, nrows, N, blockIdx.x * kVelSumFibers, sums);
  const int i = blockIdx.x * kVelSumFibers + threadIdx.x;
  if (threadIdx.x >= kVelSumFibers || i >= N) return;
  const float* S = sums[threadIdx.x];
  const float4 t = ori[i];
  const float d = tab.d;
  const float Fz = 2.f * tab.fz_half;            // F = (0, 0, -1)
  const float tF = t.z * Fz;
  const float U[3] = {(d - 2.f) * tF * t.x + S[0], (d - 2.f) * tF * t.y + S[1],
                      (d + 2.f) * Fz + (d - 2.f) * tF * t.z + S[2]};
  const float W[3] = {S[3], S[4], S[5]};
  const float tW = t.x * W[0] + t.y * W[1] + t.z * W[2];
  const float su = 0.5f / d, sr = 1.5f / d;
  const float4 u = make_float4(U[0] * su, U[1] * su, U[2] * su, 0.f);
  const float4 w = make_float4((W[0] - t.x * tW) * sr, (W[1] - t.y * tW) * sr, (W[2] - t.z * tW) * sr, 0.f);
  tvel[i] = u;
  rvel[i] = w;
  if (!velocity_finite(u, w)) *vflag = 1;   // every writer stores the same value
}

// Analytical variant: the inner integral over fiber j in closed form (FP64),
// GF_ij(qi) = G_0(qi) F/2 + sum_k G_{k+1}(qi) a_{j,k}; the outer quadrature over
// fiber i as in the numerical kernel, the far rule's points for far sources.
// This is how the reference's 100_analytic_* golden files were produced (its
// committed fortran/update_velocities.incl integrates numerically in both
// modes).  Bound: FP64 issue of the closed form.
template <int M>
__device__ __forceinline__ void analytic_apply(const double (&R0)[3], const double4& tj4, const float* __restrict__ a,
                                               double e2, float fz, float (&g)[3]) {
  const double tj[3] = {tj4.x, tj4.y, tj4.z};
  float G[6][M + 1];
  analytic_G<M>(R0, tj, e2, G);
  // F/2 = (0, 0, fz): column z of G_0
  float f0 = G[4][0] * fz, f1 = G[5][0] * fz, f2 = G[2][0] * fz;
#pragma unroll
  for (int k = 0; k < M; ++k) {
    const float a0 = a[3 * k], a1 = a[3 * k + 1], a2 = a[3 * k + 2];
    f0 += G[0][k + 1] * a0 + G[3][k + 1] * a1 + G[4][k + 1] * a2;
    f1 += G[3][k + 1] * a0 + G[1][k + 1] * a1 + G[5][k + 1] * a2;
    f2 += G[4][k + 1] * a0 + G[5][k + 1] * a1 + G[2][k + 1] * a2;
  }
  g[0] += f0; g[1] += f1; g[2] += f2;
}

// Far blocks (after the near ones): 16 fibers x 8 far points x one chunk of
// sources, lane = fiber.  Near blocks: one warp per (fiber, segment), lane =
// quadrature point.  Partial rows as the numerical kernel's.
constexpr int kAnaFibers = 16;
constexpr int kAnaThreads = kAnaFibers * kFarNodes;

template <int M, int Q>
__global__ void __launch_bounds__(kAnaThreads, 3)
k_velocity_analytical(const Tables tab, int N, const double4* __restrict__ pos, const double4* __restrict__ ori,
                      const float* __restrict__ coeff, VelSplit v, float* __restrict__ vpart,
                      int* __restrict__ vflag) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *vflag = 0;
  constexpr int M3 = 3 * M, FN = kFarNodes, B = kAnaFibers;
  const int tid = threadIdx.x, lane = tid & 31;
  const double e2 = 2.0 * (double)tab.eps * (double)tab.eps;
  const float fz = tab.fz_half, far_d2 = tab.far_d2;
  auto dist2 = [](const double4& a, const double4& b) {
    const float dx = (float)(a.x - b.x), dy = (float)(a.y - b.y), dz = (float)(a.z - b.z);
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  };
  const int b = (int)blockIdx.x - v.near_blocks;
  if (b >= 0) {
    __shared__ float sGs[3][FN][B];
    const int tile = b / v.chunks, chunk = b % v.chunks;
    const int il = tid % B, qi = tid / B, i = tile * B + il;
    float g[3] = {0.f, 0.f, 0.f};
    if (i < N) {
      const double4 xi = pos[i], ti = ori[i];
      const double s = (double)tab.far_pts[qi];
      const double pt[3] = {xi.x + s * ti.x, xi.y + s * ti.y, xi.z + s * ti.z};
      const int jend = min(N, (chunk + 1) * v.jchunk);
      for (int j = chunk * v.jchunk; j < jend; ++j) {
        const double4 xj = pos[j];
        if (!far_pair(dist2(xi, xj), far_d2)) continue;   // near, or i itself
        const double R0[3] = {pt[0] - xj.x, pt[1] - xj.y, pt[2] - xj.z};
        analytic_apply<M>(R0, ori[j], coeff + (int64_t)j * M3, e2, fz, g);
      }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) sGs[a][qi][il] = g[a];
    __syncthreads();
    if (tid < B * 6) {
      const int fl = tid % B, comp = tid / B;
      const float* w = comp >= 3 ? tab.far_W[1] : tab.far_W[0];
      float acc = 0.f;
#pragma unroll
      for (int q = 0; q < FN; ++q) acc = fmaf(w[q], sGs[comp % 3][q][fl], acc);
      if (tile * B + fl < N) vpart[((int64_t)chunk * N + tile * B + fl) * 6 + comp] = acc;
    }
    return;
  }
  const int w = (int)blockIdx.x * (kAnaThreads / 32) + (tid >> 5);
  const int i = w / v.segs, seg = w % v.segs;
  if (i >= N) return;
  constexpr int NP = (Q + 31) / 32;
  const double4 xi = pos[i], ti = ori[i];
  float g[NP][3] = {};
  const int jend = min(N, (seg + 1) * v.jseg);
  for (int js = seg * v.jseg; js < jend; js += 32) {
    const int j = js + lane;
    const bool near = j < jend && j != i && !far_pair(dist2(xi, pos[j]), far_d2);
    for (unsigned m = __ballot_sync(0xffffffffu, near); m != 0; m &= m - 1) {
      const int jj = js + __ffs(m) - 1;
      const double4 xj = pos[jj], tj = ori[jj];
#pragma unroll
      for (int h = 0; h < NP; ++h) {
        const int q = lane + 32 * h;
        if (q < Q) {
          const double s = (double)tab.pts[q];
          const double R0[3] = {xi.x + s * ti.x - xj.x, xi.y + s * ti.y - xj.y, xi.z + s * ti.z - xj.z};
          analytic_apply<M>(R0, tj, coeff + (int64_t)jj * M3, e2, fz, g[h]);
        }
      }
    }
  }
  near_row_sums<Q>(tab, g, vpart + (int64_t)(v.chunks + seg) * N * 6 + (int64_t)i * 6);
}

// Far: enough fiber-tile x chunk blocks to fill the GPU four times over, at least 8
// sources each; near: N warps alone leave the GPU idle below a few thousand fibers,
// so segments of at least near_min sources.
static VelSplit velocity_split(int N, int fibers, int threads, int near_min) {
  VelSplit v;
  const int tiles = (int)ceil_div(N, fibers);
  v.chunks = std::max(1, std::min((int)ceil_div(148 * 4 * 4, tiles), (int)ceil_div(N, 8)));
  v.jchunk = (int)ceil_div(N, v.chunks);
  v.far_blocks = tiles * v.chunks;
  v.segs = std::max(1, std::min((int)ceil_div(148 * 16, N), (int)ceil_div(N, near_min)));
  v.jseg = (int)ceil_div(N, v.segs);
  v.near_blocks = (int)ceil_div((int64_t)N * v.segs, threads / 32);
  return v;
}
// A near source costs a warp Q points on ceil(Q / 32) points a lane, so with 48
// points (4 times the work of 24) a segment is 4 times shorter (30 fibers, all
// near: 66 us with 8 sources, 50 with 2).
static VelSplit numerical_split(int N, int Q) { return velocity_split(N, kVelFibers, kVelThreads, Q > 32 ? 2 : 8); }
static VelSplit analytical_split(int N) { return velocity_split(N, kAnaFibers, kAnaThreads, 8); }

// partial rows of either velocity path (vpart: this many rows of 6 N floats)
int velocity_rows(int N, int Q) {
  const VelSplit n = numerical_split(N, Q), a = analytical_split(N);
  return std::max(n.chunks + n.segs, a.chunks + a.segs);
}

int launch_velocity_analytical(const Tables& tab, int N, const float4* ori, const double4* pos64,
                               const double4* ori64, const float* x, float* vpart, float4* tvel, float4* rvel,
                               int* vflag, cudaStream_t st) {
  const VelSplit v = analytical_split(N);
  const unsigned nb = (unsigned)(v.far_blocks + v.near_blocks);
  bool done = false;
#define RF_VA_CASE(MM, QQ)                                                                              \
  if (!done && tab.M == MM && tab.Q == QQ) {                                                            \
    k_velocity_analytical<MM, QQ><<<nb, kAnaThreads, 0, st>>>(tab, N, pos64, ori64, x, v, vpart, vflag); \
    done = true;                                                                                        \
  }
  RF_FOR_EACH_MQ(RF_VA_CASE)
#undef RF_VA_CASE
  if (!done) {
    set_last_error_str("velocity: (M, Q) combination not instantiated");
    return RF_E_UNSUPPORTED;
  }
  RF_LAUNCH_CHECK();
  k_velocity_finalize<<<(unsigned)ceil_div(N, kVelSumFibers), kVelSumThreads, 0, st>>>(
      tab, N, ori, vpart, v.chunks + v.segs, tvel, rvel, vflag);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

int launch_velocity_numerical(const Tables& tab, int N, const double4* pos64, const float4* ori, const float* x,
                              float4* fw, float* vpart, float4* tvel, float4* rvel, int* vflag, cudaStream_t st) {
  const int Q = tab.Q;
  k_source_density<<<(unsigned)std::min<int64_t>(ceil_div((int64_t)N * (Q + kFarNodes), 256), 148 * 16), 256, 0, st>>>(
      tab, N, x, fw, vflag);
  RF_LAUNCH_CHECK();
  const VelSplit v = numerical_split(N, Q);
  const unsigned nb = (unsigned)(v.far_blocks + v.near_blocks);
  switch (Q) {
    case 12: k_velocity_numerical<12><<<nb, kVelThreads, 0, st>>>(tab, N, pos64, ori, fw, v, vpart); break;
    case 24: k_velocity_numerical<24><<<nb, kVelThreads, 0, st>>>(tab, N, pos64, ori, fw, v, vpart); break;
    case 48: k_velocity_numerical<48><<<nb, kVelThreads, 0, st>>>(tab, N, pos64, ori, fw, v, vpart); break;
    default: set_last_error_str("velocity: quadrature size not instantiated"); return RF_E_UNSUPPORTED;
  }
  RF_LAUNCH_CHECK();
  k_velocity_finalize<<<(unsigned)ceil_div(N, kVelSumFibers), kVelSumThreads, 0, st>>>(
      tab, N, ori, vpart, v.chunks + v.segs, tvel, rvel, vflag);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

// first != 0: x1 = x0 + dt U0, t1 = normalize(t0 + dt W0)
// otherwise: x^{n+1} = 4/3 x^n - 1/3 x^{n-1} + 2/3 dt (2 U^n - U^{n-1}), same for t, normalised.
// The state rotates in place (the reference swaps buffers, src/simulation.cu:
// 307-311): each fiber's previous state becomes its current one, the current
// one the new state, and the previous velocities the current ones, so the
// buffers a step reads and writes never change (one CUDA graph serves every
// step).
__global__ void k_update_fibers(int N, int first, double dt, double4* __restrict__ prev_pos,
                                double4* __restrict__ cur_pos, double4* __restrict__ prev_ori,
                                double4* __restrict__ cur_ori, float4* __restrict__ prev_tv,
                                const float4* __restrict__ cur_tv, float4* __restrict__ prev_rv,
                                const float4* __restrict__ cur_rv, float4* __restrict__ pos32,
                                float4* __restrict__ ori32, const int* __restrict__ halt) {
  if (halt != nullptr && *halt) return;   // the solve failed: the state stays as it is
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  update_fiber(i, first, dt, prev_pos, cur_pos, prev_ori, cur_ori, prev_tv, cur_tv[i], prev_rv, cur_rv[i], pos32,
               ori32);
}

int launch_update_fibers(int N, int first, double dt, double4* pp, double4* cp, double4* po, double4* co,
                         float4* ptv, const float4* ctv, float4* prv, const float4* crv, float4* pos32, float4* ori32,
                         const int* halt, cudaStream_t st) {
  k_update_fibers<<<(unsigned)ceil_div(N, 128), 128, 0, st>>>(N, first, dt, pp, cp, po, co, ptv, ctv, prv, crv, pos32,
                                                              ori32, halt);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

// ---- state and results across the bus ----------------------------------------
// The kernels read and write page-locked host memory themselves: one launch and
// one wait instead of a copy (staged by the driver, waited for) per array.  An
// element a thread, so a warp's host accesses are one contiguous run.
// Setting the state of 100 fibers took 34 us with six copies, reading it 34 us
// with two; 19 and 19 us so (4000 fibers: 85 and 98 us, now 31 and 35).

// host: n positions, then n orientations (3 doubles each), into fibers i0 .. i0 + n
__global__ void __launch_bounds__(256) k_state_in(const double* __restrict__ host, int n, int i0, double4* p0,
                                                  double4* p1, double4* o0, double4* o1, float4* p32, float4* o32) {
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (e >= 6 * n) return;
  const double v = host[e];
  const bool ori = e >= 3 * n;
  const int f = (ori ? e - 3 * n : e) / 3, a = (ori ? e - 3 * n : e) % 3;
  const int64_t at = 4 * (int64_t)(i0 + f) + a;
  double* d0 = reinterpret_cast<double*>(ori ? o0 : p0);
  double* d1 = reinterpret_cast<double*>(ori ? o1 : p1);
  float* d32 = reinterpret_cast<float*>(ori ? o32 : p32);
  d0[at] = d1[at] = v;
  d32[at] = (float)v;
  if (a == 2) {
    d0[at + 1] = d1[at + 1] = 0.0;
    d32[at + 1] = 0.f;
  }
}

// fibers i0 .. i0 + n of u, then of v, 3 doubles each, to host
template <typename T>
__global__ void __launch_bounds__(256) k_rows_out(const T* __restrict__ u, const T* __restrict__ v, int n, int i0,
                                                  double* __restrict__ host) {
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (e >= 6 * n) return;
  const int k = e >= 3 * n ? e - 3 * n : e;
  host[e] = (double)(e >= 3 * n ? v : u)[4 * (int64_t)(i0 + k / 3) + k % 3];
}

int launch_state_in(const double* host, int n, int i0, double4* p0, double4* p1, double4* o0, double4* o1, float4* p32,
                    float4* o32, cudaStream_t st) {
  k_state_in<<<(unsigned)ceil_div(6 * n, 256), 256, 0, st>>>(host, n, i0, p0, p1, o0, o1, p32, o32);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

int launch_rows_out(const double4* u, const double4* v, int n, int i0, double* host, cudaStream_t st) {
  k_rows_out<<<(unsigned)ceil_div(6 * n, 256), 256, 0, st>>>(reinterpret_cast<const double*>(u),
                                                             reinterpret_cast<const double*>(v), n, i0, host);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

int launch_rows_out(const float4* u, const float4* v, int n, int i0, double* host, cudaStream_t st) {
  k_rows_out<<<(unsigned)ceil_div(6 * n, 256), 256, 0, st>>>(reinterpret_cast<const float*>(u),
                                                             reinterpret_cast<const float*>(v), n, i0, host);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

}  // namespace rf
