// Near-field preconditioner of the stored mixed-precision modes (no reference
// counterpart: the reference's GMRES runs unpreconditioned).  For every fiber i
// and its k nearest neighbours by centre distance, the (k+1) x 15 rows of the
// system A = I + C T restricted to those fibers form a small dense block B_i
// (identity diagonal blocks, the stored FP32 pair blocks off the diagonal);
// the preconditioner keeps the 15 rows of B_i^-1 that belong to fiber i and
// applies them to the neighbourhood's entries of a vector (restricted additive
// Schwarz).  The solve uses it on the right, in flexible GMRES form: the
// matvec computes z_j = P v_j, stores z_j, and applies A to it; the solution
// update reads the stored z_j, so every convergence test still sees the true
// residual of A.  All sums run in a fixed order: results are reproducible.
//
// Storage read here: the FP32 record of the unordered pair (p, q), p < q, in
// assembly tiles of 8 fibers (I = p / 8 <= J = q / 8) grouped into storage
// tiles of 16: record ((L16 * 4 + sub) * 8 + q % 8) of NQ32 x 8 floats, value
// ((kI * M + kJ) * 6 + c) of pair p % 8 at [value][p % 8]; kI is p's force
// term, kJ q's, c the symmetric component (11, 22, 33, 12, 13, 23).
#include <algorithm>

#include "rf_common.cuh"
#include "rf_kernels.cuh"

namespace rf {
namespace {

constexpr int kNfM = 5;                       // force terms (the mixed modes' M)
constexpr int kNfM3 = 3 * kNfM;               // rows per fiber
constexpr int kNfNQ32 = (kNfM + 1) * (kNfM + 1) * 6;
constexpr int kNfStride = 16;                 // floats per column of a fiber's stored rows

// k nearest fibers of fiber i (centre distance, ties by index): nb[i][0] = i,
// nb[i][1..k] in order; slots past N - 1 neighbours (or without one: non-finite
// centres) hold i.  One warp per fiber: every lane keeps the nearest of its 32nd
// of the centres (streamed through shared memory), then k rounds take the warp's
// nearest head.  N=4000: 780 us with a thread per fiber.
constexpr int kNfWarps = 8;

__global__ void __launch_bounds__(kNfWarps * 32) k_nf_neighbours(const float4* __restrict__ pos, int N, int k,
                                                                 int* __restrict__ nb) {
  constexpr int kChunk = 1024;
  __shared__ float4 sp[kChunk];
  const int lane = threadIdx.x & 31;
  const int i = (int)blockIdx.x * kNfWarps + (int)(threadIdx.x >> 5);
  float bd[kNfMaxNeighbours];
  int bi[kNfMaxNeighbours];
#pragma unroll
  for (int s = 0; s < kNfMaxNeighbours; ++s) {
    bd[s] = 3.0e38f;
    bi[s] = -1;
  }
  const float4 pi = pos[min(i, N - 1)];
  for (int c0 = 0; c0 < N; c0 += kChunk) {
    const int cn = min(kChunk, N - c0);
    __syncthreads();
    for (int u = threadIdx.x; u < cn; u += blockDim.x) sp[u] = pos[c0 + u];
    __syncthreads();
    for (int u = lane; u < cn; u += 32) {
      const int j = c0 + u;
      const float dx = sp[u].x - pi.x, dy = sp[u].y - pi.y, dz = sp[u].z - pi.z;
      const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      if (j != i && d2 < bd[kNfMaxNeighbours - 1]) {
        // insertion into the sorted list (a lane meets its candidates in index order)
        float d = d2;
        int id = j;
#pragma unroll
        for (int t = 0; t < kNfMaxNeighbours; ++t) {
          if (d < bd[t]) {
            const float td = bd[t];
            const int ti = bi[t];
            bd[t] = d;
            bi[t] = id;
            d = td;
            id = ti;
          }
        }
      }
    }
  }
  if (i >= N) return;
  if (lane == 0) nb[(int64_t)i * (k + 1)] = i;
  for (int s = 0; s < k; ++s) {
    float d = bd[0];
    int id = bi[0];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float od = __shfl_xor_sync(0xffffffffu, d, o);
      const int oi = __shfl_xor_sync(0xffffffffu, id, o);
      if (oi >= 0 && (id < 0 || od < d || (od == d && oi < id))) {
        d = od;
        id = oi;
      }
    }
    if (lane == 0) nb[(int64_t)i * (k + 1) + 1 + s] = id >= 0 ? id : i;
    if (id >= 0 && bi[0] == id) {   // the lane that had it moves on
#pragma unroll
      for (int t = 0; t + 1 < kNfMaxNeighbours; ++t) {
        bd[t] = bd[t + 1];
        bi[t] = bi[t + 1];
      }
      bd[kNfMaxNeighbours - 1] = 3.0e38f;
      bi[kNfMaxNeighbours - 1] = -1;
    }
  }
}

// One CTA per fiber i: Gauss-Jordan elimination without row exchanges on
// [B_i^T | E] (E: the first 15 columns of the identity), so that the right
// part ends as the transpose of fiber i's rows of B_i^-1; those rows go to
// W[i] as [column c][row r] (kNfStride floats per column).  A pivot below
// 1e-6 in magnitude or a non-finite one leaves fiber i unpreconditioned (its
// rows of the identity).
//
// Thread = column, its n entries in registers.  A step needs one column of
// multipliers (published by its thread, read as 16-byte broadcasts) and one
// barrier; the rows rotate by one per step, so the pivot row is always entry 0,
// the loop over the steps is not unrolled and the register indexes are
// constants.  After n steps the rows are back in order.  N=4000, k = 4: 3.63 ms
// with the block in shared memory and a flat index over its entries.
template <int KK>
struct NfShape {
  static constexpr int n = (KK + 1) * kNfM3;               // rows of B_i
  static constexpr int NT = (n + kNfM3 + 1 + 31) / 32 * 32;   // columns of [B^T | E], one more for the padding
  static constexpr int n4 = (n + 3) / 4 * 4;
};

template <int KK>
__global__ void __launch_bounds__(NfShape<KK>::NT)
k_nf_setup(const Tables tab, int k, const float4* __restrict__ ori, const float* __restrict__ S32,
           const int* __restrict__ nb, float* __restrict__ W) {
  using S = NfShape<KK>;
  constexpr int n = S::n, n4 = S::n4;
  __shared__ __align__(16) float mult[2][n4];   // the pivot column, by turns
  const int i = blockIdx.x, c = threadIdx.x;
  float col[n4];                                // col[r] = [B^T | E][r][c]
#pragma unroll
  for (int r = 0; r < n4; ++r) col[r] = 0.f;
  if (c < n) {
    // row c of B: fiber a, term ka, component d.  B(row; column of fiber b, term kb,
    // component e) = delta when a == b, else [C_{a,ka} S^{ab}_{ka,kb}]_{d,e},
    // C_k(S) = k == 0 ? g t (t^T S) : g (S - E t (t^T S)); S the stored symmetric
    // block of the unordered pair (p, q), p < q (kp p's term): record
    // ((L16 * 4 + sub) * 8 + q % 8), value ((kp M + kq) 6 + component) of pair p % 8
    const int la = c / kNfM3, ka = (c % kNfM3) / 3, d = c % 3;
    const int a = nb[(int64_t)i * (k + 1) + la];
    const float4 t4 = ori[a];
    const float t3[3] = {t4.x, t4.y, t4.z};
    const float td = d == 0 ? t3[0] : d == 1 ? t3[1] : t3[2];
    const float g = tab.gamma[ka], E = tab.eigen[ka];
#pragma unroll
    for (int lb = 0; lb <= KK; ++lb) {
      const int b = nb[(int64_t)i * (k + 1) + lb];
      const int p = min(a, b), q = max(a, b);
      const int I = p / 8, J = q / 8;
      const int64_t L16 = (int64_t)(J / 2) * (J / 2 + 1) / 2 + I / 2;
      const int64_t rec = (L16 * 4 + (I % 2) * 2 + (J % 2)) * 8 + (q % 8);
      const float* base = S32 + rec * (kNfNQ32 * 8) + (p % 8);
#pragma unroll
      for (int kb = 0; kb < kNfM; ++kb) {
        float s[6];
#pragma unroll
        for (int e = 0; e < 6; ++e)
          s[e] = lb == la ? 0.f : base[((a < b ? ka * kNfM + kb : kb * kNfM + ka) * 6 + e) * 8];
        // rows of S and t^T S
        const float S3[3][3] = {{s[0], s[3], s[4]}, {s[3], s[1], s[5]}, {s[4], s[5], s[2]}};
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const float tS = fmaf(t3[2], S3[2][e], fmaf(t3[1], S3[1][e], t3[0] * S3[0][e]));
          const float Sde = d == 0 ? S3[0][e] : d == 1 ? S3[1][e] : S3[2][e];
          const float v = ka == 0 ? g * td * tS : g * (Sde - E * td * tS);
          col[lb * kNfM3 + kb * 3 + e] = lb == la ? (kb == ka && e == d ? 1.f : 0.f) : v;
        }
      }
    }
  } else {
    // column c - n of E
#pragma unroll
    for (int r = 0; r < kNfM3; ++r) col[r] = c - n == r ? 1.f : 0.f;
  }
  if (c == 0) {
#pragma unroll
    for (int r = 0; r < n4; r += 4)
      *reinterpret_cast<float4*>(&mult[0][r]) = make_float4(col[r], col[r + 1], col[r + 2], col[r + 3]);
  }
  __syncthreads();
  bool bad = false;
  for (int piv = 0; piv < n; ++piv) {
    const float* m = mult[piv & 1];
    const float p = m[0];
    if (!(fabsf(p) >= 1e-6f) || !isfinite(p)) {   // the same in every thread
      bad = true;
      break;
    }
    const float u = col[0] * (1.f / p);
#pragma unroll
    for (int r = 0; r < n; r += 4) {
      const float4 v = *reinterpret_cast<const float4*>(m + r);
      if (r > 0) col[r - 1] = fmaf(-v.x, u, col[r]);
      if (r + 1 < n) col[r] = fmaf(-v.y, u, col[r + 1]);
      if (r + 2 < n) col[r + 1] = fmaf(-v.z, u, col[r + 2]);
      if (r + 3 < n) col[r + 2] = fmaf(-v.w, u, col[r + 3]);
    }
    col[n - 1] = u;
    if (c == piv + 1) {
#pragma unroll
      for (int r = 0; r < n4; r += 4)
        *reinterpret_cast<float4*>(&mult[(piv + 1) & 1][r]) =
            make_float4(col[r], col[r + 1], col[r + 2], col[r + 3]);
    }
    __syncthreads();
  }
  // W[i][r][e] = (B^-1)[e][r] = X[r][e]: column n + e of the eliminated system
  const int e = c - n;
  if (e >= 0 && e < kNfStride) {
    float* wi = W + (size_t)i * (kNfMaxNeighbours + 1) * kNfM3 * kNfStride;
#pragma unroll
    for (int r = 0; r < n; ++r) wi[r * kNfStride + e] = e >= kNfM3 ? 0.f : bad ? (r == e ? 1.f : 0.f) : col[r];
  }
}

// z_i = W_i v[neighbourhood of i]; lane r < 15 of one warp per fiber forms row r
__global__ void __launch_bounds__(256) k_nf_apply(int N, int k, const int* __restrict__ nb,
                                                  const float* __restrict__ W, const float* __restrict__ v,
                                                  float* __restrict__ z, const int* __restrict__ skip) {
  if (skip != nullptr && *skip) return;
  const int lane = threadIdx.x & 31;
  const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  if (i >= N) return;
  const int kk = min(k, N - 1);
  const float* wi = W + (size_t)i * (kNfMaxNeighbours + 1) * kNfM3 * kNfStride;
  float acc = 0.f;
  for (int l = 0; l <= kk; ++l) {
    const int f = nb[(int64_t)i * (k + 1) + l];
    const float* vf = v + (int64_t)f * kNfM3;
    const float* wl = wi + (size_t)l * kNfM3 * kNfStride;
#pragma unroll
    for (int c = 0; c < kNfM3; ++c) acc = fmaf(wl[c * kNfStride + (lane & 15)], vf[c], acc);
  }
  if (lane < kNfM3) z[(int64_t)i * kNfM3 + lane] = acc;
}

}  // namespace

int64_t nf_w_floats(int N) { return (int64_t)N * (kNfMaxNeighbours + 1) * kNfM3 * kNfStride; }

int launch_nf_setup(const Tables& tab, int N, int k, const float4* pos, const float4* ori, const float* S32, int* nb,
                    float* W, cudaStream_t st) {
  if (tab.M != kNfM || k < 1 || k > kNfMaxNeighbours || N < 1) return RF_E_UNSUPPORTED;
  k_nf_neighbours<<<(unsigned)ceil_div(N, kNfWarps), kNfWarps * 32, 0, st>>>(pos, N, k, nb);
  RF_LAUNCH_CHECK();
  switch (std::min(k, N - 1)) {
#define RF_NF_CASE(KK)                                                                                     \
  case KK: k_nf_setup<KK><<<(unsigned)N, NfShape<KK>::NT, 0, st>>>(tab, k, ori, S32, nb, W); break;
    RF_NF_CASE(0) RF_NF_CASE(1) RF_NF_CASE(2) RF_NF_CASE(3) RF_NF_CASE(4)
    RF_NF_CASE(5) RF_NF_CASE(6) RF_NF_CASE(7) RF_NF_CASE(8)
#undef RF_NF_CASE
  }
  RF_LAUNCH_CHECK();
  return RF_OK;
}

int launch_nf_apply(int N, int k, const int* nb, const float* W, const float* v, float* z, const int* skip,
                    cudaStream_t st) {
  k_nf_apply<<<(unsigned)ceil_div((int64_t)N * 32, 256), 256, 0, st>>>(N, k, nb, W, v, z, skip);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

}  // namespace rf
