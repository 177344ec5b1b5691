// Packed solves of many small suspensions.  A thread-block cluster of C
// CTAs (C = 1, 2, 4 or 8, chosen per member by pack_plan_ctas) runs one
// suspension's whole mixed-precision GMRES-IR -- the algorithm rf_solve runs
// for RF_PREC_MIXED_*: restart cycles of up to m Arnoldi steps on the 16-bit
// pair blocks with FP32 sums, CGS2 with FP64 dot products, Givens rotations
// and the least-squares update in FP64, x in FP64, and the residual b - A x
// recomputed from the FP32 pair blocks with FP64 sums at every restart -- so
// an ensemble of small systems is solved by a few launches instead of several
// hundred per suspension.
//
// Work of a member is cut into kParts = 8 fixed parts whatever C is: storage
// tile L belongs to partition L mod 8, whose partial rows are summed in tile
// order; row slice s is fibers [s N / 8, (s + 1) N / 8), whose dot-product
// partial its owner's warps sum in a fixed order.  A CTA of the cluster owns
// 8 / C consecutive partitions and slices; the partitions' partial rows and the
// slices' partials are added in part order through distributed shared memory
// after a cluster barrier.  So a member's solution is the same bits for any C, alone
// and in any pack (it differs from rf_solve's in summation order only), and a
// pack can give its large members more SMs when the GPU has them to spare.
//
// Per Arnoldi step each CTA stages v in shared memory, walks its storage
// tiles (one thread per pair of a 16 x 16 tile, the records brought to shared
// memory by bulk copies one tile ahead), reduces z over the tile's lanes (halving
// exchanges) and adds the tile's partial rows into its partition's rows; the
// Krylov basis stays in the suspension's V (L2-resident at these sizes), each
// CTA writing its own rows of it.
#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include <cooperative_groups.h>

#include "rf_common.cuh"
#include "rf_kernels.cuh"
#include "rf_krylov.cuh"

namespace rf {
namespace cg = cooperative_groups;
namespace {

constexpr int kPT = 256;                              // threads per CTA
constexpr int kParts = 8;                             // tile partitions and row slices of a member
constexpr int kPM = 5;                                // force terms of the packed kernel
constexpr int kPM3 = 3 * kPM;
constexpr int kNW = s16_record_words(kPM);            // 16-bit record words per pair
constexpr int kNQ32 = (kPM + 1) * (kPM + 1) * 6;      // FP32 values per pair
constexpr int kTileDoubles = 8 * 16 * 16 + 16 * 16;   // a tile's partial sums (i side, j side)
static_assert(kTileDoubles >= 8 * 80, "the warp partials of one slice at the longest restart");
constexpr int kRecU = kNW / 4;                        // 16-byte units of a pair's 16-bit record
constexpr int kWarpU = 32 * kRecU;                    // units of a warp's 32 records of a tile
static_assert(kNW % 4 == 0 && kRecU % 2 == 1, "16-byte reads of eight consecutive records hit different banks");

// Shared memory offsets: the 16-bit products' sums are FP32, so the records are
// staged from the upper half of the partition rows on, and past their end where
// the rows are short.
__host__ __device__ __forceinline__ int pack_stage_offset(int Rmax, int slots) {   // in 16-byte units
  return ((2 + slots) * Rmax + 3) / 4;
}
__host__ __device__ __forceinline__ int pack_tail_offset(int Rmax, int slots) {    // in doubles
  const int rows = (1 + slots) * Rmax, staged = 2 * (pack_stage_offset(Rmax, slots) + kPT / 32 * kWarpU);
  return rows > staged ? rows : staged;
}

__device__ __forceinline__ uint32_t psmem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Wait for an mbarrier's phase.  Past limit_ns (0: at once) *late is set, and the
// wait goes on for a second, so that the copy does not land on what comes next.
constexpr uint64_t kPackDrainNs = 1000000000ull;
__device__ __forceinline__ void pack_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns, int* late) {
  uint64_t t0 = 0, now, left = limit_ns;
  bool over = false;
  for (int n = 0;; ++n) {
    if (left == 0) {
      if (over) return;
      over = true;
      *late = 1;   // every writer stores the same value
      left = kPackDrainNs;
      t0 = 0;
    }
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(psmem(bar)), "r"(parity)
        : "memory");
    if (done) return;
    if ((n & 63) == 63) {
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      if (now - t0 > left) left = 0;
    }
  }
}

template <typename T>
__device__ __forceinline__ T pshfl(T v, int m) {
  return __shfl_xor_sync(0xffffffffu, v, m);
}

__device__ __forceinline__ float pfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double pfma(double a, double b, double c) { return fma(a, b, c); }

// acc += sym(t) v, t = (t00, t11, t22, t01, t02, t12)
template <typename T>
__device__ __forceinline__ void psym(const T (&t)[6], const T* v, T* acc) {
  acc[0] = pfma(t[4], v[2], pfma(t[3], v[1], pfma(t[0], v[0], acc[0])));
  acc[1] = pfma(t[5], v[2], pfma(t[1], v[1], pfma(t[3], v[0], acc[1])));
  acc[2] = pfma(t[2], v[2], pfma(t[5], v[1], pfma(t[4], v[0], acc[2])));
}

// v[G], G = 4, 8 or 16, summed over the 16 lanes that differ in lane bits 0..3 by
// halving exchanges (then plain ones); lane l gets the sum of v[(l & 15) / (16 / G)].
// The lanes are added in the same order for every G.
template <int H, int O, typename T, int G>
__device__ __forceinline__ void psum_step(T (&a)[G], int lane) {
  if constexpr (O > 0) {
    if constexpr (H > 0) {
      const bool up = lane & O;
#pragma unroll
      for (int k = 0; k < H; ++k) {
        const T s = up ? a[k] : a[k + H], kp = up ? a[k + H] : a[k];
        a[k] = kp + pshfl(s, O);
      }
    } else {
      a[0] += pshfl(a[0], O);
    }
    psum_step<H / 2, O / 2>(a, lane);
  }
}
template <typename T, int G>
__device__ __forceinline__ T psum(const T (&v)[G], int lane) {
  T a[G];
#pragma unroll
  for (int k = 0; k < G; ++k) a[k] = v[k];
  psum_step<G / 2, 8>(a, lane);
  return a[0];
}

template <typename H16>
__device__ __forceinline__ float2 punpack(uint32_t w) {
  if constexpr (std::is_same<H16, __half>::value) return __half22float2(*reinterpret_cast<const __half2*>(&w));
  else return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
}

// z_i += T x_j, z_j += T^T x_i over the 25 blocks of one pair record
template <typename H16>
__device__ __forceinline__ void ppair16(const uint32_t (&w)[kNW], const float (&xi)[kPM3], const float (&xj)[kPM3],
                                        float (&zi)[16], float (&zj)[16]) {
#pragma unroll
  for (int kI = 0; kI < kPM; ++kI)
#pragma unroll
    for (int kJ = 0; kJ < kPM; ++kJ) {
      const int blk = kI * kPM + kJ;
      float tv[6];
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        const float2 f = punpack<H16>(w[3 * blk + h]);
        tv[2 * h] = f.x;
        tv[2 * h + 1] = f.y;
      }
      psym(tv, xj + 3 * kJ, zi + 3 * kI);
      psym(tv, xi + 3 * kI, zj + 3 * kJ);
    }
}

// Shared memory (doubles): [staged vector Rmax][partition rows: 8/C x Rmax, or
// FP32 rows and a tile's records][i-side tile partials 8 x 16 x 16][j-side tile
// sums 16 x 16][H: column j of j + 2 entries]
// [cs m][sn m][g m+1][y m][h m+1][h2 m+2][slice partials 3 x 8 x (m+2)]
// [scalar 2][flags]; the dot products' warp partials use the tile sums' room
// kClustered: launched with clusters of 2, 4 or 8 CTAs; otherwise one CTA per
// member (the same arithmetic in the same order, without cluster barriers and
// distributed shared memory)
template <bool kClustered>
__global__ void __launch_bounds__(kPT) k_pack_gmres_ir(const PackMember* __restrict__ members, int Rmax, int m) {
  extern __shared__ __align__(16) unsigned char psm[];
  int C = 1, rank = 0;
  if constexpr (kClustered) {
    C = (int)cg::this_cluster().num_blocks();
    rank = (int)cg::this_cluster().block_rank();
  }
  const PackMember& P = members[blockIdx.x / C];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int N = P.N;
  const int R = kPM3 * N;
  const int T16 = (N + 15) / 16;
  const int ntiles = T16 * (T16 + 1) / 2;
  const int spc = kParts / C;                                   // partitions (and row slices) per CTA
  const int p0 = rank * spc;                                    // this CTA's first partition
  const int q0 = kPM3 * ((rank * N) / C), q1 = kPM3 * (((rank + 1) * N) / C);   // its rows
  double* sxd = reinterpret_cast<double*>(psm);
  float* sxf = reinterpret_cast<float*>(psm);
  double* zpd = sxd + Rmax;                                     // partition rows, slot stride Rmax
  float* zpf = reinterpret_cast<float*>(zpd);
  double* tail = sxd + pack_tail_offset(Rmax, spc);
  double (*zip)[16][16] = reinterpret_cast<double (*)[16][16]>(tail);
  float (*zipf)[16][16] = reinterpret_cast<float (*)[16][16]>(tail);
  double (*zjs)[16] = reinterpret_cast<double (*)[16]>(tail + 8 * 16 * 16);
  float (*zjsf)[16] = reinterpret_cast<float (*)[16]>(tail + 8 * 16 * 16);
  double* H = tail + kTileDoubles;
  double* cs = H + m * (m + 3) / 2;
  double* sn = cs + m;
  double* g = sn + m;
  double* yv = g + m + 1;
  double* hh = yv + m;
  double* hh2 = hh + m + 1;                                     // m + 2: dots and the norm
  double* dpart = hh2 + m + 2;                                  // [3][kParts][m+2]
  double* red = tail;                                           // warp partials, outside the products
  double* scal = dpart + 3 * kParts * (m + 2);
  // [0] cycle done, [2] non-finite, [3] a wait for records of a product gave up ([1]: of one not wanted)
  int* flags = reinterpret_cast<int*>(scal + 2);
  float* V = P.V;
  const int64_t ldv = P.ldv;
  const int i16 = t & 15, j16 = t >> 4;
  const int sub = (i16 >> 3) * 2 + (j16 >> 3);
  // a warp's pairs (16 i, 2 j) are two runs of 16 records of a storage tile
  uint4* stage = reinterpret_cast<uint4*>(psm) + pack_stage_offset(Rmax, spc) + warp * kWarpU;
  const uint4* mine = stage + ((i16 >> 3) * 16 + (j16 & 1) * 8 + (i16 & 7)) * kRecU;
  const int rec32 = sub * 8 + (j16 & 7);                       // FP32 record (8 pairs, [value][i])
  __shared__ uint64_t copied[kPT / 32];                        // a warp's records have arrived
  if (t < kPT / 32) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(psmem(&copied[t])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (t == 0) flags[3] = 0;
  __syncthreads();
  uint32_t phase = 0;                                          // of this warp's copies
  int rb = 0;                                                  // reduction buffer in use (of 3)
  // a cluster barrier, or the block barrier when the member has one CTA
  auto csync = [&]() {
    if constexpr (kClustered) cg::this_cluster().sync();
    else __syncthreads();
  };
  // a pointer into CTA r's shared memory at the offset of p in this CTA's
  auto at_rank = [&](auto* p, int r) {
    if constexpr (kClustered) return cg::this_cluster().map_shared_rank(p, r);
    else return p;
  };

  // out[k] = sum over the member's rows of a[r] * V_k[r] for k < nv, FP64, and with
  // `norm` out[nv] = sum of a[r]^2.  A slice's partial is that of nvw virtual warps
  // (1 up to 32 fibers, 8 from 233 on: at most two rows a lane): lane l of virtual
  // warp w adds rows 32 w + l and 32 (w + nvw) + l of the slice, the lanes meet in
  // halving exchanges, the virtual warps add in order; the CTA's warps share all
  // its slices' virtual warps.  4, 8 or 16 values at a time (32 fibers: 1.8k cycles
  // a call with 16 for any number, of which most cycles hold few values).  The
  // partials go into the owning CTA's buffer; after the cluster barrier every CTA
  // adds the 8 of them in slice order.  Three buffers in turn: a buffer is written
  // again only after two more cluster barriers, when every CTA has read it.
  const int nvw = min(8, (kPM3 * ((N + kParts - 1) / kParts) + 63) / 64);
  auto cdots = [&](const float* a, int nv, bool norm, double* out) {
    __syncthreads();                                           // this CTA's rows of a are written
    double* part = dpart + (size_t)rb * kParts * (m + 2);
    const int n = nv + (norm ? 1 : 0);
    const int npad = (n + 15) / 16 * 16;
    const int per = min(spc, kTileDoubles / (nvw * npad));     // slices whose warp partials fit at once
    for (int s0 = 0; s0 < spc; s0 += per) {
      const int cnt = min(per, spc - s0);
      for (int e = warp; e < cnt * nvw; e += kPT / 32) {
        const int s = p0 + s0 + e / nvw;
        const int r0 = kPM3 * ((s * N) / kParts), r1 = kPM3 * (((s + 1) * N) / kParts);
        // G values from g on, of this virtual warp's rows of the slice
        auto values = [&](auto width, int g) {
          constexpr int G = decltype(width)::value;
          double acc[G];
#pragma unroll
          for (int u = 0; u < G; ++u) acc[u] = 0.0;
          for (int r = r0 + (e % nvw) * 32 + lane; r < r1; r += nvw * 32) {
            const float af = a[r];
            const double ar = (double)af;
            float v[G];
#pragma unroll
            for (int u = 0; u < G; ++u) {
              const int k = g + u;
              v[u] = k < nv ? V[(int64_t)k * ldv + r] : k < n ? af : 0.f;
            }
#pragma unroll
            for (int u = 0; u < G; ++u) acc[u] = fma(ar, (double)v[u], acc[u]);
          }
          double v = psum(acc, lane);
          v += pshfl(v, 16);
          const int k = g + lane / (16 / G);
          if (lane < 16 && lane % (16 / G) == 0 && k < n) {
            if (nvw == 1) part[s * (m + 2) + k] = v;
            else red[(size_t)e * npad + k] = v;
          }
        };
        if (n <= 4) values(std::integral_constant<int, 4>(), 0);
        else if (n <= 8) values(std::integral_constant<int, 8>(), 0);
        else
          for (int g = 0; g < npad; g += 16) values(std::integral_constant<int, 16>(), g);
      }
      if (nvw == 1) continue;   // a slice is one virtual warp
      __syncthreads();
      for (int e = t; e < cnt * n; e += kPT) {
        const int sl = e / n, k = e % n;
        const double* rp = red + (size_t)sl * nvw * npad + k;
        double v = rp[0];
        for (int w = 1; w < nvw; ++w) v += rp[w * npad];
        part[(p0 + s0 + sl) * (m + 2) + k] = v;
      }
      __syncthreads();
    }
    csync();
    for (int k = t; k < n; k += kPT) {
      double sum = 0.0;
#pragma unroll
      for (int s = 0; s < kParts; ++s) sum += at_rank(part, s / spc)[s * (m + 2) + k];
      out[k] = sum;
    }
    __syncthreads();
    rb = rb == 2 ? 0 : rb + 1;
  };
  // sum of a[r]^2
  auto sumsq = [&](const float* a) -> double {
    cdots(a, 0, true, scal);
    return scal[0];
  };
  // this CTA's next storage tile after L, in tile order: partitions p0 .. p0 + spc - 1
  auto next_own = [&](int L) {
    const int p = (L + 1) % kParts;
    return p >= p0 && p < p0 + spc ? L + 1 : L + 1 + (p0 - p + kParts) % kParts;
  };
  // this warp's records of storage tile L into its part of the stage
  auto fetch = [&](int L) {
    if (lane < 2) {
      constexpr uint32_t bytes = 16 * kRecU * 16;
      const int rec = ((lane * 2 + (warp >> 2)) * 8 + ((2 * warp) & 7)) * 8;
      asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(psmem(&copied[warp])), "r"(bytes)
                   : "memory");
      asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       psmem(stage + lane * 16 * kRecU)),
                   "l"(reinterpret_cast<const uint4*>(P.S16) + ((int64_t)L * 256 + rec) * kRecU), "r"(bytes),
                   "r"(psmem(&copied[warp]))
                   : "memory");
    }
    __syncwarp();
    if (lane == 0)
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(psmem(&copied[warp])) : "memory");
  };
  // a member's vector into shared memory, 8 loads in flight
  auto copy_in = [&](auto* dst, const auto* src) {
    for (int r0 = t; r0 < R; r0 += 8 * kPT) {
      std::remove_reference_t<decltype(*dst)> v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = r0 + u * kPT < R ? src[r0 + u * kPT] : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (r0 + u * kPT < R) dst[r0 + u * kPT] = v[u];
    }
  };
  // v into shared memory, this CTA's rows of T v cleared and the first tile's
  // records on their way; meanwhile one thread runs `aside`
  auto stage_vector = [&](const float* v, auto&& aside) {
    if (p0 < ntiles) fetch(p0);
    csync();                                                   // every CTA's rows of v are written
    if (t == kPT - 1) aside();
    copy_in(sxf, v);
    for (int q = t; q < spc * Rmax; q += kPT) zpf[q] = 0.f;
    __syncthreads();
  };
  // the staged product is not wanted: the records that were fetched must still
  // arrive before their room is used again or the CTA ends
  auto unstage = [&]() {
    if (p0 < ntiles) {
      pack_wait(&copied[warp], phase, kPackDrainNs, &flags[1]);
      phase ^= 1;
    }
  };
  // w = v + C (T v) of the staged v with the 16-bit blocks, FP32 sums; this CTA
  // writes its rows of w
  //
  // A thread reading its pair's 304-byte record from memory puts 32 cache lines
  // behind each of a warp's 19 loads: 7.4k cycles a tile of 256 pairs, against
  // ~2.4k of arithmetic.  The warp's records are two contiguous runs, so two bulk
  // copies bring the next tile's to shared memory as soon as this one's are in
  // registers (16-byte reads 19 units apart: no bank conflicts): 4.2k cycles.
  // The same through 16-byte asynchronous copies: 6.9k, their issue alone 2.8k.
  auto matvec16 = [&](float* w) {
    int L = p0, I = p0, J = 0;
    while (L < ntiles) {
      float* zs = zpf + (size_t)(L % kParts - p0) * Rmax;
      while (I > J) I -= ++J;   // storage tile L = J (J + 1) / 2 + I
      const int i = I * 16 + i16, j = J * 16 + j16;
      pack_wait(&copied[warp], phase, P.wait_ns, &flags[3]);
      phase ^= 1;
      uint32_t wv[kNW];
#pragma unroll
      for (int u = 0; u < kRecU; ++u) {
        const uint4 q4 = mine[u];
        wv[4 * u] = q4.x; wv[4 * u + 1] = q4.y; wv[4 * u + 2] = q4.z; wv[4 * u + 3] = q4.w;
      }
      __syncwarp();
      const int Ln = next_own(L);
      if (Ln < ntiles) fetch(Ln);
      float zi[16], zj[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) zi[q] = zj[q] = 0.f;
      if (i < j && j < N) {
        float xi[kPM3], xj[kPM3];
#pragma unroll
        for (int q = 0; q < kPM3; ++q) {
          xi[q] = sxf[i * kPM3 + q];
          xj[q] = sxf[j * kPM3 + q];
        }
        if (P.smode == 2) ppair16<__nv_bfloat16>(wv, xi, xj, zi, zj);
        else ppair16<__half>(wv, xi, xj, zi, zj);
      }
      const float sj = psum(zj, lane);   // z_j over this half-warp's 16 i
      const bool b4 = lane & 16;
      float u8[8];                          // z_i over this warp's two j: one halving exchange
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float s = b4 ? zi[k] : zi[k + 8], kp = b4 ? zi[k + 8] : zi[k];
        u8[k] = kp + pshfl(s, 16);
      }
      __syncthreads();   // the previous tile's sums have been read
      zjsf[j16][lane & 15] = sj;
#pragma unroll
      for (int k = 0; k < 8; ++k) zipf[warp][i16][8 * (b4 ? 1 : 0) + k] = u8[k];
      __syncthreads();
      if (t < 16 * kPM3) {
        const int f = t / kPM3, q = t % kPM3;
        float s8[8];
#pragma unroll
        for (int w8 = 0; w8 < 8; ++w8) s8[w8] = zipf[w8][f][q];
        const float si = ((s8[0] + s8[1]) + (s8[2] + s8[3])) + ((s8[4] + s8[5]) + (s8[6] + s8[7]));
        const int fi = I * 16 + f, fj = J * 16 + f;
        if (fi < N) zs[fi * kPM3 + q] += si;
        if (fj < N) zs[fj * kPM3 + q] += zjsf[f][q];
      }
      I += Ln - L;
      L = Ln;
    }
    csync();                                                   // every partition's rows are complete
    const bool late = flags[3] != 0;                           // the solve ends as non-finite, in every CTA
    for (int u = t; u < (q1 - q0) / 3; u += kPT) {
      const int r0 = q0 + 3 * u, i = r0 / kPM3, k = (r0 % kPM3) / 3;
      float z3[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int p = 0; p < kParts; ++p) {
        const float* zr = at_rank(zpf, p / spc) + (size_t)(p % spc) * Rmax + r0;
        z3[0] += zr[0];
        z3[1] += zr[1];
        z3[2] += zr[2];
      }
      const float4 o = P.ori[i];
      const float t3[3] = {o.x, o.y, o.z};
      const float tz = t3[0] * z3[0] + t3[1] * z3[1] + t3[2] * z3[2];
      const float coef = P.coef[k], E = P.eig[k];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float cz = k == 0 ? coef * t3[a] * tz : coef * (z3[a] - E * t3[a] * tz);
        w[r0 + a] = late ? nanf("") : sxf[r0 + a] + cz;
      }
    }
  };
  // r = b - (x + C (T x)) with the FP32 blocks, x and sums in FP64; this CTA writes its rows of r
  auto residual64 = [&](float* r) {
    for (int q = t; q < spc * Rmax; q += kPT) zpd[q] = 0.0;
    csync();                                                   // every CTA's rows of x are written
    copy_in(sxd, static_cast<const double*>(P.x64));
    __syncthreads();
    int I = p0, J = 0;
    for (int L = p0; L < ntiles;) {
      double* zs = zpd + (size_t)(L % kParts - p0) * Rmax;
      while (I > J) I -= ++J;
      const int i = I * 16 + i16, j = J * 16 + j16;
      double zi[16], zj[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) zi[q] = zj[q] = 0.0;
      if (i < j && j < N) {
        const float* base = P.S32 + ((int64_t)L * 32 + rec32) * (kNQ32 * 8) + (i16 & 7);
        const double* xi = sxd + i * kPM3;
        const double* xj = sxd + j * kPM3;
        // a row of blocks (30 loads) on its way while the one before is summed
        float next[6 * kPM];
#pragma unroll
        for (int c = 0; c < 6 * kPM; ++c) next[c] = base[c * 8];
#pragma unroll
        for (int kI = 0; kI < kPM; ++kI) {
          float row[6 * kPM];
#pragma unroll
          for (int c = 0; c < 6 * kPM; ++c) row[c] = next[c];
          if (kI + 1 < kPM) {
#pragma unroll
            for (int c = 0; c < 6 * kPM; ++c) next[c] = base[((kI + 1) * 6 * kPM + c) * 8];
          }
#pragma unroll
          for (int kJ = 0; kJ < kPM; ++kJ) {
            double tv[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) tv[c] = (double)row[6 * kJ + c];
            psym(tv, xj + 3 * kJ, zi + 3 * kI);
            psym(tv, xi + 3 * kI, zj + 3 * kJ);
          }
        }
      }
      const double sj = psum(zj, lane);
      const bool b4 = lane & 16;
      double u8[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double s = b4 ? zi[k] : zi[k + 8], kp = b4 ? zi[k + 8] : zi[k];
        u8[k] = kp + pshfl(s, 16);
      }
      __syncthreads();
      zjs[j16][lane & 15] = sj;
#pragma unroll
      for (int k = 0; k < 8; ++k) zip[warp][i16][8 * (b4 ? 1 : 0) + k] = u8[k];
      __syncthreads();
      if (t < 16 * kPM3) {
        const int f = t / kPM3, q = t % kPM3;
        double s8[8];
#pragma unroll
        for (int w8 = 0; w8 < 8; ++w8) s8[w8] = zip[w8][f][q];
        const double si = ((s8[0] + s8[1]) + (s8[2] + s8[3])) + ((s8[4] + s8[5]) + (s8[6] + s8[7]));
        const int fi = I * 16 + f, fj = J * 16 + f;
        if (fi < N) zs[fi * kPM3 + q] += si;
        if (fj < N) zs[fj * kPM3 + q] += zjs[f][q];
      }
      const int Ln = next_own(L);
      I += Ln - L;
      L = Ln;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the next records land on these rows
    csync();
    for (int u = t; u < (q1 - q0) / 3; u += kPT) {
      const int r0 = q0 + 3 * u, i = r0 / kPM3, k = (r0 % kPM3) / 3;
      double z3[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int p = 0; p < kParts; ++p) {
        const double* zr = at_rank(zpd, p / spc) + (size_t)(p % spc) * Rmax + r0;
        z3[0] += zr[0];
        z3[1] += zr[1];
        z3[2] += zr[2];
      }
      const float4 o = P.ori[i];
      const double t3[3] = {(double)o.x, (double)o.y, (double)o.z};
      const double tz = t3[0] * z3[0] + t3[1] * z3[1] + t3[2] * z3[2];
      const double coef = (double)P.coef[k], E = (double)P.eig[k];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double cz = k == 0 ? coef * t3[a] * tz : coef * (z3[a] - E * t3[a] * tz);
        const double yr = sxd[r0 + a] + cz;
        r[r0 + a] = (float)((double)P.b[r0 + a] - yr);
      }
    }
  };

  for (int q = q0 + t; q < q1; q += kPT) P.x64[q] = 0.0;
  const double bnorm = sqrt(sumsq(P.b));
  const double tol = P.tol * bnorm;
  int total = 0, restarts = 0, refinements = 0, status = 0;
  double beta = bnorm;
  bool conv = bnorm == 0.0, bad = !isfinite(bnorm);
  float* V0 = V;
  for (int cycle = 0; !conv && !bad; ++cycle) {
    if (cycle == 0) {
      for (int q = q0 + t; q < q1; q += kPT) V0[q] = P.b[q];
    } else {
      residual64(V0);
      ++refinements;
    }
    beta = sqrt(sumsq(V0));
    conv = beta <= tol;
    bad = !isfinite(beta);
    if (conv || bad || total >= P.maxit) break;
    const float inv = (float)(1.0 / beta);
    for (int q = q0 + t; q < q1; q += kPT) V0[q] *= inv;
    if (t == 0) {
      g[0] = beta;
      for (int k = 1; k <= m; ++k) g[k] = 0.0;
    }
    __syncthreads();
    int jc = 0;
    double nrm = 0.0;
    // column j's rotation and the decision to stop, by one thread: the same
    // values in every CTA of the cluster, so the same decisions
    auto rotate = [&](int j) {
      double* Hc = H + j * (j + 3) / 2;
      for (int k = 0; k <= j; ++k) Hc[k] = hh[k] + hh2[k];
      for (int k = 0; k < j; ++k) {
        const double x0 = Hc[k], x1 = Hc[k + 1];
        Hc[k] = cs[k] * x0 + sn[k] * x1;
        Hc[k + 1] = -sn[k] * x0 + cs[k] * x1;
      }
      const double x0 = Hc[j], x1 = nrm;
      const double rr = hypot(x0, x1);
      const double c = rr > 0.0 ? x0 / rr : 1.0, s = rr > 0.0 ? x1 / rr : 0.0;
      cs[j] = c;
      sn[j] = s;
      Hc[j] = rr;
      g[j + 1] = -s * g[j];
      g[j] = c * g[j];
      const double est = fabs(g[j + 1]);
      const bool nf = !isfinite(est);
      flags[2] = nf ? 1 : 0;
      flags[0] = (nf || est <= tol || j + 1 >= m || total >= P.maxit || nrm == 0.0) ? 1 : 0;
    };
    for (;;) {
      // the last column's rotation runs beside the staging of the next product
      stage_vector(V + (int64_t)jc * ldv, [&]() {
        if (jc > 0) rotate(jc - 1);
      });
      if (jc > 0) {
        bad = flags[2];
        if (flags[0]) {
          unstage();
          break;
        }
      }
      float* w = V + (int64_t)(jc + 1) * ldv;
      matvec16(w);
      const int nv = jc + 1;
      cdots(w, nv, false, hh);
      for (int q = q0 + t; q < q1; q += kPT) {
        double s = (double)w[q];
        for (int k = 0; k < nv; ++k) s -= hh[k] * (double)V[(int64_t)k * ldv + q];
        w[q] = (float)s;
      }
      // ||w|| after the second pass is ||w'||^2 - sum h2^2 from that pass's own
      // sums, from the entries when that cancels (the same in every CTA)
      cdots(w, nv, true, hh2);
      double nrm2 = hh2[nv];
      const double ww = nrm2;
      for (int k = 0; k < nv; ++k) nrm2 = fma(-hh2[k], hh2[k], nrm2);
      const bool direct = nrm2 > 1e-3 * ww && isfinite(nrm2);
      nrm = sqrt(nrm2);
      const float sc = direct ? (float)(1.0 / nrm) : 1.f;
      for (int q = q0 + t; q < q1; q += kPT) {
        double s = (double)w[q];
        for (int k = 0; k < nv; ++k) s -= hh2[k] * (double)V[(int64_t)k * ldv + q];
        w[q] = (float)s * sc;
      }
      if (!direct) {
        nrm2 = sumsq(w);
        nrm = sqrt(nrm2);
        if (nrm2 > 0.0 && isfinite(nrm2)) {
          const float winv = (float)(1.0 / nrm);
          for (int q = q0 + t; q < q1; q += kPT) w[q] *= winv;
        }
      }
      ++total;
      ++jc;
    }
    if (bad) break;
    // x += V y, H y = g (upper triangular, jc x jc)
    if (t == 0) {
      for (int i = jc - 1; i >= 0; --i) {
        double s = g[i];
        for (int k = i + 1; k < jc; ++k) s -= H[k * (k + 3) / 2 + i] * yv[k];
        yv[i] = s / H[i * (i + 3) / 2 + i];
      }
    }
    __syncthreads();
    for (int q = q0 + t; q < q1; q += kPT) {
      double s = 0.0;
      for (int k = 0; k < jc; ++k) s += yv[k] * (double)V[(int64_t)k * ldv + q];
      P.x64[q] += s;
    }
    ++restarts;
  }
  status = bad ? 2 : (conv ? 0 : 1);
  if (bad && rank == 0 && t == 0)
    for (int r = 0; r < C; ++r)
      if (at_rank(flags, r)[3]) status = 3;
  for (int q = q0 + t; q < q1; q += kPT) P.x[q] = (float)P.x64[q];
  if (rank == 0 && t == 0) {
    P.out[0] = total;
    P.out[1] = restarts;
    P.out[2] = refinements;
    P.out[3] = status;
    P.relres[0] = bnorm > 0.0 ? beta / bnorm : 0.0;
  }
  csync();   // the other CTAs may still read this CTA's shared memory
}

}  // namespace

void pack_plan_ctas(const int* fibers, int n, int sms, int* ctas, int max_cluster) {
  int total = 0;
  for (int i = 0; i < n; ++i) {
    ctas[i] = fibers[i] > kPackSingleMaxFibers ? 2 : 1;
    total += ctas[i];
  }
  for (;;) {
    int best = -1;
    double most = 0.0;
    for (int i = 0; i < n; ++i) {
      const int T = (fibers[i] + 15) / 16, tiles = T * (T + 1) / 2;
      if (2 * ctas[i] > max_cluster || tiles < 4 * ctas[i]) continue;   // at least two tiles per CTA after doubling
      const double w = (double)tiles / ctas[i];
      if (w > most) {
        most = w;
        best = i;
      }
    }
    if (best < 0 || total + ctas[best] > sms) break;
    total += ctas[best];
    ctas[best] *= 2;
  }
}

size_t pack_smem_bytes(int Rmax, int m, int csize) {
  const size_t slots = (size_t)(kParts / csize);
  const size_t doubles = (size_t)pack_tail_offset(Rmax, (int)slots) + kTileDoubles + (size_t)(m * (m + 3) / 2) +
                         2 * (size_t)m +
                         (size_t)(m + 1) + (size_t)m + (size_t)(m + 1) + (size_t)(m + 2) +
                         3 * kParts * (size_t)(m + 2) + 2;
  return doubles * sizeof(double) + 4 * sizeof(int);
}

int pack_max_cluster() {
  // one query per device and cluster size with the largest shared memory a
  // pack can ask for (kPackMaxFibers rows, restart kMaxRestart): smaller packs
  // fit wherever it does.  The answer is the largest C with every size from 2
  // to C schedulable.
  static std::mutex mu;
  static std::map<int, int> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  std::lock_guard<std::mutex> lk(mu);
  auto it = known.find(dev);
  if (it != known.end()) return it->second;
  int best = 1;
  for (int c = 2; c <= kParts && best == c / 2; c *= 2) {
    const size_t smem = pack_smem_bytes(kPM3 * kPackMaxFibers, kMaxRestart, c);
    if (cudaFuncSetAttribute(k_pack_gmres_ir<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      break;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3(kPT);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_pack_gmres_ir<true>, &cfg) == cudaSuccess && clusters > 0)
      best = c;
  }
  cudaGetLastError();   // a refused query leaves no error behind
  known[dev] = best;
  return best;
}

void pack_lanes_release(PackLanes& l) {
  for (auto& s : l.aux)
    if (s) cudaStreamDestroy(s), s = nullptr;
  for (auto& e : l.join)
    if (e) cudaEventDestroy(e), e = nullptr;
  if (l.fork) cudaEventDestroy(l.fork), l.fork = nullptr;
}

int launch_pack_gmres_ir(const PackMember* members, const int (&counts)[4], const int (&rmax)[4], int m,
                         cudaStream_t st, PackLanes& lanes) {
  int n = 0;
  bool sizes_ok = m >= 1 && m <= kMaxRestart;
  size_t smax = 0;
  for (int c = 0; c < 4; ++c) {
    if (counts[c] < 0) sizes_ok = false;
    if (counts[c] <= 0) continue;
    n += counts[c];
    // one CTA holds all 8 partitions' rows: at most kPackSingleMaxFibers fibers
    const int limit = kPM3 * (c == 3 ? kPackSingleMaxFibers : kPackMaxFibers);
    if (rmax[c] < 1 || rmax[c] > limit) sizes_ok = false;
    else smax = std::max(smax, pack_smem_bytes(rmax[c], m, kParts >> c));
  }
  if (n < 1 || !sizes_ok) {
    set_last_error_str("packed solve: bad sizes");
    return RF_E_INPUT;
  }
  RF_CUDA_TRY(cudaFuncSetAttribute(k_pack_gmres_ir<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smax));
  RF_CUDA_TRY(cudaFuncSetAttribute(k_pack_gmres_ir<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smax));
  // one launch per cluster size, the largest first; the classes after the
  // first on their own streams, forked from st before the first launch, so
  // that they run beside it
  int classes = 0;
  for (int c = 0; c < 4; ++c) classes += counts[c] > 0 ? 1 : 0;
  if (classes > 1) {
    if (!lanes.fork) RF_CUDA_TRY(cudaEventCreateWithFlags(&lanes.fork, cudaEventDisableTiming));
    for (int k = 0; k < classes - 1; ++k)
      if (!lanes.aux[k]) {
        RF_CUDA_TRY(cudaStreamCreateWithFlags(&lanes.aux[k], cudaStreamNonBlocking));
        RF_CUDA_TRY(cudaEventCreateWithFlags(&lanes.join[k], cudaEventDisableTiming));
      }
    RF_CUDA_TRY(cudaEventRecord(lanes.fork, st));
  }
  int used = 0, off = 0;
  for (int c = 0; c < 4; ++c) {
    if (counts[c] == 0) continue;
    const int csize = kParts >> c;
    cudaStream_t s = st;
    if (used > 0) {
      s = lanes.aux[used - 1];
      RF_CUDA_TRY(cudaStreamWaitEvent(s, lanes.fork, 0));
    }
    const int Rmax = rmax[c];
    if (csize == 1) {
      k_pack_gmres_ir<false><<<counts[c], kPT, pack_smem_bytes(Rmax, m, 1), s>>>(members + off, Rmax, m);
      RF_LAUNCH_CHECK();
    } else {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(counts[c] * csize));
      cfg.blockDim = dim3(kPT);
      cfg.dynamicSmemBytes = pack_smem_bytes(Rmax, m, csize);
      cfg.stream = s;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)csize;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      RF_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_pack_gmres_ir<true>, members + off, Rmax, m));
    }
    if (used > 0) RF_CUDA_TRY(cudaEventRecord(lanes.join[used - 1], s));
    off += counts[c];
    ++used;
  }
  for (int k = 1; k < used; ++k) RF_CUDA_TRY(cudaStreamWaitEvent(st, lanes.join[k - 1], 0));
  return RF_OK;
}

}  // namespace rf

extern "C" int rf_debug_pack_plan(const int* fibers, int n, int sms, int* ctas) {
  if (!fibers || !ctas || n < 1 || sms < 1) return RF_E_INPUT;
  for (int i = 0; i < n; ++i)
    if (fibers[i] < 1 || fibers[i] > rf::kPackMaxFibers) return RF_E_INPUT;
  rf::pack_plan_ctas(fibers, n, sms, ctas, 8);
  return RF_OK;
}
