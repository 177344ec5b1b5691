// Assembly of the rigid-fiber linear system (numerical inner integrals).
//
// Reference: fortran/assemble_matrix.incl:1-161 with
// fortran/compute_inner_integral_numerically.incl:1-40, and the CUDA kernels
// src/kernels/assemble_system_2D.cu:8-367 + compute_inner_integral_numerically.cu.
//
// What is computed is the reference's: for every ordered pair (i, j), i != j,
//   T^{ij}_{ki,kj} = sum_qi sum_qj W[ki][qi] K(R_ij(qi,qj)) W[kj][qj]      (3x3 sym)
// with W[k][q] = w_q P_k(s_q), then the 15x15 block A_(i,j) = C_i T^{ij} and
// b_i -= C_i T^{ij}_{.,P0} F/2, where C_i is D1 t t^T (force index 0) or
// gamma_k (I - E_k t t^T).  How it is computed is not the reference's:
//  * K is even in R, so T^{ji}_{kj,ki} = T^{ij}_{ki,kj}: one CTA tile of
//    unordered fiber pairs evaluates K once per (qi, qj) and serves both
//    blocks (i,j) and (j,i)  -- half the kernel evaluations;
//  * the reference re-evaluates K once per k_j (M times); here once;
//  * the sum over fiber j's points splits each separation at its projection
//    onto fiber j's axis (r = d + u t_j, d perpendicular to t_j), so the six
//    components of K contract to four scalar moments (see phase 1);
//  * the quadrature is mirror-symmetric (s_{Q-1-q} = -s_q, w equal, P_k of
//    parity k), so both contractions fold q with Q-1-q into an even and an
//    odd part and use half the multiply-adds;
//  * the force terms F_i[k] = sum_j T^{ij}_{k,P0} F/2 are reduced
//    deterministically (per-tile partial rows, then a fixed-order sum)
//    instead of with float atomics; b_i = -C_i F_i.
//
// Two outputs share the pair-tile core:
//  * dense:      A column-major with leading dimension lda >= R (padded to 32
//                so every column starts on a 128-byte boundary), A[r + c*lda];
//  * structured: the blocks T^{ij}_{k,kj}, k,kj = P_0..P_M, once per
//                unordered pair, in FP32 (all (M+1)^2 blocks) and in 16 bits
//                (the M^2 blocks of the operator), laid out per 16x16 fiber
//                storage tile as [tile][sub-tile][j][value][i] so that one
//                CTA's writes for one j are contiguous and the matvec reads
//                whole 32-byte sectors (see rf_struct.cu).
#include "rf_common.cuh"
#include "rf_kernels.cuh"
#include "rf_analytic.cuh"

namespace rf {

// Decode a linear index over the upper triangle (I <= J) of T x T tiles.
__device__ __forceinline__ void tile_pair(int64_t L, int& I, int& J) {
  int64_t j = (int64_t)((sqrt(8.0 * (double)L + 1.0) - 1.0) * 0.5);
  while ((j + 1) * (j + 2) / 2 <= L) ++j;
  while (j * (j + 1) / 2 > L) --j;
  J = (int)j;
  I = (int)(L - j * (j + 1) / 2);
}

// kAsmApply: nothing stored; the pair blocks are applied to a vector (the
// matrix-free product) or, without a vector, only the force terms are formed
enum AsmMode { kAsmDense = 0, kAsmStructF16 = 1, kAsmStructBF16 = 2, kAsmApply = 3 };

template <int M, int Q>
struct AsmShape {
  static constexpr int TI = 192 / Q;     // fibers per tile side
  static constexpr int U = TI * Q;       // (fiber, quadrature point) units = threads used
  static constexpr int K1 = M + 1;       // P_0..P_M
  static constexpr int NC = 6 * K1;      // G columns per unit
  static constexpr int H = Q / 2;        // folded quadrature points
  static constexpr int NT = 192;         // threads per CTA
  // dynamic shared memory: G as NC columns of U units (unit u = qi * TI + il),
  // then the T blocks (6 floats each).  The column stride is TI (mod 32)
  // words: phase 2 has lanes (col, tl), TI consecutive tl per column and
  // 32 / TI columns per warp, and reads 32 distinct banks.
  static constexpr int GS = (U + 31) / 32 * 32 + TI;
  // the T blocks start on a 16-byte boundary (they are copied out as float4);
  // NC * GS is odd for odd M + 1
  static constexpr int GOFF = (NC * GS + 3) / 4 * 4;
  static constexpr size_t kGBytes = sizeof(float) * GOFF;
  // T pair stride padded so that 8 consecutive pairs start on distinct banks
  // that are multiples of 4 (stride = 4 * odd mod 32)
  static constexpr int TP = (K1 * K1 * 6 + 7) / 8 * 8 + 4;
  static constexpr size_t kTBytes = sizeof(float) * TI * TP;
  static constexpr size_t kSmem = kGBytes + 2 * kTBytes;   // T double-buffered across j
  static_assert(GOFF % 4 == 0 && TP % 4 == 0, "T buffers must be 16-byte aligned");
  // structured storage
  static constexpr int SUB = kStoreTile / TI;      // assembly tiles per storage-tile side
  static constexpr int NQ32 = K1 * K1 * 6;         // FP32 values per pair
  static constexpr int NQ16 = M * M * 6 / 2;       // 16-bit pairs per pair (M*M*6 is even)
  static_assert(kStoreTile % TI == 0, "assembly tile must divide the storage tile");
};

struct AsmOut {
  // dense
  float* A;
  int64_t lda;
  // structured
  float* S32;
  uint32_t* S16;
  // both: partial force terms ffpart[X][i][k][3]
  float* ffpart;
  // analytical: the FP64 fiber state (the closed-form integral is ~7x more
  // sensitive to the rounding of its inputs than the quadrature)
  const double4* pos64;
  const double4* ori64;
  // kAsmApply: z partial rows of T x (null x: force terms only) into
  // zpart[(assemble tiles + 1) x R]; skip: a device word that, when set,
  // makes the launch return at once (a converged Krylov solve)
  const float* x;
  float* zpart;
  const int* skip;
};

// Phase 1 of a pair tile, numerical: G[c][k] = sum_q K_c(p - s_q t_j) W[k][q]
// for one point p of fiber i (relative to fiber j's centre) against the Q
// points of fiber j, written to gcol[(6 k + c) GS].
//
// The separation r = p - s_q t_j is split at p's projection onto fiber j's
// axis: r = d + u_q t_j with d = p - s* t_j perpendicular to t_j and
// u_q = s* - s_q, so |r|^2 = |d|^2 + u_q^2 and
//   K(r) = a I + b r r^T = a I + b [d d^T + u (d t^T + t d^T) + u^2 t t^T]
// (a = 1/|r| + 2eps^2/|r|^3, b = 1/|r|^3 - 6eps^2/|r|^5).  The sum over q then
// needs four scalar moments per k instead of six tensor components,
//   A_k = sum W a,  B0_k = sum W b,  B1_k = sum W b u,  B2_k = sum W b u^2,
// and every term of the recombination is bounded by |r|^2 (|d|, |u| <= |r|),
// so nothing cancels.  s* is refined once (d . t_j, already ~1e-7 |p|, is
// folded back) so that d is perpendicular to t_j to rounding.  Points q and
// Q-1-q are evaluated together and their values folded into even and odd
// parts (W[k][Q-1-q] = (-1)^k W[k][q]).
//
// P2 = true evaluates the two mirror points in the two lanes of packed FP32
// instructions (add/mul/fma .f32x2) and accumulates the moments in lane pairs
// (A, B0), (B1, B2) against the duplicated weights W2; every rounding is the
// same as in the scalar form (all steps are explicit _rn operations, none can
// be contracted), so both give bit-identical G.
//
// FAR: the rule of the far pairs (far_pts, far_W) instead of the full one.
template <int K1, int Q, int GS, bool P2, bool FAR>
__device__ __forceinline__ void stokeslet_moments_G(const Tables& tab, const float p[3], const float4 tj, float e2,
                                                    float e2x3, float* __restrict__ gcol) {
  static_assert(P2 || !FAR, "the far rule runs packed");
  constexpr int H = Q / 2;
  const float* const pts = FAR ? tab.far_pts : tab.pts;
  float ss = fmaf(p[0], tj.x, fmaf(p[1], tj.y, p[2] * tj.z));
  float dx = fmaf(-ss, tj.x, p[0]), dy = fmaf(-ss, tj.y, p[1]), dz = fmaf(-ss, tj.z, p[2]);
  const float dl = fmaf(dx, tj.x, fmaf(dy, tj.y, dz * tj.z));
  ss += dl;
  dx = fmaf(-dl, tj.x, dx);
  dy = fmaf(-dl, tj.y, dy);
  dz = fmaf(-dl, tj.z, dz);
  const float dd = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  float2 m01[K1], m23[K1];   // (A_k, B0_k), (B1_k, B2_k)
#pragma unroll
  for (int k = 0; k < K1; ++k) m01[k] = m23[k] = make_float2(0.f, 0.f);
  // the scalar form keeps more live values per point: unrolled less, no spills
  constexpr int kUnroll = P2 ? H : 3;
#pragma unroll kUnroll
  for (int q = 0; q < H; ++q) {
    float2 fa, fb, fc, fd;   // lane x: point q, lane y: point Q-1-q
    if constexpr (P2) {
      const float2 u = __fadd2_rn(make_float2(ss, ss), make_float2(-pts[q], -pts[Q - 1 - q]));
      const float2 r2 = __ffma2_rn(u, u, make_float2(dd, dd));
      float2 inv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
      if constexpr (FAR) {
        // one Newton step: a ninth of the kernel values carry a ninth of the
        // averaging of their roundings, so each is made more exact
        const float2 e = __ffma2_rn(__fmul2_rn(r2, inv), make_float2(-inv.x, -inv.y), make_float2(1.f, 1.f));
        inv = __ffma2_rn(__fmul2_rn(inv, make_float2(0.5f, 0.5f)), e, inv);
      }
      const float2 inv2 = __fmul2_rn(inv, inv);
      const float2 inv3 = __fmul2_rn(inv2, inv);
      const float2 inv5 = __fmul2_rn(inv3, inv2);
      fa = __ffma2_rn(make_float2(e2, e2), inv3, inv);
      fb = __ffma2_rn(make_float2(e2x3, e2x3), inv5, inv3);
      fc = __fmul2_rn(fb, u);
      fd = __fmul2_rn(fc, u);
    } else {
      float r[4][2];
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        const float u = __fadd_rn(ss, -pts[side == 0 ? q : Q - 1 - q]);
        const float r2 = __fmaf_rn(u, u, dd);
        const float inv = rsqrtf(r2);
        const float inv2 = __fmul_rn(inv, inv);
        const float inv3 = __fmul_rn(inv2, inv);
        const float inv5 = __fmul_rn(inv3, inv2);
        r[0][side] = __fmaf_rn(e2, inv3, inv);
        r[1][side] = __fmaf_rn(e2x3, inv5, inv3);
        r[2][side] = __fmul_rn(r[1][side], u);
        r[3][side] = __fmul_rn(r[2][side], u);
      }
      fa = make_float2(r[0][0], r[0][1]);
      fb = make_float2(r[1][0], r[1][1]);
      fc = make_float2(r[2][0], r[2][1]);
      fd = make_float2(r[3][0], r[3][1]);
    }
    const float2 e01 = make_float2(__fadd_rn(fa.x, fa.y), __fadd_rn(fb.x, fb.y));
    const float2 o01 = make_float2(__fsub_rn(fa.x, fa.y), __fsub_rn(fb.x, fb.y));
    const float2 e23 = make_float2(__fadd_rn(fc.x, fc.y), __fadd_rn(fd.x, fd.y));
    const float2 o23 = make_float2(__fsub_rn(fc.x, fc.y), __fsub_rn(fd.x, fd.y));
#pragma unroll
    for (int k = 0; k < K1; ++k) {
      if constexpr (P2) {
        const float2 w2 = FAR ? tab.far_W2[k][FAR ? q : 0] : tab.W2[k][q];
        m01[k] = __ffma2_rn((k & 1) ? o01 : e01, w2, m01[k]);
        m23[k] = __ffma2_rn((k & 1) ? o23 : e23, w2, m23[k]);
      } else {
        const float w = tab.W[k][q];
        m01[k].x = __fmaf_rn((k & 1) ? o01.x : e01.x, w, m01[k].x);
        m01[k].y = __fmaf_rn((k & 1) ? o01.y : e01.y, w, m01[k].y);
        m23[k].x = __fmaf_rn((k & 1) ? o23.x : e23.x, w, m23[k].x);
        m23[k].y = __fmaf_rn((k & 1) ? o23.y : e23.y, w, m23[k].y);
      }
    }
  }
  // components in the order (11, 22, 33, 12, 13, 23)
  const float Dd[6] = {dx * dx, dy * dy, dz * dz, dx * dy, dx * dz, dy * dz};
  const float Sd[6] = {2.f * dx * tj.x, 2.f * dy * tj.y, 2.f * dz * tj.z, fmaf(dx, tj.y, dy * tj.x),
                       fmaf(dx, tj.z, dz * tj.x), fmaf(dy, tj.z, dz * tj.y)};
  const float Tt[6] = {tj.x * tj.x, tj.y * tj.y, tj.z * tj.z, tj.x * tj.y, tj.x * tj.z, tj.y * tj.z};
#pragma unroll
  for (int c = 0; c < 6; ++c)
#pragma unroll
    for (int k = 0; k < K1; ++k)
      gcol[(k * 6 + c) * GS] =
          fmaf(m01[k].y, Dd[c], fmaf(m23[k].x, Sd[c], fmaf(m23[k].y, Tt[c], c < 3 ? m01[k].x : 0.f)));
}

// ---------------------------------------------------------------------------
// Numerical pair tiles: TI x TI fibers, unordered pairs, both blocks of a pair
// from one evaluation of K.  A pair whose centres are at least sqrt(far_d2)
// apart takes the far rule, the kFarNodes-point Gauss rule of the quadrature's
// own discrete measure (make_tables), on both fibers: 64 kernel evaluations
// instead of Q^2 = 576, within 3e-10 of the full rule's blocks (below their
// FP32 rounding).  The others take the full rule.
//
// Bound: FP32 issue in the matrix-free product, HBM stores in the structured
// assembly.  The far pairs run in batches of 32 (four j of the tile at once:
// 32 pairs x 8 points = the CTA's 256 threads), so that every phase has one
// unit per thread and lane = pair keeps shared memory free of conflicts; the
// near pairs are compacted per tile and run in groups of TI pairs x Q points.
// ---------------------------------------------------------------------------
template <int M, int Q>
struct NumShape {
  using A = AsmShape<M, Q>;
  static constexpr int TI = A::TI, K1 = A::K1, NC = A::NC, NQ32 = A::NQ32;
  static constexpr int NT = 256;
  static constexpr int FN = kFarNodes;
  // far pairs per batch: 32 (one per lane); 16 where the tile has no more, and
  // for M > 5, whose G and T of 32 pairs would leave one CTA per SM
  static constexpr int PB = (M <= 5 && TI * TI >= 32) ? 32 : 16;
  static constexpr int JB = PB / TI;                       // j of a batch
  static constexpr int GSF = PB * FN + PB % 32;            // G column stride (words): lanes (col, pair)
  static constexpr int QP = Q + 1;                         // near: words per slot of a G column
  static constexpr int GSN = TI * QP + (TI * QP + 1) % 2;  // odd: lanes = columns read distinct banks
  static constexpr int GFLOATS = (NC * (GSF > GSN ? GSF : GSN) + 3) / 4 * 4;
  // T of a far batch, structured and matrix-free: [jj][value][i], the j
  // stride = TI (mod 32) past a multiple of 16 so that 32 pairs hit distinct
  // banks; dense and near: [pair][value] with AsmShape's padded stride
  static constexpr int JS = NQ32 * TI + TI;
  static constexpr int TP = A::TP;
  static constexpr int TF0 = JB * JS, TF1 = PB * TP, TF2 = TI * TP;
  static constexpr int TFLOATS = TF0 > TF1 ? (TF0 > TF2 ? TF0 : TF2) : (TF1 > TF2 ? TF1 : TF2);
  static constexpr size_t kSmem = sizeof(float) * (GFLOATS + TFLOATS);
  static_assert(PB % TI == 0 && JS % 4 == 0 && TP % 4 == 0, "batches are whole j; T is copied out as float4");
  static_assert(TI % JB == 0, "batches cover the tile's j");
};

// Block (rows of fiber a, columns of fiber b) of the dense matrix from the
// symmetric T6: dst[r + c lda] = [C_k T]_{rc}, C_k of fiber a.
__device__ __forceinline__ void dense_block(float* __restrict__ dst, int64_t lda, const float* T6, const float4 ta,
                                            int k, float coef, float E) {
  const float t3[3] = {ta.x, ta.y, ta.z};
  float Qv[3];
#pragma unroll
  for (int b = 0; b < 3; ++b)
    Qv[b] = sym_get(T6, b, 0) * t3[0] + sym_get(T6, b, 1) * t3[1] + sym_get(T6, b, 2) * t3[2];
#pragma unroll
  for (int b = 0; b < 3; ++b)
#pragma unroll
    for (int a = 0; a < 3; ++a)
      dst[a + b * lda] = k == 0 ? coef * t3[a] * Qv[b] : coef * (sym_get(T6, a, b) - E * t3[a] * Qv[b]);
}

// One CTA's tile pair (I, J) of one suspension (the body of k_assemble_pairs and
// of the packed assembly, which maps its blocks onto many suspensions' tiles).
// P2 selects the near pairs' phase-1 form; the far pairs always take the
// packed one (the same roundings).
template <int M, int Q, int MODE, bool P2>
__device__ __forceinline__ void assemble_pair_tile(const Tables& tab, int N, const float4* __restrict__ ori,
                                                   const AsmOut& out, int I, int J) {
  using S = NumShape<M, Q>;
  constexpr int TI = S::TI, K1 = S::K1, NC = S::NC, NT = S::NT, PB = S::PB, JB = S::JB, TP = S::TP, JS = S::JS;
  constexpr int NQ32 = S::NQ32, NC2 = NC / 2;
  constexpr int M3 = 3 * M;
  constexpr int FF = K1 * 3;   // force-term floats per fiber
  constexpr bool STRUCT = MODE == kAsmStructF16 || MODE == kAsmStructBF16;
  constexpr bool APPLY = MODE == kAsmApply;
  constexpr bool QT = MODE != kAsmDense;   // far T as [jj][value][i]
  static_assert(Q % 2 == 0, "mirror folding needs an even number of quadrature points");

  __shared__ float4 sTi[TI], sTj[TI];    // orientations
  __shared__ float sD[TI * TI][3];       // pair jl * TI + il: x_i - x_j, formed in FP64 and rounded once
  __shared__ unsigned char sFar[TI * TI];
  __shared__ unsigned char sNear[TI * TI];   // the near pairs, in pair order
  __shared__ int sNearW[NT / 32];            // near pairs per warp of the classification
  extern __shared__ __align__(16) float smem_dyn[];
  float* const sG = smem_dyn;
  float* const sT = smem_dyn + S::GFLOATS;
  __shared__ float sCoef[kMaxTerms], sEig[kMaxTerms];
  __shared__ float sFi[TI * FF], sFj[TI * FF];   // force terms of the tile's i and j
  __shared__ short sMapS[STRUCT ? NQ32 : 1];     // stored value q (s32_block order) -> offset of its T entry

  const bool diag = (I == J);
  const int tid = threadIdx.x, lane = tid & 31;
  const int i0 = I * TI, j0 = J * TI;
  // kAsmApply with a vector applies the blocks; without one it forms the force terms
  const bool do_apply = APPLY && out.x != nullptr;
  const bool do_force = !do_apply;
  constexpr int XW = APPLY ? TI * M3 : 1;
  __shared__ float sXi[XW], sXj[XW], sZi[XW], sZj[XW];   // x and z rows of the I and J tiles
  __shared__ float sNz[APPLY ? 2 * TI * M3 : 1];         // near pairs' products of one group

  if (tid < M) { sCoef[tid] = tab.gamma[tid]; sEig[tid] = tab.eigen[tid]; }
  if (tid < TI) {
    sTi[tid] = ori[min(i0 + tid, N - 1)];
    sTj[tid] = ori[min(j0 + tid, N - 1)];
  }
  bool near_pair = false;
  if (tid < TI * TI) {
    // the separation of quadrature points is formed as (x_i - x_j) + s_qi t_i -
    // s_qj t_j with the centre difference taken in FP64 and rounded once, so
    // its error scales with the fibers' distance rather than with their
    // distance from the origin (FP32 points x + s t far from the origin lose
    // ~1e-6 absolutely, which for nearly touching fibers is ~1e-4 of the kernel)
    const int il = tid % TI, jl = tid / TI;
    const double4 xi = out.pos64[min(i0 + il, N - 1)], xj = out.pos64[min(j0 + jl, N - 1)];
    const float dx = (float)(xi.x - xj.x), dy = (float)(xi.y - xj.y), dz = (float)(xi.z - xj.z);
    sD[tid][0] = dx;
    sD[tid][1] = dy;
    sD[tid][2] = dz;
    const bool valid = i0 + il < N && j0 + jl < N && (!diag || il < jl);
    near_pair = valid && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < tab.far_d2;
    sFar[tid] = valid && !near_pair;
  }
  const unsigned near_mask = __ballot_sync(0xffffffffu, near_pair);
  if (lane == 0) sNearW[tid >> 5] = __popc(near_mask);
  for (int k = tid; k < TI * FF; k += NT) sFi[k] = sFj[k] = 0.f;
  if constexpr (APPLY) {
    if (do_apply) {
      for (int k = tid; k < TI * M3; k += NT) {
        const int f = k / M3, c = k % M3;
        sXi[k] = i0 + f < N ? out.x[(int64_t)(i0 + f) * M3 + c] : 0.f;
        sXj[k] = j0 + f < N ? out.x[(int64_t)(j0 + f) * M3 + c] : 0.f;
        sZi[k] = sZj[k] = 0.f;
      }
    }
  }
  if constexpr (STRUCT) {
    for (int q = tid; q < NQ32; q += NT) {
      const int c = q % 6, blk = q / 6;
      int row = 0, col = 0;
      if (blk < M * M) {
        row = blk / M + 1;
        col = blk % M + 1;
      } else if (blk < M * M + K1) {
        col = blk - M * M;
      } else {
        row = blk - M * M - M;
      }
      sMapS[q] = (short)((row * K1 + col) * 6 + c);
    }
  }
  const float e2 = tab.e2;
  const float e2x3 = -3.f * e2;
  const float fz = tab.fz_half;
  __syncthreads();
  int nnear = 0;
  {
    int before = 0;
#pragma unroll
    for (int w = 0; w < (TI * TI + 31) / 32; ++w) {
      if (w < (tid >> 5)) before += sNearW[w];
      nnear += sNearW[w];
    }
    // read after the barriers of the far batches
    if (near_pair) sNear[before + __popc(near_mask & ((1u << lane) - 1))] = (unsigned char)tid;
  }

  // structured storage: the record of j = j0 + jl
  constexpr int SUB = kStoreTile / TI;
  const int64_t rec0 = (((int64_t)(J / SUB) * (J / SUB + 1) / 2 + I / SUB) * SUB * SUB + (I % SUB) * SUB + (J % SUB)) * TI;
  constexpr int NW = s16_record_words(M);
  constexpr int NQ16 = AsmShape<M, Q>::NQ16;
  // words 4 w4 .. 4 w4 + 3 of the 16-bit record whose T entries are t[sMapS[.] * stride]
  auto words16 = [&](const float* t, int stride, int w4) -> uint4 {
    uint32_t w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int q2 = 4 * w4 + u;
      const float lo = q2 < NQ16 ? t[sMapS[2 * q2] * stride] : 0.f;
      const float hi = q2 < NQ16 ? t[sMapS[2 * q2 + 1] * stride] : 0.f;
      if constexpr (MODE == kAsmStructF16) {
        __half2 hv = __floats2half2_rn(lo, hi);
        w[u] = *reinterpret_cast<uint32_t*>(&hv);
      } else {
        __nv_bfloat162 hv = __floats2bfloat162_rn(lo, hi);
        w[u] = *reinterpret_cast<uint32_t*>(&hv);
      }
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  };

  // i-side sums of task (jj, k, il) = this thread, over the batches: force
  // terms (k <= M) or z (k < M)
  float iacc[3] = {0.f, 0.f, 0.f};
  const int jcount = min(TI, N - j0);

  // ---- far pairs, JB rows of the tile per batch -----------------------------
  for (int jb = 0; jb < jcount; jb += JB) {
    // phase 1: G[c][k] = sum_qj K_c(qi, qj) W[k][qj], unit u = qi * PB + pair
    if (tid < PB * S::FN) {
      const int p = tid % PB, qi = tid / PB;
      const int il = p % TI, jl = jb + p / TI;
      float* const gcol = sG + tid;
      if (sFar[jl * TI + il]) {
        const float4 ti = sTi[il];
        const float si = tab.far_pts[qi];
        const float* D = sD[jl * TI + il];
        const float pp[3] = {fmaf(si, ti.x, D[0]), fmaf(si, ti.y, D[1]), fmaf(si, ti.z, D[2])};
        stokeslet_moments_G<K1, S::FN, S::GSF, true, true>(tab, pp, sTj[jl], e2, e2x3, gcol);
      } else {
#pragma unroll
        for (int c = 0; c < NC; ++c) gcol[c * S::GSF] = 0.f;
      }
    }
    __syncthreads();
    // phase 2: T[ki][kj][c] = sum_qi W[ki][qi] G[qi][c][kj], folded over qi;
    // lanes = pairs, a lane takes columns col and col + NC/2 in the two lanes of
    // packed FP32 instructions
    for (int task = tid; task < PB * NC2; task += NT) {
      const int col = task / PB, p = task % PB;
      const float* ga = sG + col * S::GSF + p;
      const float* gb = ga + NC2 * S::GSF;
      float2 acc[K1];
#pragma unroll
      for (int k = 0; k < K1; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < S::FN / 2; ++q) {
        const float2 lo = make_float2(ga[q * PB], gb[q * PB]);
        const float2 hi = make_float2(ga[(S::FN - 1 - q) * PB], gb[(S::FN - 1 - q) * PB]);
        const float2 ev = __fadd2_rn(lo, hi), od = __ffma2_rn(hi, make_float2(-1.f, -1.f), lo);
#pragma unroll
        for (int k = 0; k < K1; ++k) acc[k] = __ffma2_rn((k & 1) ? od : ev, tab.far_W2[k][q], acc[k]);
      }
      // column col = kj * 6 + c; T entry (k * K1 + kj) * 6 + c = k * NC + col
      float* const dst = QT ? sT + (p / TI) * JS + p % TI : sT + p * TP;
      constexpr int QS = QT ? TI : 1;
#pragma unroll
      for (int k = 0; k < K1; ++k) {
        dst[(k * NC + col) * QS] = acc[k].x;
        dst[(k * NC + col + NC2) * QS] = acc[k].y;
      }
    }
    __syncthreads();
    // phase 3: the batch's blocks to their destination (the next batch's phase 1
    // writes G only, and its phase 2 follows a barrier)
    if constexpr (MODE == kAsmDense) {
      // block (i, j): rows of fiber i, columns of fiber j
      for (int task = tid; task < PB * M * M; task += NT) {
        const int jj = task / (TI * M * M), r0 = task % (TI * M * M);
        const int kJp = r0 / (TI * M), rem = r0 % (TI * M);
        const int tl = rem / M, kIp = rem % M, jl = jb + jj;
        float* dst = out.A + (int64_t)(i0 * M3 + 3 * rem) + (int64_t)((j0 + jl) * M3 + 3 * kJp) * out.lda;
        if (diag && tl == jl && jl < jcount) {
#pragma unroll
          for (int b = 0; b < 3; ++b)
#pragma unroll
            for (int a = 0; a < 3; ++a) dst[a + b * out.lda] = (kIp == kJp && a == b) ? 1.f : 0.f;
          continue;
        }
        if (!sFar[jl * TI + tl]) continue;
        dense_block(dst, out.lda, sT + (jj * TI + tl) * TP + ((kIp + 1) * K1 + kJp + 1) * 6, sTi[tl], kIp, sCoef[kIp],
                    sEig[kIp]);
      }
      // block (j, i): rows of fiber j, columns of fiber i
      for (int task = tid; task < PB * M * M; task += NT) {
        const int jj = task / (TI * M * M), r0 = task % (TI * M * M);
        const int tl = r0 / (M * M), rem = r0 % (M * M);
        const int kIp = rem / M, kJp = rem % M, jl = jb + jj;
        if (!sFar[jl * TI + tl]) continue;
        float* dst = out.A + (int64_t)((j0 + jl) * M3 + 3 * kJp) + (int64_t)((i0 + tl) * M3 + 3 * kIp) * out.lda;
        dense_block(dst, out.lda, sT + (jj * TI + tl) * TP + ((kIp + 1) * K1 + kJp + 1) * 6, sTj[jl], kJp, sCoef[kJp],
                    sEig[kJp]);
      }
    } else if constexpr (STRUCT) {
      // T is [jj][q][il] with q in (row, col) order, stored in s32_block order:
      // one j is a contiguous run of NQ32 x TI floats.  Near pairs and pairs
      // that do not exist (i >= N, i >= j on a diagonal tile) are exact zeros
      // here (the near pairs' blocks follow below).  No FP32 copy in the
      // recompute modes (out.S32 null)
      const int jn = min(JB, jcount - jb);
      if (out.S32 != nullptr) {
        float4* d32 = reinterpret_cast<float4*>(out.S32 + (rec0 + jb) * (int64_t)(NQ32 * TI));
        constexpr int V = NQ32 * TI / 4;   // float4 per j
        for (int v = tid; v < jn * V; v += NT) {
          const int jj = v / V, r = v % V;
          const int q = r / (TI / 4), g4 = (r % (TI / 4)) * 4;
          d32[v] = *reinterpret_cast<const float4*>(sT + jj * JS + sMapS[q] * TI + g4);
        }
      }
      // 16-bit records [il][NW]: pair il's words are contiguous
      uint32_t* d16 = out.S16 + (rec0 + jb) * (int64_t)(NW * TI);
      for (int v = tid; v < jn * (TI * NW / 4); v += NT) {
        const int jj = v / (TI * NW / 4), r = v % (TI * NW / 4);
        const int tl = r % TI, w4 = r / TI;
        *reinterpret_cast<uint4*>(&d16[(jj * TI + tl) * NW + 4 * w4]) = words16(sT + jj * JS + tl, TI, w4);
      }
    }
    // i side: sums over the thread's own j of each batch; j side: sums over the
    // tile's i by halving shuffles in groups of TI lanes
    if (APPLY && do_apply) {
      if constexpr (APPLY) {
        for (int task = tid; task < 2 * PB * M; task += NT) {
          const bool iside = task < PB * M;
          const int u = iside ? task : task - PB * M;
          const int jj = u / (TI * M), k = (u / TI) % M, tl = u % TI, jl = jb + jj;
          const float* xv = iside ? sXj + jl * M3 : sXi + tl * M3;
          float zs[3] = {0.f, 0.f, 0.f};
#pragma unroll
          for (int l = 0; l < M; ++l) {
            const float* t = sT + jj * JS + ((iside ? (k + 1) * K1 + l + 1 : (l + 1) * K1 + k + 1) * 6) * TI + tl;
            const float T6[6] = {t[0], t[TI], t[2 * TI], t[3 * TI], t[4 * TI], t[5 * TI]};
#pragma unroll
            for (int a = 0; a < 3; ++a)
              zs[a] = fmaf(sym_get(T6, a, 0), xv[3 * l],
                           fmaf(sym_get(T6, a, 1), xv[3 * l + 1], fmaf(sym_get(T6, a, 2), xv[3 * l + 2], zs[a])));
          }
          if (iside) {
#pragma unroll
            for (int a = 0; a < 3; ++a) iacc[a] += zs[a];
          } else {
            const unsigned grp = (TI == 32 ? 0xffffffffu : ((1u << TI) - 1u)) << (lane & ~(TI - 1));
#pragma unroll
            for (int o = TI / 2; o > 0; o >>= 1)
#pragma unroll
              for (int a = 0; a < 3; ++a) zs[a] += __shfl_xor_sync(grp, zs[a], o);
            if (tl == 0)
#pragma unroll
              for (int a = 0; a < 3; ++a) sZj[jl * M3 + 3 * k + a] = zs[a];
          }
        }
      }
    } else {
      // force terms F_i[k] += T^{ij}[k][P0] F/2 and F_j[kj] += T^{ij}[P0][kj] F/2
      // (F/2 = (0, 0, fz): column z of the block)
      for (int task = tid; task < 2 * PB * K1; task += NT) {
        const bool iside = task < PB * K1;
        const int u = iside ? task : task - PB * K1;
        const int jj = u / (TI * K1), k = (u / TI) % K1, tl = u % TI, jl = jb + jj;
        const int q0 = (iside ? k * K1 : k) * 6;
        const float* t = QT ? sT + jj * JS + q0 * TI + tl : sT + (jj * TI + tl) * TP + q0;
        constexpr int QS = QT ? TI : 1;
        float f3[3] = {t[4 * QS], t[5 * QS], t[2 * QS]};
        if (iside) {
#pragma unroll
          for (int a = 0; a < 3; ++a) iacc[a] = fmaf(f3[a], fz, iacc[a]);
        } else {
          const unsigned grp = (TI == 32 ? 0xffffffffu : ((1u << TI) - 1u)) << (lane & ~(TI - 1));
#pragma unroll
          for (int o = TI / 2; o > 0; o >>= 1)
#pragma unroll
            for (int a = 0; a < 3; ++a) f3[a] += __shfl_xor_sync(grp, f3[a], o);
          if (tl == 0)
#pragma unroll
            for (int a = 0; a < 3; ++a) sFj[jl * FF + 3 * k + a] = f3[a] * fz;
        }
      }
    }
  }

  // ---- near pairs, groups of up to TI ----------------------------------------
  for (int n0 = 0; n0 < nnear; n0 += TI) {
    const int cnt = min(TI, nnear - n0);
    __syncthreads();   // G and T of the previous batch or group are read
    if (tid < cnt * Q) {
      const int slot = tid / Q, qi = tid % Q;
      const int pr = sNear[n0 + slot], il = pr % TI, jl = pr / TI;
      const float4 ti = sTi[il];
      const float si = tab.pts[qi];
      const float pp[3] = {fmaf(si, ti.x, sD[pr][0]), fmaf(si, ti.y, sD[pr][1]), fmaf(si, ti.z, sD[pr][2])};
      stokeslet_moments_G<K1, Q, S::GSN, P2, false>(tab, pp, sTj[jl], e2, e2x3, sG + slot * S::QP + qi);
    }
    __syncthreads();
    // lanes = columns; P2 as in the far phase 2 (lo - hi as fma(hi, -1, lo): the
    // same rounding as the scalar subtraction)
    if constexpr (P2) {
      for (int task = tid; task < cnt * NC2; task += NT) {
        const int slot = task / NC2, col = task % NC2;
        const float* ga = sG + col * S::GSN + slot * S::QP;
        const float* gb = ga + NC2 * S::GSN;
        float2 acc[K1];
#pragma unroll
        for (int k = 0; k < K1; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll
        for (int q = 0; q < Q / 2; ++q) {
          const float2 lo = make_float2(ga[q], gb[q]), hi = make_float2(ga[Q - 1 - q], gb[Q - 1 - q]);
          const float2 ev = __fadd2_rn(lo, hi), od = __ffma2_rn(hi, make_float2(-1.f, -1.f), lo);
#pragma unroll
          for (int k = 0; k < K1; ++k) acc[k] = __ffma2_rn((k & 1) ? od : ev, tab.W2[k][q], acc[k]);
        }
#pragma unroll
        for (int k = 0; k < K1; ++k) {
          sT[slot * TP + k * NC + col] = acc[k].x;
          sT[slot * TP + k * NC + col + NC2] = acc[k].y;
        }
      }
    } else {
      for (int task = tid; task < cnt * NC; task += NT) {
        const int slot = task / NC, col = task % NC;
        const float* gp = sG + col * S::GSN + slot * S::QP;
        float acc[K1];
#pragma unroll
        for (int k = 0; k < K1; ++k) acc[k] = 0.f;
#pragma unroll 4
        for (int q = 0; q < Q / 2; ++q) {
          const float lo = gp[q], hi = gp[Q - 1 - q];
          const float ev = __fadd_rn(lo, hi), od = __fsub_rn(lo, hi);
#pragma unroll
          for (int k = 0; k < K1; ++k) acc[k] = __fmaf_rn((k & 1) ? od : ev, tab.W[k][q], acc[k]);
        }
#pragma unroll
        for (int k = 0; k < K1; ++k) sT[slot * TP + k * NC + col] = acc[k];
      }
    }
    __syncthreads();
    if constexpr (MODE == kAsmDense) {
      for (int task = tid; task < 2 * cnt * M * M; task += NT) {
        const int side = task / (cnt * M * M), rem = task % (cnt * M * M);
        const int slot = rem / (M * M), kJp = (rem % (M * M)) / M, kIp = rem % M;
        const int pr = sNear[n0 + slot], il = pr % TI, jl = pr / TI;
        const int64_t ri = (int64_t)(i0 + il) * M3 + 3 * kIp, rj = (int64_t)(j0 + jl) * M3 + 3 * kJp;
        const float* T6 = sT + slot * TP + ((kIp + 1) * K1 + kJp + 1) * 6;
        if (side == 0) dense_block(out.A + ri + rj * out.lda, out.lda, T6, sTi[il], kIp, sCoef[kIp], sEig[kIp]);
        else dense_block(out.A + rj + ri * out.lda, out.lda, T6, sTj[jl], kJp, sCoef[kJp], sEig[kJp]);
      }
    } else if constexpr (STRUCT) {
      // over the zeros that the far batches of this CTA stored (ordered by the
      // barriers above)
      if (out.S32 != nullptr)
        for (int v = tid; v < cnt * NQ32; v += NT) {
          const int slot = v / NQ32, q = v % NQ32;
          const int pr = sNear[n0 + slot];
          out.S32[(rec0 + pr / TI) * (int64_t)(NQ32 * TI) + q * TI + pr % TI] = sT[slot * TP + sMapS[q]];
        }
      for (int v = tid; v < cnt * (NW / 4); v += NT) {
        const int slot = v / (NW / 4), w4 = v % (NW / 4);
        const int pr = sNear[n0 + slot];
        uint32_t* d16 = out.S16 + ((rec0 + pr / TI) * TI + pr % TI) * (int64_t)NW;
        *reinterpret_cast<uint4*>(&d16[4 * w4]) = words16(sT + slot * TP, 1, w4);
      }
    }
    if (APPLY && do_apply) {
      if constexpr (APPLY) {
        for (int task = tid; task < 2 * cnt * M; task += NT) {
          const int side = task / (cnt * M), slot = (task % (cnt * M)) / M, k = task % M;
          const int pr = sNear[n0 + slot];
          const float* xv = side == 0 ? sXj + (pr / TI) * M3 : sXi + (pr % TI) * M3;
          float zs[3] = {0.f, 0.f, 0.f};
#pragma unroll
          for (int l = 0; l < M; ++l) {
            const float* T6 = sT + slot * TP + (side == 0 ? (k + 1) * K1 + l + 1 : (l + 1) * K1 + k + 1) * 6;
#pragma unroll
            for (int a = 0; a < 3; ++a)
              zs[a] = fmaf(sym_get(T6, a, 0), xv[3 * l],
                           fmaf(sym_get(T6, a, 1), xv[3 * l + 1], fmaf(sym_get(T6, a, 2), xv[3 * l + 2], zs[a])));
          }
#pragma unroll
          for (int a = 0; a < 3; ++a) sNz[(side * TI + slot) * M3 + 3 * k + a] = zs[a];
        }
        __syncthreads();
        for (int u = tid; u < 2 * M3; u += NT) {
          const int side = u / M3, c = u % M3;
          for (int slot = 0; slot < cnt; ++slot) {
            const int pr = sNear[n0 + slot];
            (side == 0 ? sZi[(pr % TI) * M3 + c] : sZj[(pr / TI) * M3 + c]) += sNz[(side * TI + slot) * M3 + c];
          }
        }
      }
    } else if (tid < 2 * FF) {
      // component a of force term k of one side: the group's pairs in order
      const int side = tid / FF, k = (tid % FF) / 3, a = tid % 3;
      const int q0 = (side == 0 ? k * K1 : k) * 6 + (a == 0 ? 4 : a == 1 ? 5 : 2);
      for (int slot = 0; slot < cnt; ++slot) {
        const int pr = sNear[n0 + slot];
        float& f = side == 0 ? sFi[(pr % TI) * FF + 3 * k + a] : sFj[(pr / TI) * FF + 3 * k + a];
        f = fmaf(sT[slot * TP + q0], fz, f);
      }
    }
  }
  __syncthreads();

  // ---- i-side sums over the JB rows of a batch, added to the near pairs' -----
  if (APPLY && do_apply) {
    if constexpr (APPLY) {
      if (tid < PB * M) {
        const int jj = tid / (TI * M), k = (tid / TI) % M, tl = tid % TI;
#pragma unroll
        for (int a = 0; a < 3; ++a) sG[(jj * TI + tl) * M3 + 3 * k + a] = iacc[a];
      }
      __syncthreads();
      // partial rows of z: the i side of tile (I, J) to slot J, the j side to
      // slot I (a diagonal tile's j side to slot T): every slot of every fiber
      // is written exactly once per product
      const int64_t R = (int64_t)M3 * N;
      const int T8 = (N + TI - 1) / TI;
      float* zi = out.zpart + (int64_t)J * R + (int64_t)i0 * M3;
      float* zj = out.zpart + (int64_t)(diag ? T8 : I) * R + (int64_t)j0 * M3;
      for (int u = tid; u < TI * M3; u += NT) {
        float v = sZi[u];
#pragma unroll
        for (int jj = 0; jj < JB; ++jj) v += sG[jj * TI * M3 + u];
        if (i0 + u / M3 < N) zi[u] = v;
        if (j0 + u / M3 < N) zj[u] = sZj[u];
      }
    }
    return;
  }
  if (tid < PB * K1) {
    const int jj = tid / (TI * K1), k = (tid / TI) % K1, tl = tid % TI;
#pragma unroll
    for (int a = 0; a < 3; ++a) sG[(jj * TI + tl) * FF + 3 * k + a] = iacc[a];
  }
  __syncthreads();
  // partial force terms: ffpart[X][fiber of Y][k][3] written exactly once
  for (int u = tid; u < TI * FF; u += NT) {
    float v = sFi[u];
#pragma unroll
    for (int jj = 0; jj < JB; ++jj) v += sG[jj * TI * FF + u];
    if (diag) v += sFj[u];
    if (i0 + u / FF < N) out.ffpart[((int64_t)J * N + i0) * FF + u] = v;
    if (!diag && j0 + u / FF < N) out.ffpart[((int64_t)I * N + j0) * FF + u] = sFj[u];
  }
}

template <int M, int Q, int MODE, bool P2>
__global__ void __launch_bounds__(256, M <= 5 ? 3 : 2)
k_assemble_pairs(const Tables tab, int N, const float4* __restrict__ ori, AsmOut out) {
  if (MODE == kAsmApply && out.skip != nullptr && *out.skip) return;
  int I, J;
  tile_pair(blockIdx.x, I, J);
  assemble_pair_tile<M, Q, MODE, P2>(tab, N, ori, out, I, J);
}

// ---------------------------------------------------------------------------
// Analytical pair tiles: ordered pairs (the inner integral over fiber j is
// exact, the outer one over fiber i a quadrature, so the blocks of (i, j) and
// (j, i) are different numbers), dense output only.
// ---------------------------------------------------------------------------
template <int M, int Q>
__global__ void __launch_bounds__(192, 2)
k_assemble_analytical(const Tables tab, int N, const float4* __restrict__ ori, AsmOut out) {
  using S = AsmShape<M, Q>;
  constexpr int TI = S::TI, K1 = S::K1, NC = S::NC, H = S::H, TP = S::TP;
  constexpr int M3 = 3 * M;
  constexpr int FF = K1 * 3;
  __shared__ float4 sTi[TI];
  extern __shared__ __align__(16) float smem_dyn[];
  float (*sG)[S::GS] = reinterpret_cast<float (*)[S::GS]>(smem_dyn);   // [NC][GS]
  float* const sTbase = smem_dyn + S::GOFF;                            // 2 x [TI][TP]
  __shared__ float sCoef[kMaxTerms], sEig[kMaxTerms];
  const int T = (N + TI - 1) / TI;
  const int I = blockIdx.x / T, J = blockIdx.x % T;
  const bool diag = (I == J);
  const int tid = threadIdx.x;
  const int i0 = I * TI, j0 = J * TI;
  if (tid < M) { sCoef[tid] = tab.gamma[tid]; sEig[tid] = tab.eigen[tid]; }
  if (tid < TI) sTi[tid] = ori[min(i0 + tid, N - 1)];
  // own unit: u = qi * TI + il (a warp holds 32 / TI points of TI fibers)
  const int il = tid % TI, qi = tid / TI;
  const int i = i0 + il;
  const bool unit_ok = (tid < S::U) && (i < N);
  const float fz = tab.fz_half;
  // force-term accumulator of task (tl, k) = (tid / K1, tid % K1): F_i[k]
  float facc[3] = {0.f, 0.f, 0.f};
  __syncthreads();
  const int jcount = min(TI, N - j0);
  for (int jl = 0; jl < jcount; ++jl) {
    // T is double-buffered: phase 2 of step jl+1 may run while phase 3 of
    // step jl still reads, so one barrier per step suffices after phase 2
    float* const sT = sTbase + (jl & 1) * (TI * TP);
    const bool pair_ok = unit_ok && (!diag || il != jl);
    // ---- phase 1: the closed-form integrals G[c][k] of this unit
    float* const gcol = &sG[0][0] + tid;
    if (tid < S::U) {
      float g[6][K1];
#pragma unroll
      for (int c = 0; c < 6; ++c)
#pragma unroll
        for (int k = 0; k < K1; ++k) g[c][k] = 0.f;
      if (pair_ok) {
        const double4 xi4 = out.pos64[i], ti4 = out.ori64[i];
        const double4 xj4 = out.pos64[j0 + jl], tj4 = out.ori64[j0 + jl];
        const double s = (double)tab.pts[qi];
        const double R0[3] = {xi4.x + s * ti4.x - xj4.x, xi4.y + s * ti4.y - xj4.y, xi4.z + s * ti4.z - xj4.z};
        const double tj[3] = {tj4.x, tj4.y, tj4.z};
        analytic_G<M>(R0, tj, 2.0 * (double)tab.eps * (double)tab.eps, g);
      }
#pragma unroll
      for (int c = 0; c < 6; ++c)
#pragma unroll
        for (int k = 0; k < K1; ++k) gcol[(k * 6 + c) * S::GS] = g[c][k];
    }
    __syncthreads();
    // ---- phase 2: T[ki][kj][c] = sum_qi W[ki][qi] G[qi][c][kj], folded over qi
    // lanes (col, tl), tl fastest; column col = kj * 6 + c
    for (int task = tid; task < TI * NC; task += S::NT) {
      const int col = task / TI, tl = task % TI;
      const float* gp = &sG[col][tl];
      float acc[K1];
#pragma unroll
      for (int k = 0; k < K1; ++k) acc[k] = 0.f;
#pragma unroll
      for (int q = 0; q < H; ++q) {
        const float lo = gp[q * TI], hi = gp[(Q - 1 - q) * TI];
        const float ev = __fadd_rn(lo, hi), od = __fsub_rn(lo, hi);
#pragma unroll
        for (int k = 0; k < K1; ++k) acc[k] = __fmaf_rn((k & 1) ? od : ev, tab.W[k][q], acc[k]);
      }
#pragma unroll
      for (int k = 0; k < K1; ++k) sT[tl * TP + k * NC + col] = acc[k];
    }
    __syncthreads();
    // ---- phase 3: block (i, j) -- rows of fiber i, columns of fiber j
    const int j = j0 + jl;
    for (int task = tid; task < TI * M * M; task += S::NT) {
      const int kJp = task / (TI * M), rem = task % (TI * M);
      const int tl = rem / M, kIp = rem % M;
      const int ii = i0 + tl;
      if (ii >= N) continue;
      float* dst = out.A + (int64_t)(i0 * M3 + 3 * rem) + (int64_t)(j * M3 + 3 * kJp) * out.lda;
      if (diag && tl == jl) {
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
          for (int a = 0; a < 3; ++a) dst[a + b * out.lda] = (kIp == kJp && a == b) ? 1.f : 0.f;
        continue;
      }
      dense_block(dst, out.lda, sT + tl * TP + ((kIp + 1) * K1 + kJp + 1) * 6, sTi[tl], kIp, sCoef[kIp], sEig[kIp]);
    }
    // ---- force terms F_i[k] += T^{ij}[k][P0] F/2 (F/2 = (0, 0, fz): column z of the block)
    if (tid < TI * K1) {
      const int tl = tid / K1, k = tid % K1;
      if (i0 + tl < N && (!diag || tl != jl)) {
        const float* t = sT + tl * TP + k * NC;
        facc[0] = fmaf(t[4], fz, facc[0]);
        facc[1] = fmaf(t[5], fz, facc[1]);
        facc[2] = fmaf(t[2], fz, facc[2]);
      }
    }
  }
  // ---- partial force terms: ffpart[J][fiber of I][k][3] written exactly once
  if (tid < TI * K1) {
    const int tl = tid / K1, k = tid % K1;
    if (i0 + tl < N) {
      float* dst = out.ffpart + ((int64_t)J * N + i0 + tl) * FF + 3 * k;
#pragma unroll
      for (int a = 0; a < 3; ++a) dst[a] = facc[a];
    }
  }
}

// F[i][k] = sum_X ffpart[X][i][k] (fixed order); b[i][k'] = -C_i(k') F[i][k'+1]
// for unit u = (i, k) of N (M + 1).
__device__ __forceinline__ void force_term_unit(const Tables& tab, int N, const float4* __restrict__ ori,
                                                const float* __restrict__ ffpart, int nparts, float* __restrict__ F,
                                                float* __restrict__ b, int64_t u) {
  const int M = tab.M, K1 = M + 1, FFn = 3 * K1;
  {
    const int i = (int)(u / K1), k = (int)(u % K1);
    float s[3] = {0.f, 0.f, 0.f};
    for (int p = 0; p < nparts; ++p) {
      const float* src = ffpart + ((int64_t)p * N + i) * FFn + 3 * k;
      s[0] += src[0]; s[1] += src[1]; s[2] += src[2];
    }
    float* f = F + (int64_t)i * FFn + 3 * k;
    f[0] = s[0]; f[1] = s[1]; f[2] = s[2];
    if (k >= 1) {
      const int kp = k - 1;
      const float4 t = ori[i];
      const float t3[3] = {t.x, t.y, t.z};
      const float QF = s[0] * t3[0] + s[1] * t3[1] + s[2] * t3[2];
      const float coef = tab.gamma[kp], E = tab.eigen[kp];
      float* dst = b + (int64_t)i * 3 * M + 3 * kp;
#pragma unroll
      for (int a = 0; a < 3; ++a) dst[a] = kp == 0 ? -coef * t3[a] * QF : -coef * (s[a] - E * t3[a] * QF);
    }
  }
}

__global__ void k_force_terms(const Tables tab, int N, const float4* __restrict__ ori,
                              const float* __restrict__ ffpart, int nparts, float* __restrict__ F,
                              float* __restrict__ b) {
  const int64_t n = (int64_t)N * (tab.M + 1);
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.x * blockDim.x)
    force_term_unit(tab, N, ori, ffpart, nparts, F, b, u);
}

// ---- packed step: every member of a group (one Tables) in one launch ------
// Block b belongs to the member whose tile pairs it falls in; the member's
// blocks run exactly the single-suspension kernel's tile code, so a member's
// system is bit for bit the one k_assemble_pairs forms.
template <int MODE>
__global__ void __launch_bounds__(256, 3)
k_pack_assemble(const Tables tab, const PackStepMember* __restrict__ mem, int n) {
  const int L = (int)blockIdx.x;
  const PackStepMember& p = mem[pack_member_of(n, L, [&](int m) { return mem[m].asm_start; })];
  AsmOut out{};
  out.S32 = p.S32;
  out.S16 = p.S16;
  out.ffpart = p.ffpart;
  out.pos64 = p.pos64;
  int I, J;
  tile_pair(L - p.asm_start, I, J);
  assemble_pair_tile<5, 24, MODE, true>(tab, p.N, p.ori32, out, I, J);
}

// one block per member: its force terms and right-hand side
__global__ void __launch_bounds__(256) k_pack_force_terms(const Tables tab, const PackStepMember* __restrict__ mem) {
  const PackStepMember& p = mem[blockIdx.x];
  const int N = p.N;
  const int64_t n = (int64_t)N * (tab.M + 1);
  const int nparts = (N + AsmShape<5, 24>::TI - 1) / AsmShape<5, 24>::TI;
  for (int64_t u = threadIdx.x; u < n; u += blockDim.x) force_term_unit(tab, N, p.ori32, p.ffpart, nparts, p.F, p.b, u);
}

int launch_pack_assemble(const Tables& tab, const PackStepMember* members, int n, int64_t blocks, bool bf16,
                         cudaStream_t st) {
  if (tab.M != 5 || tab.Q != 24 || n < 1 || blocks < 1) return RF_E_UNSUPPORTED;
  constexpr size_t smem = NumShape<5, 24>::kSmem;
  if (bf16) {
    static const cudaError_t attr = cudaFuncSetAttribute(k_pack_assemble<kAsmStructBF16>,
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    RF_CUDA_TRY(attr);
    k_pack_assemble<kAsmStructBF16><<<(unsigned)blocks, NumShape<5, 24>::NT, smem, st>>>(tab, members, n);
  } else {
    static const cudaError_t attr = cudaFuncSetAttribute(k_pack_assemble<kAsmStructF16>,
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    RF_CUDA_TRY(attr);
    k_pack_assemble<kAsmStructF16><<<(unsigned)blocks, NumShape<5, 24>::NT, smem, st>>>(tab, members, n);
  }
  RF_LAUNCH_CHECK();
  k_pack_force_terms<<<(unsigned)n, 256, 0, st>>>(tab, members);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

// out[r] = sum over parts p of part[p][r], fixed order.
__global__ void k_reduce_rows(const float* __restrict__ part, int nparts, int64_t R, float* __restrict__ out) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < R; r += (int64_t)gridDim.x * blockDim.x) {
    float s = 0.f;
    for (int p = 0; p < nparts; ++p) s += part[(int64_t)p * R + r];
    out[r] = s;
  }
}

int launch_reduce_rows(const float* part, int nparts, int64_t R, float* out, cudaStream_t st) {
  const int threads = 256;
  const int blocks = (int)std::min<int64_t>(ceil_div(R, threads), 148 * 8);
  k_reduce_rows<<<blocks, threads, 0, st>>>(part, nparts, R, out);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

int assemble_tiles(int M, int Q, int N) { return (int)ceil_div(N, 192 / Q); }

int64_t struct_store_tiles(int N) {
  const int64_t T16 = ceil_div(N, kStoreTile);
  return T16 * (T16 + 1) / 2;
}

int64_t struct_floats32(int M, int N) {
  return struct_store_tiles(N) * (int64_t)kStoreTile * kStoreTile * (M + 1) * (M + 1) * 6;
}

int64_t struct_words16(int M, int N) {
  return struct_store_tiles(N) * (int64_t)kStoreTile * kStoreTile * s16_record_words(M);
}

template <int M, int Q, int MODE, bool P2>
static int launch_pairs(const Tables& tab, int N, const float4* ori, const AsmOut& out, cudaStream_t st) {
  using S = NumShape<M, Q>;
  const int64_t T = ceil_div(N, S::TI);
  // once per process (thread-safe static initialisation; handles of a serving
  // loop launch from several threads)
  static const cudaError_t attr = cudaFuncSetAttribute(k_assemble_pairs<M, Q, MODE, P2>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem);
  RF_CUDA_TRY(attr);
  k_assemble_pairs<M, Q, MODE, P2><<<(unsigned)(T * (T + 1) / 2), S::NT, S::kSmem, st>>>(tab, N, ori, out);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

template <int M, int Q>
static int launch_analytical(const Tables& tab, int N, const float4* ori, const AsmOut& out, cudaStream_t st) {
  using S = AsmShape<M, Q>;
  const int64_t T = ceil_div(N, S::TI);
  static const cudaError_t attr = cudaFuncSetAttribute(k_assemble_analytical<M, Q>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem);
  RF_CUDA_TRY(attr);
  k_assemble_analytical<M, Q><<<(unsigned)(T * T), S::NT, S::kSmem, st>>>(tab, N, ori, out);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

static int launch_force_terms(const Tables& tab, int N, const float4* ori, const AsmOut& out, float* F, float* b,
                              cudaStream_t st) {
  const int64_t n = (int64_t)N * (tab.M + 1);
  k_force_terms<<<(unsigned)std::min<int64_t>(ceil_div(n, 256), 148 * 8), 256, 0, st>>>(
      tab, N, ori, out.ffpart, assemble_tiles(tab.M, tab.Q, N), F, b);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

template <int MODE>
static int dispatch_assemble(const Tables& tab, int N, const float4* ori, const AsmOut& out, float* F, float* b,
                             int variant, cudaStream_t st) {
  if (variant < 0 || variant >= kAsmVariants) {
    set_last_error_str("assemble: unknown kernel variant");
    return RF_E_INPUT;
  }
  int rc = RF_E_UNSUPPORTED;
#define RF_ASM_CASE(MM, QQ)                                                              \
  if (tab.M == MM && tab.Q == QQ)                                                        \
    rc = variant == 1 ? launch_pairs<MM, QQ, MODE, true>(tab, N, ori, out, st)           \
                      : launch_pairs<MM, QQ, MODE, false>(tab, N, ori, out, st);
  RF_FOR_EACH_MQ(RF_ASM_CASE)
#undef RF_ASM_CASE
  if (rc == RF_E_UNSUPPORTED) set_last_error_str("assemble: (M, Q) combination not instantiated");
  if (rc != RF_OK) return rc;
  if (MODE == kAsmApply && out.x != nullptr) return RF_OK;   // the product: no force terms
  return launch_force_terms(tab, N, ori, out, F, b, st);
}

int launch_assemble_numerical(const Tables& tab, int N, const float4* pos, const float4* ori, const double4* pos64,
                              float* A, int64_t lda, float* ffpart, float* F, float* b, cudaStream_t st,
                              int variant) {
  AsmOut out{};
  out.pos64 = pos64;
  out.A = A;
  out.lda = lda;
  out.ffpart = ffpart;
  (void)pos;
  return dispatch_assemble<kAsmDense>(tab, N, ori, out, F, b, variant, st);
}

int launch_assemble_analytical(const Tables& tab, int N, const float4* pos, const float4* ori,
                               const double4* pos64, const double4* ori64, float* A, int64_t lda, float* ffpart,
                               float* F, float* b, cudaStream_t st) {
  AsmOut out{};
  out.pos64 = pos64;
  out.ori64 = ori64;
  out.A = A;
  out.lda = lda;
  out.ffpart = ffpart;
  int rc = RF_E_UNSUPPORTED;
#define RF_ASM_CASE(MM, QQ) \
  if (tab.M == MM && tab.Q == QQ) rc = launch_analytical<MM, QQ>(tab, N, ori, out, st);
  RF_FOR_EACH_MQ(RF_ASM_CASE)
#undef RF_ASM_CASE
  if (rc == RF_E_UNSUPPORTED) set_last_error_str("assemble: (M, Q) combination not instantiated");
  if (rc != RF_OK) return rc;
  return launch_force_terms(tab, N, ori, out, F, b, st);
}

int launch_assemble_apply(const Tables& tab, int N, const float4* pos, const float4* ori, const double4* pos64,
                          const float* x, float* zpart, const int* skip, float* ffpart, float* F, float* b,
                          cudaStream_t st, int variant) {
  AsmOut out{};
  out.pos64 = pos64;
  out.x = x;
  out.zpart = zpart;
  out.skip = skip;
  out.ffpart = ffpart;
  return dispatch_assemble<kAsmApply>(tab, N, ori, out, F, b, variant, st);
}

int launch_assemble_structured(const Tables& tab, int N, const float4* pos, const float4* ori, const double4* pos64,
                               float* S32, uint32_t* S16, bool bf16, float* ffpart, float* F, float* b,
                               cudaStream_t st, int variant) {
  AsmOut out{};
  out.pos64 = pos64;
  out.S32 = S32;
  out.S16 = S16;
  out.ffpart = ffpart;
  if (bf16) return dispatch_assemble<kAsmStructBF16>(tab, N, ori, out, F, b, variant, st);
  return dispatch_assemble<kAsmStructF16>(tab, N, ori, out, F, b, variant, st);
}

}  // namespace rf
