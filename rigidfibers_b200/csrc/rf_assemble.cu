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
#include <type_traits>

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
  static constexpr int K1 = M + 1;       // P_0..P_M
  static constexpr int NC = 6 * K1;      // G columns per unit (a point of i against a fiber j)
  // T of one pair as [value] padded so that 8 consecutive pairs start on
  // distinct banks that are multiples of 4 (stride = 4 * odd mod 32)
  static constexpr int TP = (K1 * K1 * 6 + 7) / 8 * 8 + 4;
  // structured storage
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
// instructions (add/mul/fma .f32x2); every rounding is the same as in the scalar
// form (all steps are explicit _rn operations, none can be contracted), so both
// give bit-identical G.  Either way the moments of P_2i and P_2i+1 accumulate in
// the two lanes against the weight pair W2[i][q] (the even part for P_2i, the
// odd part for P_2i+1), and their six components are recombined and stored as
// pairs: gcol[(i * 6 + c) * GS2] = (P_2i, P_2i+1).
// FAR: the rule of the far pairs (far_pts, far_W2) instead of the full one, with a
// Newton step on the reciprocal root (NEWTON) or with a0 taken off A_0 from the start.

// the point (x, y, z) on t's axis: d and s*
__device__ __forceinline__ float4 project(float x, float y, float z, const float4 t) {
  float ss = fmaf(x, t.x, fmaf(y, t.y, z * t.z));
  float dx = fmaf(-ss, t.x, x), dy = fmaf(-ss, t.y, y), dz = fmaf(-ss, t.z, z);
  const float dl = fmaf(dx, t.x, fmaf(dy, t.y, dz * t.z));
  ss += dl;
  dx = fmaf(-dl, t.x, dx);
  dy = fmaf(-dl, t.y, dy);
  dz = fmaf(-dl, t.z, dz);
  return make_float4(dx, dy, dz, ss);
}

// 2 / |x_i - x_j|
__device__ __forceinline__ float mean_kernel(float x, float y, float z) {
  return 2.f * rsqrtf(fmaf(x, x, fmaf(y, y, z * z)));
}

// d: project() of the point
template <int K1, int Q, int GS2, bool P2, bool FAR, bool NEWTON = false>
__device__ __forceinline__ void stokeslet_moments_G(const Tables& tab, const float4 d, const float4 tj, float e2,
                                                    float e2x3, float a0, float2* __restrict__ gcol) {
  static_assert(P2 || !FAR, "the far rule runs packed");
  constexpr int H = Q / 2, KP = (K1 + 1) / 2;
  const float* const pts = FAR ? tab.far_pts : tab.pts;
  const float dx = d.x, dy = d.y, dz = d.z, ss = d.w;
  const float dd = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  float2 mA[KP], m0[KP], m1[KP], m2[KP];
#pragma unroll
  for (int i = 0; i < KP; ++i) mA[i] = m0[i] = m1[i] = m2[i] = make_float2(0.f, 0.f);
  if (FAR) mA[0].x = -a0;
  // the full rule's 12 folded points unrolled whole would spill
  constexpr int kUnroll = FAR ? H : 3;
#pragma unroll kUnroll
  for (int q = 0; q < H; ++q) {
    float2 fa, fb, fc, fd;   // lane x: point q, lane y: point Q-1-q
    if constexpr (P2) {
      const float2 u = __fadd2_rn(make_float2(ss, ss), make_float2(-pts[q], -pts[Q - 1 - q]));
      const float2 r2 = __ffma2_rn(u, u, make_float2(dd, dd));
      float2 inv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
      if constexpr (NEWTON) {
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
    // (even, odd) parts
    const float2 ga = make_float2(__fadd_rn(fa.x, fa.y), __fsub_rn(fa.x, fa.y));
    const float2 gb = make_float2(__fadd_rn(fb.x, fb.y), __fsub_rn(fb.x, fb.y));
    const float2 gc = make_float2(__fadd_rn(fc.x, fc.y), __fsub_rn(fc.x, fc.y));
    const float2 gd = make_float2(__fadd_rn(fd.x, fd.y), __fsub_rn(fd.x, fd.y));
#pragma unroll
    for (int i = 0; i < KP; ++i) {
      const float2 w = FAR ? tab.far_W2[i][FAR ? q : 0] : tab.W2[i][q];
      mA[i] = __ffma2_rn(ga, w, mA[i]);
      m0[i] = __ffma2_rn(gb, w, m0[i]);
      m1[i] = __ffma2_rn(gc, w, m1[i]);
      m2[i] = __ffma2_rn(gd, w, m2[i]);
    }
  }
  // components in the order (11, 22, 33, 12, 13, 23)
  const float Dd[6] = {dx * dx, dy * dy, dz * dz, dx * dy, dx * dz, dy * dz};
  const float Sd[6] = {2.f * dx * tj.x, 2.f * dy * tj.y, 2.f * dz * tj.z, fmaf(dx, tj.y, dy * tj.x),
                       fmaf(dx, tj.z, dz * tj.x), fmaf(dy, tj.z, dz * tj.y)};
  const float Tt[6] = {tj.x * tj.x, tj.y * tj.y, tj.z * tj.z, tj.x * tj.y, tj.x * tj.z, tj.y * tj.z};
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const float2 D2 = make_float2(Dd[c], Dd[c]), S2 = make_float2(Sd[c], Sd[c]), T2 = make_float2(Tt[c], Tt[c]);
#pragma unroll
    for (int i = 0; i < KP; ++i) {
      const float2 t = c < 3 ? __ffma2_rn(m2[i], T2, mA[i]) : __fmul2_rn(m2[i], T2);
      gcol[(i * 6 + c) * GS2] = __ffma2_rn(m0[i], D2, __ffma2_rn(m1[i], S2, t));
    }
  }
}

// ---------------------------------------------------------------------------
// Numerical pair tiles: TI x TI fibers, unordered pairs, both blocks of a pair
// from one evaluation of K.  A pair whose centres are at least sqrt(far_d2)
// apart takes the far rule, the kFarNodes-point Gauss rule of the quadrature's
// own discrete measure (make_tables), on both fibers: 64 kernel evaluations
// instead of Q^2 = 576, within 3e-10 of the full rule's blocks (below their
// FP32 rounding).  The others take the full rule.
//
// A third of the points average the roundings of G a third as well, and the blocks
// of P_1 and up against P_0 (the right-hand side) are small differences of G.  A
// Newton step on the reciprocal root makes up for it in sums over hundreds of pairs
// (forces of 400 dilute fibers against 64 bits: 1.7e-6, 2.1e-6 without the far rule),
// not in smaller ones (nine packs of 8 and 12 members: 1.27e-6 against 1.16e-6).
// Up to kFarSmall fibers what all points of fiber i share is therefore taken out of
// the sums: a point's projection on fiber j's axis is the centre difference's plus s
// times t_i's, and 2 / |x_i - x_j|, about the sum of W_0 a, is taken off G[.][P_0]'s
// diagonal components where their sum starts and put back into T[P_0][P_0]
// (far_sum).  Roundings of T[k][P_0], k = 1 .. 5, times the distance (FP32 emulation):
// 3.9 5.6 2.3 2.9 1.8 e-8 by the full rule, 5.2 5.2 3.5 3.6 2.8 by the far rule with
// the step, 4.1 3.3 2.8 2.3 2.3 so (the step is left out); the packs' forces 0.98e-6.
// Larger systems and the product keep the step, with which their errors are below
// the full rule's; the choice costs them 0.7 % of the assembly (N=4000: 2.44 ms).
//
// Bound: FP32 issue in the matrix-free product, HBM stores in the structured
// assembly.  The far pairs run in batches of whole j (2 or 4 of the tile: 16 or
// 32 pairs x 8 points = the CTA's threads), so that every phase has one unit per
// thread and lane = pair keeps shared memory free of conflicts; the near pairs
// of those rows are compacted and run in groups of up to TI pairs x Q points.
// ---------------------------------------------------------------------------
constexpr int kFarSmall = kPackMaxFibers;

// Threads per CTA.  Structured output: 128 (six CTAs per SM instead of three of
// 256: barriers of four warps, more CTAs to fill them; N=4000 3.09 -> 2.42 ms).
// Matrix-free product and dense output: 256, where the product's 160 and the
// block stores' 800 tasks of a batch split better (N=2500 product 0.90 against
// 1.23 ms, N=2000 dense 1.55 against 1.77).  More than 5 terms: batches of 16
// pairs, since G and T of 32 would leave one CTA per SM, on 128 threads; on 192 for
// the product, which takes 8 near pairs at once then instead of 5 (whole steps of 37
// and 1500 fibers, 6 terms: 0.43 and 10.5 ms against 0.50 and 10.9); on 256 for 8
// terms, whose 144 force-term sums of a batch need a thread each (whole matrix-free
// steps of 37 and 1500 fibers: 0.54 and 18.2 ms, with 160 threads 0.68 and 19.7).
constexpr int num_threads(int M, int mode) {
  return M > 7 ? 256 : mode == kAsmStructF16 || mode == kAsmStructBF16 ? 128 : M <= 5 ? 256 : mode == kAsmApply ? 192 : 128;
}
constexpr int min_ctas(int M, int mode) {
  const int threads = num_threads(M, mode);
  return M > 7 ? 2 : threads == 192 ? 3 : M > 5 ? 4 : threads == 128 ? 6 : 3;
}

template <int M, int Q, int NTH>
struct NumShape {
  using A = AsmShape<M, Q>;
  static constexpr int TI = A::TI, K1 = A::K1, NQ32 = A::NQ32;
  static constexpr int KP = (K1 + 1) / 2;                  // Legendre index pairs (2i, 2i + 1) of fiber j
  static constexpr int NC2 = 6 * KP;                       // G columns, pairs of floats
  static constexpr int NT = NTH;
  static constexpr int FN = kFarNodes;
  static constexpr int FB = (M > 5 ? 128 : NT) / FN;
  static constexpr int PB = FB < TI * TI ? FB : TI * TI;   // far pairs per batch
  static constexpr int JB = PB / TI;                       // j of a batch
  static constexpr int GSF = PB * FN + PB % 32;            // G column stride (float2): lanes (col, pair)
  static constexpr int NS = NT / Q < TI ? NT / Q : TI;     // near pairs per group
  static constexpr int QP = Q + 1;                         // near: float2 per slot of a G column
  static constexpr int GSN = NS * QP + (NS * QP + 1) % 2;  // odd: lanes = columns
  static constexpr int GFLOATS = (2 * NC2 * (GSF > GSN ? GSF : GSN) + 3) / 4 * 4;
  // T of a batch.  Structured and matrix-free: [jj][value][i], the storage
  // record's own order (s32_block), so one j is the contiguous run that a bulk
  // copy stores; the j stride is TI past a multiple of 16 words so that a
  // batch's pairs write distinct banks.  Dense: [pair][row, col, component].
  static constexpr int JS = NQ32 * TI + TI;
  static constexpr int TP = A::TP;
  static constexpr int TFLOATS = JB * JS > PB * TP ? JB * JS : PB * TP;
  static constexpr size_t kSmem = sizeof(float) * (GFLOATS + TFLOATS);
  static_assert(PB % TI == 0 && TI % JB == 0 && 32 % PB == 0, "batches are whole j and part of one mask word");
  static_assert(PB * FN <= NT && PB * K1 <= NT, "a far point and an i-side sum (force terms, or fewer: z) per thread");
  static_assert(JS % 4 == 0 && NQ32 * TI % 4 == 0, "a j's values are copied out from a 16-byte boundary");
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
  using S = NumShape<M, Q, num_threads(M, MODE)>;
  constexpr int TI = S::TI, K1 = S::K1, NC2 = S::NC2, NT = S::NT, PB = S::PB, JB = S::JB, TP = S::TP, JS = S::JS;
  constexpr int NQ32 = S::NQ32;
  constexpr int M3 = 3 * M;
  constexpr int FF = K1 * 3;   // force-term floats per fiber
  constexpr bool STRUCT = MODE == kAsmStructF16 || MODE == kAsmStructBF16;
  constexpr bool APPLY = MODE == kAsmApply;
  constexpr bool QT = MODE != kAsmDense;   // T as [jj][value][i]
  static_assert(Q % 2 == 0, "mirror folding needs an even number of quadrature points");

  __shared__ float4 sTi[TI], sTj[TI];        // orientations
  __shared__ float sD[TI * TI][3];           // pair jl * TI + il: x_i - x_j, formed in FP64 and rounded once
  __shared__ unsigned char sKind[TI * TI];   // 0: no such pair, 1: far, 2: near
  __shared__ unsigned char sNear[TI * TI];   // the near pairs, in pair order
  __shared__ unsigned sMask[(TI * TI + 31) / 32];   // near pairs as bits
  extern __shared__ __align__(16) float smem_dyn[];
  float2* const sG = reinterpret_cast<float2*>(smem_dyn);
  float* const sT = smem_dyn + S::GFLOATS;
  __shared__ float sCoef[kMaxTerms], sEig[kMaxTerms];
  __shared__ float sFj[TI * FF];             // force terms of the tile's j

  const bool diag = (I == J);
  const bool small = !APPLY && N <= kFarSmall;
  const int tid = threadIdx.x, lane = tid & 31;
  const int i0 = I * TI, j0 = J * TI;
  // kAsmApply with a vector applies the blocks; without one it forms the force terms
  const bool do_apply = APPLY && out.x != nullptr;
  constexpr int XW = APPLY ? TI * M3 : 1;
  __shared__ float sXi[XW], sXj[XW], sZj[XW];   // x rows of the I and J tiles, z of this tile's j

  if (tid < M) { sCoef[tid] = tab.gamma[tid]; sEig[tid] = tab.eigen[tid]; }
  if (tid < TI) {
    sTi[tid] = ori[min(i0 + tid, N - 1)];
    sTj[tid] = ori[min(j0 + tid, N - 1)];
  }
  for (int pr0 = 0; pr0 < TI * TI; pr0 += NT) {
    // the separation of quadrature points is formed as (x_i - x_j) + s_qi t_i -
    // s_qj t_j with the centre difference taken in FP64 and rounded once, so
    // its error scales with the fibers' distance rather than with their
    // distance from the origin (FP32 points x + s t far from the origin lose
    // ~1e-6 absolutely, which for nearly touching fibers is ~1e-4 of the kernel)
    const int pr = pr0 + tid;
    bool near_pair = false;
    if (pr < TI * TI) {
      const int il = pr % TI, jl = pr / TI;
      const double4 xi = out.pos64[min(i0 + il, N - 1)], xj = out.pos64[min(j0 + jl, N - 1)];
      const float dx = (float)(xi.x - xj.x), dy = (float)(xi.y - xj.y), dz = (float)(xi.z - xj.z);
      sD[pr][0] = dx;
      sD[pr][1] = dy;
      sD[pr][2] = dz;
      const bool valid = i0 + il < N && j0 + jl < N && (!diag || il < jl);
      near_pair = valid && !far_pair(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), tab.far_d2);
      sKind[pr] = near_pair ? 2 : valid ? 1 : 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, near_pair);
    if (lane == 0 && pr < TI * TI) sMask[pr / 32] = m;
  }
  if constexpr (APPLY) {
    if (do_apply) {
      for (int k = tid; k < TI * M3; k += NT) {
        const int f = k / M3, c = k % M3;
        sXi[k] = i0 + f < N ? out.x[(int64_t)(i0 + f) * M3 + c] : 0.f;
        sXj[k] = j0 + f < N ? out.x[(int64_t)(j0 + f) * M3 + c] : 0.f;
      }
    }
  }
  const float e2 = tab.e2;
  const float e2x3 = -3.f * e2;
  const float fz = tab.fz_half;
  __syncthreads();
  for (int pr = tid; pr < TI * TI; pr += NT)   // read after the barriers of the first batch
    if (sKind[pr] == 2) {
      int at = __popc(sMask[pr / 32] & ((1u << lane) - 1));
      for (int w = 0; w < pr / 32; ++w) at += __popc(sMask[w]);
      sNear[at] = (unsigned char)pr;
    }

  // structured storage: the record of j = j0 + jl is rec0 + jl
  constexpr int SUB = kStoreTile / TI;
  const int64_t rec0 =
      (((int64_t)(J / SUB) * (J / SUB + 1) / 2 + I / SUB) * SUB * SUB + (I % SUB) * SUB + (J % SUB)) * TI;

  // phase 2: T[ki][kj][c] = sum_qi W[ki][qi] G[qi][c][kj], folded over qi, for the
  // two kj of column (i, c) in the lanes of packed FP32 instructions, into the
  // pair's T at dst (stride QS per value); lo - hi as fma(hi, -1, lo): the same
  // rounding as a scalar subtraction
  auto contract = [&](const float2* g, auto points, auto far, int stride, int col, float* dst) {
    constexpr int NQ = decltype(points)::value;
    constexpr bool FAR = decltype(far)::value;
    constexpr int QS = QT ? TI : 1;
    float2 acc[K1];
#pragma unroll
    for (int k = 0; k < K1; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < NQ / 2; ++q) {
      const float2 lo = g[q * stride], hi = g[(NQ - 1 - q) * stride];
      const float2 ev = __fadd2_rn(lo, hi), od = __ffma2_rn(hi, make_float2(-1.f, -1.f), lo);
#pragma unroll
      for (int k = 0; k < K1; ++k) {
        const float w = FAR ? tab.far_W[k][FAR ? q : 0] : tab.W[k][q];
        acc[k] = __ffma2_rn((k & 1) ? od : ev, make_float2(w, w), acc[k]);
      }
    }
    const int i = col / 6, c = col % 6;
#pragma unroll
    for (int lane2 = 0; lane2 < 2; ++lane2) {
      const int kj = 2 * i + lane2;
      if (lane2 == 1 && K1 % 2 == 1 && kj == K1) break;   // odd M + 1: no such index
      // block (k, kj): dense order k K1 + kj; storage order s32_block
      const int b0 = QT ? M * M + kj : kj;                                     // k = 0
      const int b1 = QT ? (kj > 0 ? kj - 1 : M * M + K1) : K1 + kj;            // k = 1
      const int bs = QT ? (kj > 0 ? M : 1) : K1;                               // per k after that
#pragma unroll
      for (int k = 0; k < K1; ++k)
        dst[((k == 0 ? b0 : b1 + (k - 1) * bs) * 6 + c) * QS] = lane2 == 0 ? acc[k].x : acc[k].y;
    }
  };
  auto t_of = [&](int jj, int il) { return QT ? sT + jj * JS + il : sT + (jj * TI + il) * TP; };

  // i-side sums of task (jj, k, il) = this thread, over the batches: force
  // terms (k <= M) or z (k < M)
  float iacc[3] = {0.f, 0.f, 0.f};
  const int jcount = min(TI, N - j0);
  int near0 = 0;   // near pairs of the batches done

  for (int jb = 0; jb < jcount; jb += JB) {
    // ---- far pairs.  Phase 1: G[c][k] = sum_qj K_c(qi, qj) W[k][qj], unit
    // u = qi * PB + pair; zeros for the others
    if (tid < PB * S::FN) {
      const int p = tid % PB, qi = tid / PB;
      const int pr = jb * TI + p;
      float2* const gcol = sG + tid;
      if (sKind[pr] == 1) {
        const float4 ti = sTi[pr % TI], tj = sTj[pr / TI];
        const float si = tab.far_pts[qi];
        const float dx = sD[pr][0], dy = sD[pr][1], dz = sD[pr][2];
        if (small) {
          const float4 d = project(dx, dy, dz, tj), e = project(ti.x, ti.y, ti.z, tj);
          stokeslet_moments_G<K1, S::FN, S::GSF, true, true>(
              tab, make_float4(fmaf(si, e.x, d.x), fmaf(si, e.y, d.y), fmaf(si, e.z, d.z), fmaf(si, e.w, d.w)), tj, e2,
              e2x3, mean_kernel(dx, dy, dz), gcol);
        } else {
          stokeslet_moments_G<K1, S::FN, S::GSF, true, true, true>(
              tab, project(fmaf(si, ti.x, dx), fmaf(si, ti.y, dy), fmaf(si, ti.z, dz), tj), tj, e2, e2x3, 0.f, gcol);
        }
      } else {
#pragma unroll
        for (int c = 0; c < NC2; ++c) gcol[c * S::GSF] = make_float2(0.f, 0.f);
      }
    }
    // T of the last batch has left shared memory before phase 2 overwrites it
    if (STRUCT && tid < JB) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncthreads();
    // phase 2, lanes = pairs
    for (int task = tid; task < PB * NC2; task += NT) {
      const int col = task / PB, p = task % PB;
      contract(sG + col * S::GSF + p, std::integral_constant<int, S::FN>(), std::true_type(), PB, col,
               t_of(p / TI, p % TI));
    }
    if (small && tid < 3 * PB) {   // what P_0's diagonal components lack, in this thread's first column
      const int col = tid / PB, p = tid % PB, pr = jb * TI + p;
      float* const t = t_of(p / TI, p % TI);
      const float a0 = sKind[pr] == 1 ? mean_kernel(sD[pr][0], sD[pr][1], sD[pr][2]) : 0.f;
#pragma unroll
      for (int k = 0; k < K1; k += k == 0 ? 6 : 2)   // the sums of W_2 and W_4 are 0
        t[((QT ? s32_block(M, k, 0) : k * K1) * 6 + col) * (QT ? TI : 1)] += a0 * tab.far_sum[k];
    }
    // ---- near pairs of these rows, in groups of up to NS, into the same T
    const unsigned bits = (sMask[jb * TI / 32] >> (jb * TI % 32)) & (PB == 32 ? 0xffffffffu : (1u << PB % 32) - 1u);
    const int near1 = near0 + __popc(bits);
    for (int n0 = near0; n0 < near1; n0 += S::NS) {
      const int cnt = min(S::NS, near1 - n0);
      __syncthreads();   // G is read
      if (tid < cnt * Q) {
        const int slot = tid / Q, qi = tid % Q;
        const int pr = sNear[n0 + slot];
        const float4 ti = sTi[pr % TI], tj = sTj[pr / TI];
        const float si = tab.pts[qi];
        const float px = fmaf(si, ti.x, sD[pr][0]), py = fmaf(si, ti.y, sD[pr][1]), pz = fmaf(si, ti.z, sD[pr][2]);
        stokeslet_moments_G<K1, Q, S::GSN, P2, false>(tab, project(px, py, pz, tj), tj, e2, e2x3, 0.f,
                                                      sG + slot * S::QP + qi);
      }
      __syncthreads();
      for (int task = tid; task < cnt * NC2; task += NT) {   // lanes = columns
        const int slot = task / NC2, col = task % NC2;
        const int pr = sNear[n0 + slot];
        contract(sG + col * S::GSN + slot * S::QP, std::integral_constant<int, Q>(), std::false_type(), 1, col,
                 t_of(pr / TI - jb, pr % TI));
      }
    }
    near0 = near1;
    // the bulk copy below reads T through the async proxy
    if (STRUCT) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    // ---- phase 3: the batch's blocks to their destination (the next batch's
    // phase 1 writes G only, and its phase 2 follows a barrier).  Pairs that do
    // not exist (i >= N, i >= j on a diagonal tile) came out as exact zeros
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
        if (!sKind[jl * TI + tl]) continue;
        dense_block(dst, out.lda, t_of(jj, tl) + ((kIp + 1) * K1 + kJp + 1) * 6, sTi[tl], kIp, sCoef[kIp], sEig[kIp]);
      }
      // block (j, i): rows of fiber j, columns of fiber i
      for (int task = tid; task < PB * M * M; task += NT) {
        const int jj = task / (TI * M * M), r0 = task % (TI * M * M);
        const int tl = r0 / (M * M), rem = r0 % (M * M);
        const int kIp = rem / M, kJp = rem % M, jl = jb + jj;
        if (!sKind[jl * TI + tl]) continue;
        float* dst = out.A + (int64_t)((j0 + jl) * M3 + 3 * kJp) + (int64_t)((i0 + tl) * M3 + 3 * kIp) * out.lda;
        dense_block(dst, out.lda, t_of(jj, tl) + ((kIp + 1) * K1 + kJp + 1) * 6, sTj[jl], kJp, sCoef[kJp], sEig[kJp]);
      }
    } else if constexpr (STRUCT) {
      // FP32: one bulk copy per j (no FP32 copy in the recompute modes: out.S32 null)
      const int jn = min(JB, jcount - jb);
      if (out.S32 != nullptr && tid < jn) {
        const float* dst = out.S32 + (rec0 + jb + tid) * (int64_t)(NQ32 * TI);
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                     "r"(static_cast<uint32_t>(__cvta_generic_to_shared(sT + tid * JS))), "r"(NQ32 * TI * 4)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      // 16-bit records [i][NW]: the M^2 operator blocks, which lead the FP32
      // record, two values per word; lane = pair
      constexpr int NW = s16_record_words(M), NQ16 = AsmShape<M, Q>::NQ16;
      uint32_t* d16 = out.S16 + (rec0 + jb) * (int64_t)(NW * TI);
      for (int v = tid; v < PB * (NW / 4); v += NT) {
        const int p = v % PB, w4 = v / PB;
        if (p / TI >= jn) continue;
        const float* t = t_of(p / TI, p % TI) + 8 * w4 * TI;
        uint32_t w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool in = NQ16 % 4 == 0 || 4 * w4 + u < NQ16;
          const float lo = in ? t[2 * u * TI] : 0.f, hi = in ? t[(2 * u + 1) * TI] : 0.f;
          if constexpr (MODE == kAsmStructF16) {
            __half2 hv = __floats2half2_rn(lo, hi);
            w[u] = *reinterpret_cast<uint32_t*>(&hv);
          } else {
            __nv_bfloat162 hv = __floats2bfloat162_rn(lo, hi);
            w[u] = *reinterpret_cast<uint32_t*>(&hv);
          }
        }
        *reinterpret_cast<uint4*>(&d16[p * NW + 4 * w4]) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    // i side: sums over the thread's own j of each batch; j side: sums over the
    // tile's i by halving shuffles in groups of TI lanes
    const unsigned grp = ((1u << TI) - 1u) << (lane & ~(TI - 1));
    if (APPLY && do_apply) {
      if constexpr (APPLY) {
        // z_i[k] += T(k+1, l+1) x_j[l], z_j[k] += T(l+1, k+1) x_i[l] (blocks symmetric)
        for (int task = tid; task < 2 * PB * M; task += NT) {
          const bool iside = task < PB * M;
          const int u = iside ? task : task - PB * M;
          const int jj = u / (TI * M), k = (u / TI) % M, tl = u % TI, jl = jb + jj;
          const float* xv = iside ? sXj + jl * M3 : sXi + tl * M3;
          const float* t = t_of(jj, tl) + (iside ? k * M : k) * 6 * TI;
          const int ts = (iside ? 1 : M) * 6 * TI;
          float zs[3] = {0.f, 0.f, 0.f};
#pragma unroll
          for (int l = 0; l < M; ++l) {
            const float* b = t + l * ts;
            const float T6[6] = {b[0], b[TI], b[2 * TI], b[3 * TI], b[4 * TI], b[5 * TI]};
#pragma unroll
            for (int a = 0; a < 3; ++a)
              zs[a] = fmaf(sym_get(T6, a, 0), xv[3 * l],
                           fmaf(sym_get(T6, a, 1), xv[3 * l + 1], fmaf(sym_get(T6, a, 2), xv[3 * l + 2], zs[a])));
          }
          if (iside) {
#pragma unroll
            for (int a = 0; a < 3; ++a) iacc[a] += zs[a];
          } else {
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
        const int blk = QT ? (iside ? s32_block(M, k, 0) : s32_block(M, 0, k)) : (iside ? k * K1 : k);
        constexpr int QS = QT ? TI : 1;
        const float* t = t_of(jj, tl) + blk * 6 * QS;
        float f3[3] = {t[4 * QS], t[5 * QS], t[2 * QS]};
        if (iside) {
#pragma unroll
          for (int a = 0; a < 3; ++a) iacc[a] = fmaf(f3[a], fz, iacc[a]);
        } else {
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
  if (STRUCT && tid < JB) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");

  // ---- i-side sums over the JB rows of a batch (G is free: its last readers
  // passed a barrier), then the partial rows, each written exactly once
  float* const red = smem_dyn;
  if (APPLY && do_apply) {
    if constexpr (APPLY) {
      if (tid < PB * M) {
        const int jj = tid / (TI * M), k = (tid / TI) % M, tl = tid % TI;
#pragma unroll
        for (int a = 0; a < 3; ++a) red[(jj * TI + tl) * M3 + 3 * k + a] = iacc[a];
      }
      __syncthreads();
      // the i side of tile (I, J) to slot J, the j side to slot I (a diagonal
      // tile's j side to the slot after the last tile)
      const int64_t R = (int64_t)M3 * N;
      float* zi = out.zpart + (int64_t)J * R + (int64_t)i0 * M3;
      float* zj = out.zpart + (int64_t)(diag ? (N + TI - 1) / TI : I) * R + (int64_t)j0 * M3;
      for (int u = tid; u < TI * M3; u += NT) {
        float v = red[u];
#pragma unroll
        for (int jj = 1; jj < JB; ++jj) v += red[jj * TI * M3 + u];
        if (i0 + u / M3 < N) zi[u] = v;
        if (j0 + u / M3 < N) zj[u] = sZj[u];
      }
    }
    return;
  }
  if (tid < PB * K1) {
    const int jj = tid / (TI * K1), k = (tid / TI) % K1, tl = tid % TI;
#pragma unroll
    for (int a = 0; a < 3; ++a) red[(jj * TI + tl) * FF + 3 * k + a] = iacc[a];
  }
  __syncthreads();
  // partial force terms ffpart[X][fiber of Y][k][3]
  for (int u = tid; u < TI * FF; u += NT) {
    float v = red[u];
#pragma unroll
    for (int jj = 1; jj < JB; ++jj) v += red[jj * TI * FF + u];
    const bool jin = j0 + u / FF < N;
    if (diag && jin) v += sFj[u];
    if (i0 + u / FF < N) out.ffpart[((int64_t)J * N + i0) * FF + u] = v;
    if (!diag && jin) out.ffpart[((int64_t)I * N + j0) * FF + u] = sFj[u];
  }
}

template <int M, int Q, int MODE, bool P2>
__global__ void __launch_bounds__(num_threads(M, MODE), min_ctas(M, MODE))
k_assemble_pairs(const Tables tab, int N, const float4* __restrict__ ori, AsmOut out) {
  if (MODE == kAsmApply && out.skip != nullptr && *out.skip) return;
  int I, J;
  tile_pair(blockIdx.x, I, J);
  assemble_pair_tile<M, Q, MODE, P2>(tab, N, ori, out, I, J);
}

// ---------------------------------------------------------------------------
// Analytical assembly: ordered pairs (the inner integral over fiber j is exact,
// the outer one over fiber i a quadrature, so the blocks of (i, j) and (j, i)
// are different numbers), dense output only.  Bound: FP64 issue and latency of
// the closed form (analytic_G), so far pairs evaluate it at the far rule's 8
// outer points instead of Q (the outer integrand is as smooth as the numerical
// path's).  One launch: the first N blocks take the near pairs of one fiber i
// each, the others the far pairs of a tile; kept apart, neither waits for the
// other's barriers.  N=777, one B200: 4.09 ms with Q points for every pair and
// divisions in analytic_G, 1.70 ms with the near pairs inside the tiles.
// ---------------------------------------------------------------------------
template <int M, int Q>
struct AnaShape {
  using A = AsmShape<M, Q>;
  static constexpr int TI = A::TI, K1 = A::K1, NC = A::NC, TP = A::TP;
  static constexpr int NT = 192;
  static constexpr int FN = kFarNodes;
  static constexpr int JB = TI == 8 ? 3 : TI == 4 ? 4 : 1;   // rows of a far batch: PB x FN <= NT units
  static constexpr int PB = JB * TI;
  static constexpr int GSF = (PB * FN + 31) / 32 * 32 + PB;  // lanes (column, pair)
  static constexpr int NS = 192 / Q;                         // near pairs per group
  static constexpr int QP = Q + 1;
  static constexpr int GSN = NS * QP + (NS * QP + 1) % 2;    // near: lanes = columns
  static constexpr int GFLOATS = (NC * (GSF > GSN ? GSF : GSN) + 3) / 4 * 4;
  static constexpr size_t kSmem = sizeof(float) * (GFLOATS + (PB > NS ? PB : NS) * TP);
  static_assert(PB * FN <= NT && NS * Q <= NT, "one unit per thread");
};

// the closed-form integrals G[c][k] over fiber j for the point s of fiber i, into
// column k * 6 + c of g (column stride cs)
template <int M>
__device__ __forceinline__ void closed_form(const AsmOut& out, float eps, int i, int j, float s, float* g, int cs) {
  const double4 xi = out.pos64[i], ti = out.ori64[i], xj = out.pos64[j], tj4 = out.ori64[j];
  const double sd = (double)s;
  const double R0[3] = {xi.x + sd * ti.x - xj.x, xi.y + sd * ti.y - xj.y, xi.z + sd * ti.z - xj.z};
  const double tj[3] = {tj4.x, tj4.y, tj4.z};
  float v[6][M + 1];
  analytic_G<M>(R0, tj, 2.0 * (double)eps * (double)eps, v);
#pragma unroll
  for (int c = 0; c < 6; ++c)
#pragma unroll
    for (int k = 0; k <= M; ++k) g[(k * 6 + c) * cs] = v[c][k];
}

// dst[k * NC] = sum_qi W[k][qi] g[qi * stride], folded over qi
template <int K1, int NQ, bool FAR>
__device__ __forceinline__ void fold_points(const Tables& tab, const float* g, int stride, float* dst) {
  float acc[K1];
#pragma unroll
  for (int k = 0; k < K1; ++k) acc[k] = 0.f;
#pragma unroll 4
  for (int q = 0; q < NQ / 2; ++q) {
    const float lo = g[q * stride], hi = g[(NQ - 1 - q) * stride];
    const float ev = __fadd_rn(lo, hi), od = __fsub_rn(lo, hi);
#pragma unroll
    for (int k = 0; k < K1; ++k)
      acc[k] = __fmaf_rn((k & 1) ? od : ev, FAR ? tab.far_W[k][FAR ? q : 0] : tab.W[k][q], acc[k]);
  }
#pragma unroll
  for (int k = 0; k < K1; ++k) dst[k * 6 * K1] = acc[k];
}

__device__ __forceinline__ float centre_dist2(const double4& a, const double4& b) {
  const float dx = (float)(a.x - b.x), dy = (float)(a.y - b.y), dz = (float)(a.z - b.z);
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// The near pairs (i, j) of fiber i, found NT centres at a time and taken in index
// order in groups of NS; their force terms to partial row T
template <int M, int Q>
__device__ __forceinline__ void analytical_near(const Tables& tab, int N, const float4* __restrict__ ori,
                                                const AsmOut& out, int i, int T, float* smem) {
  using S = AnaShape<M, Q>;
  constexpr int K1 = S::K1, NC = S::NC, TP = S::TP, NT = S::NT, NS = S::NS, M3 = 3 * M, FF = 3 * K1;
  constexpr int QUEUE = NT + NS;
  __shared__ int queue[QUEUE];
  __shared__ int warp_near[NT / 32];
  float* const sG = smem;
  float* const sT = smem + S::GFLOATS;   // [slot][TP]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double4 xi = out.pos64[i];
  float facc = 0.f;                      // component tid % 3 of F_i[tid / 3]
  int count = 0;
  for (int js = 0; js < N; js += NT) {
    const int j = js + tid;
    const bool near = j < N && j != i && !far_pair(centre_dist2(xi, out.pos64[j]), tab.far_d2);
    const unsigned m = __ballot_sync(0xffffffffu, near);
    if (lane == 0) warp_near[warp] = __popc(m);
    __syncthreads();
    int at = count, total = count;
    for (int w = 0; w < NT / 32; ++w) {
      if (w < warp) at += warp_near[w];
      total += warp_near[w];
    }
    if (near) queue[at + __popc(m & ((1u << lane) - 1))] = j;
    __syncthreads();
    count = total;
    const bool last = js + NT >= N;
    int done = 0;
    for (; count - done >= NS || (last && done < count); done += NS) {
      const int cnt = min(NS, count - done);
      if (tid < cnt * Q) {
        const int slot = tid / Q, qi = tid % Q;
        closed_form<M>(out, tab.eps, i, queue[done + slot], tab.pts[qi], sG + slot * S::QP + qi, S::GSN);
      }
      __syncthreads();
      for (int task = tid; task < cnt * NC; task += NT) {   // lanes = columns
        const int slot = task / NC, col = task % NC;
        fold_points<K1, Q, false>(tab, sG + col * S::GSN + slot * S::QP, 1, sT + slot * TP + col);
      }
      __syncthreads();
      for (int task = tid; task < cnt * M * M; task += NT) {
        const int slot = task / (M * M), kJp = task % (M * M) / M, kIp = task % M;
        float* dst = out.A + (int64_t)i * M3 + 3 * kIp + ((int64_t)queue[done + slot] * M3 + 3 * kJp) * out.lda;
        dense_block(dst, out.lda, sT + slot * TP + ((kIp + 1) * K1 + kJp + 1) * 6, ori[i], kIp, tab.gamma[kIp],
                    tab.eigen[kIp]);
      }
      if (tid < FF) {
        const int a = tid % 3;
        for (int slot = 0; slot < cnt; ++slot)
          facc = fmaf(sT[slot * TP + (tid / 3) * NC + (a == 0 ? 4 : a == 1 ? 5 : 2)], tab.fz_half, facc);
      }
      __syncthreads();
    }
    // what is left of the queue (fewer than NS) to its front
    const int left = max(0, count - done);
    const int keep = tid < left ? queue[done + tid] : 0;
    __syncthreads();
    if (tid < left) queue[tid] = keep;
    count = left;
  }
  if (tid < FF) out.ffpart[((int64_t)T * N + i) * FF + tid] = facc;
}

template <int M, int Q>
__global__ void __launch_bounds__(192, 2)
k_assemble_analytical(const Tables tab, int N, const float4* __restrict__ ori, AsmOut out) {
  using S = AnaShape<M, Q>;
  constexpr int TI = S::TI, K1 = S::K1, NC = S::NC, TP = S::TP, NT = S::NT, JB = S::JB, PB = S::PB;
  constexpr int M3 = 3 * M;
  constexpr int FF = K1 * 3;
  extern __shared__ __align__(16) float smem_dyn[];
  const int T = (N + TI - 1) / TI;
  if ((int)blockIdx.x < N) {
    analytical_near<M, Q>(tab, N, ori, out, (int)blockIdx.x, T, smem_dyn);
    return;
  }
  __shared__ float4 sTi[TI];
  __shared__ unsigned char sKind[TI * TI];   // pair jl * TI + il.  0: no such pair, 1: far, 2: near
  float* const sG = smem_dyn;
  float* const sT = smem_dyn + S::GFLOATS;   // [pair of the batch][TP]
  __shared__ float sCoef[kMaxTerms], sEig[kMaxTerms];
  const int I = ((int)blockIdx.x - N) / T, J = ((int)blockIdx.x - N) % T;
  const bool diag = (I == J);
  const int tid = threadIdx.x;
  const int i0 = I * TI, j0 = J * TI;
  if (tid < M) { sCoef[tid] = tab.gamma[tid]; sEig[tid] = tab.eigen[tid]; }
  if (tid < TI) sTi[tid] = ori[min(i0 + tid, N - 1)];
  for (int pr = tid; pr < TI * TI; pr += NT) {
    const int il = pr % TI, jl = pr / TI;
    const bool valid = i0 + il < N && j0 + jl < N && (!diag || il != jl);
    const float d2 = centre_dist2(out.pos64[min(i0 + il, N - 1)], out.pos64[min(j0 + jl, N - 1)]);
    sKind[pr] = !valid ? 0 : far_pair(d2, tab.far_d2) ? 1 : 2;
  }
  const float fz = tab.fz_half;
  // force-term accumulator of task (tl, k) = (tid / K1, tid % K1): F_i[k]
  float facc[3] = {0.f, 0.f, 0.f};
  __syncthreads();
  const int jcount = min(TI, N - j0);
  for (int jb = 0; jb < jcount; jb += JB) {
    const int jn = min(JB, jcount - jb);
    // phase 1: unit u = qi * PB + pair; zeros for the pairs that are not far
    if (tid < PB * S::FN) {
      const int p = tid % PB, qi = tid / PB;
      const int pr = jb * TI + p;
      float* const gcol = sG + tid;
      if (p < jn * TI && sKind[pr] == 1) {
        closed_form<M>(out, tab.eps, i0 + pr % TI, j0 + pr / TI, tab.far_pts[qi], gcol, S::GSF);
      } else {
#pragma unroll
        for (int c = 0; c < NC; ++c) gcol[c * S::GSF] = 0.f;
      }
    }
    __syncthreads();
    // phase 2: lanes (column, pair), pair fastest
    for (int task = tid; task < PB * NC; task += NT) {
      const int col = task / PB, p = task % PB;
      fold_points<K1, S::FN, true>(tab, sG + col * S::GSF + p, PB, sT + p * TP + col);
    }
    __syncthreads();
    // phase 3: block (i, j) -- rows of fiber i, columns of fiber j (the next
    // batch's phase 1 writes G only, and its phase 2 follows a barrier)
    for (int task = tid; task < jn * TI * M * M; task += NT) {
      const int jj = task / (TI * M * M), r0 = task % (TI * M * M);
      const int kJp = r0 / (TI * M), rem = r0 % (TI * M);
      const int tl = rem / M, kIp = rem % M, jl = jb + jj;
      float* dst = out.A + (int64_t)(i0 * M3 + 3 * rem) + (int64_t)((j0 + jl) * M3 + 3 * kJp) * out.lda;
      if (diag && tl == jl) {
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
          for (int a = 0; a < 3; ++a) dst[a + b * out.lda] = (kIp == kJp && a == b) ? 1.f : 0.f;
        continue;
      }
      if (sKind[jl * TI + tl] != 1) continue;
      dense_block(dst, out.lda, sT + (jj * TI + tl) * TP + ((kIp + 1) * K1 + kJp + 1) * 6, sTi[tl], kIp, sCoef[kIp],
                  sEig[kIp]);
    }
    // force terms F_i[k] += T^{ij}[k][P0] F/2 (F/2 = (0, 0, fz): column z of the
    // block; zeros for the pairs that are not far)
    if (tid < TI * K1) {
      const int tl = tid / K1, k = tid % K1;
      for (int jj = 0; jj < jn; ++jj) {
        const float* t = sT + (jj * TI + tl) * TP + k * NC;
        facc[0] = fmaf(t[4], fz, facc[0]);
        facc[1] = fmaf(t[5], fz, facc[1]);
        facc[2] = fmaf(t[2], fz, facc[2]);
      }
    }
  }
  // partial force terms: ffpart[J][fiber of I][k][3] written exactly once
  if (tid < TI * K1) {
    const int tl = tid / K1, k = tid % K1;
    if (i0 + tl < N) {
      float* dst = out.ffpart + ((int64_t)J * N + i0 + tl) * FF + 3 * k;
#pragma unroll
      for (int a = 0; a < 3; ++a) dst[a] = facc[a];
    }
  }
}

// F[i] = sum_X ffpart[X][i] (rows X = g (mod 8) in order for each of 8 groups, then
// the groups in order) and b[i][k'] = -C_i(k') F[i][k'+1], for the kForceFibers
// fibers from i0.  Thread (group, component): 8 loads in flight per thread.
// Bound: the partial rows (N=4000: 144 MB, 227 us with one thread per (i, k)).
constexpr int kForceFibers = 4, kForceGroups = 8;
static inline int force_threads(int M) { return kForceFibers * 3 * (M + 1) * kForceGroups; }

__device__ __forceinline__ void force_terms_block(const Tables& tab, int N, const float4* __restrict__ ori,
                                                  const float* __restrict__ ffpart, int nparts, float* __restrict__ F,
                                                  float* __restrict__ b, int i0) {
  __shared__ float red[kForceGroups][kForceFibers * 3 * (kMaxTerms + 1)];
  __shared__ float sum[kForceFibers * 3 * (kMaxTerms + 1)];
  const int M = tab.M, FFn = 3 * (M + 1), C = kForceFibers * FFn;
  const int c = (int)threadIdx.x % C, g = (int)threadIdx.x / C;
  const bool in = i0 + c / FFn < N;
  const int64_t row = (int64_t)N * FFn;
  float s = 0.f;
  if (in) {
    const float* src = ffpart + (int64_t)i0 * FFn + c;
    int p = g;
    for (; p + 7 * kForceGroups < nparts; p += 8 * kForceGroups) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = src[(p + u * kForceGroups) * row];
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; p < nparts; p += kForceGroups) s += src[p * row];
  }
  red[g][c] = s;
  __syncthreads();
  if (g == 0) {
    float v = red[0][c];
#pragma unroll
    for (int q = 1; q < kForceGroups; ++q) v += red[q][c];
    sum[c] = v;
    if (in) F[(int64_t)i0 * FFn + c] = v;
  }
  __syncthreads();
  const int u = (int)threadIdx.x, il = u / M, kp = u % M;
  if (u >= kForceFibers * M || i0 + il >= N) return;
  const float* f = sum + il * FFn + 3 * (kp + 1);
  const float4 t = ori[i0 + il];
  const float t3[3] = {t.x, t.y, t.z};
  const float QF = fmaf(f[2], t3[2], fmaf(f[1], t3[1], __fmul_rn(f[0], t3[0])));
  const float coef = tab.gamma[kp], E = tab.eigen[kp];
  float* dst = b + (int64_t)(i0 + il) * 3 * M + 3 * kp;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float tq = __fmul_rn(t3[a], QF);
    dst[a] = __fmul_rn(-coef, kp == 0 ? tq : fmaf(-E, tq, f[a]));
  }
}

__global__ void k_force_terms(const Tables tab, int N, const float4* __restrict__ ori,
                              const float* __restrict__ ffpart, int nparts, float* __restrict__ F,
                              float* __restrict__ b) {
  force_terms_block(tab, N, ori, ffpart, nparts, F, b, (int)blockIdx.x * kForceFibers);
}

// ---- packed step: every member of a group (one Tables) in one launch ------
// Block b belongs to the member whose tile pairs it falls in; the member's
// blocks run exactly the single-suspension kernel's tile code, so a member's
// system is bit for bit the one k_assemble_pairs forms.
template <int MODE>
__global__ void __launch_bounds__(128, 6)
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

// blockIdx.x: member, blockIdx.y: kForceFibers of its fibers (the grid covers
// the largest member the packed solve takes)
__global__ void k_pack_force_terms(const Tables tab, const PackStepMember* __restrict__ mem) {
  const PackStepMember& p = mem[blockIdx.x];
  const int i0 = (int)blockIdx.y * kForceFibers;
  if (i0 >= p.N) return;
  const int nparts = (p.N + AsmShape<5, 24>::TI - 1) / AsmShape<5, 24>::TI;
  force_terms_block(tab, p.N, p.ori32, p.ffpart, nparts, p.F, p.b, i0);
}

int launch_pack_assemble(const Tables& tab, const PackStepMember* members, int n, int64_t blocks, bool bf16,
                         cudaStream_t st) {
  if (tab.M != 5 || tab.Q != 24 || n < 1 || blocks < 1) return RF_E_UNSUPPORTED;
  using S = NumShape<5, 24, num_threads(5, kAsmStructF16)>;
  constexpr size_t smem = S::kSmem;
  if (bf16) {
    static const cudaError_t attr = cudaFuncSetAttribute(k_pack_assemble<kAsmStructBF16>,
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    RF_CUDA_TRY(attr);
    k_pack_assemble<kAsmStructBF16><<<(unsigned)blocks, S::NT, smem, st>>>(tab, members, n);
  } else {
    static const cudaError_t attr = cudaFuncSetAttribute(k_pack_assemble<kAsmStructF16>,
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    RF_CUDA_TRY(attr);
    k_pack_assemble<kAsmStructF16><<<(unsigned)blocks, S::NT, smem, st>>>(tab, members, n);
  }
  RF_LAUNCH_CHECK();
  k_pack_force_terms<<<dim3((unsigned)n, kPackMaxFibers / kForceFibers), force_threads(5), 0, st>>>(tab, members);
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
  using S = NumShape<M, Q, num_threads(M, MODE)>;
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
  using S = AnaShape<M, Q>;
  const int64_t T = ceil_div(N, S::TI);
  static const cudaError_t attr = cudaFuncSetAttribute(k_assemble_analytical<M, Q>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem);
  RF_CUDA_TRY(attr);
  k_assemble_analytical<M, Q><<<(unsigned)(N + T * T), S::NT, S::kSmem, st>>>(tab, N, ori, out);
  RF_LAUNCH_CHECK();
  return RF_OK;
}

static int launch_force_terms(const Tables& tab, int N, const float4* ori, const AsmOut& out, int nparts, float* F,
                              float* b, cudaStream_t st) {
  k_force_terms<<<(unsigned)ceil_div(N, kForceFibers), force_threads(tab.M), 0, st>>>(
      tab, N, ori, out.ffpart, nparts, F, b);
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
  return launch_force_terms(tab, N, ori, out, assemble_tiles(tab.M, tab.Q, N), F, b, st);
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
  // one partial row per tile column, and the near pairs'
  return launch_force_terms(tab, N, ori, out, assemble_tiles(tab.M, tab.Q, N) + 1, F, b, st);
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
