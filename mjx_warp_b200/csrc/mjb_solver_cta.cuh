// The chosen form's constraint solver for large models (nv > 32, dense or sparse mass matrix): one
// CTA of NW warps per world (solver.py:26-1000, the same algorithm as solve_generic).
//
// A world with hundreds of dofs and constraint rows is too much for one warp: the Newton
// Hessian's factorisation (nv^3 / 3 multiply-adds) and the row loops (dense nv-wide Jacobian
// rows) serialise on 32 lanes, and with 16 such warps per SM the per-world matrices (nv^2 floats
// each) no longer fit in L2.  Here all NW warps of a CTA work on one world: per-row dot products
// are warp-per-row (coalesced reads of the dense Jacobian rows), per-row scalars thread-per-row,
// per-dof vectors thread-per-dof, and every per-world sum is a CTA reduction in a fixed order
// (warp sums, then the warps' partials in warp order), identical in every thread, so control flow
// stays uniform across the CTA.  The Hessian H = tril(qM) + sum_active D J'J is assembled in efc_h
// (each warp updates the H rows it owns, row by row in constraint order, so no two warps touch the
// same entry; or, selected by the autotuner and always in the precision form, as split-TF32
// tensor-core tiles, assemble_hessian_tc) and factored by chol_cta: a left-looking blocked
// Cholesky with 32-column panels whose panel updates A[r, p] -= L[r, :p] L[p, :p]^T run on the
// tensor pipe in split TF32 (mjb_tc.cuh), the 32 x 32 diagonal blocks by chol_tile and the panel
// rows below by substitution.  The precision form factors and solves in FP64 in shared memory.
// Models of 2 to 64 kinematic trees take the same steps over nonzero trees and tiles only
// (SparseShape); the dense routines remain for one tree, for more trees, dofs, rows or fill than the
// structure holds, and for the tensor-core assembly.
#pragma once

#include <type_traits>

#include "mjb_solver.cuh"

#pragma nv_diag_suppress 20168  // an unroll value of 0 (CtaSolver::kU) leaves a loop without a pragma

namespace mjb {

// CTA sums of K values: warp sums, then the NW warps' partials added in warp order; every thread
// returns the totals.  red: K * NW elements of shared memory.
template <int NW, int K, typename T>
__device__ __forceinline__ void cta_sum(T (&v)[K], T* red, int warp, int lane) {
  constexpr bool kEach = K < 4 || sizeof(T) == 8;  // (16 doubles would not stay in registers)
#pragma unroll
  for (int k = 0; kEach && k < K; k++) v[k] = warp_sum_t(v[k]);
  if constexpr (kEach) {
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < K; k++) red[k * NW + warp] = v[k];
    }
  } else {
    // butterfly sums of up to 16 values with halving exchanges: lanes whose bit is set keep the
    // upper half of the values, so 16 shuffles serve all of them (each sum's tree is unchanged)
    static_assert(K <= 16, "values per exchange");
    T x[16];
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = k < K ? v[k] : T(0);
#pragma unroll
    for (int h = 8; h > 0; h >>= 1) {
      const bool up = (lane & (2 * h)) != 0;
#pragma unroll
      for (int k = 0; k < h; k++) {
        const T mine = up ? x[h + k] : x[k], other = up ? x[k] : x[h + k];
        x[k] = mine + __shfl_xor_sync(WARP_FULL, other, 2 * h);
      }
    }
    x[0] += __shfl_xor_sync(WARP_FULL, x[0], 1);
    if ((lane & 1) == 0 && (lane >> 1) < K) red[(lane >> 1) * NW + warp] = x[0];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; k++) {
    T s = red[k * NW];
#pragma unroll
    for (int q = 1; q < NW; q++) s += red[k * NW + q];
    v[k] = s;
  }
  __syncthreads();
}

// the dof tree block [a, a + size) that contains dof i (binary search over block_adr)
__device__ __forceinline__ void dof_block(const MjbModel& m, int i, int& a, int& size) {
  int lo = 0, hi = m.nblock - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (m.block_adr[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  a = m.block_adr[lo];
  size = m.block_size[lo];
}

// Left-looking blocked Cholesky of the n x n SPD lower triangle of A (row stride ld, global
// memory) by a CTA of NW warps: per 32-column panel p, (i) the panel's rows are updated with the
// finished columns, A[r, p] -= L[r, :p] L[p, :p]^T for every row r >= p, as m16n8k8 tensor-core
// tiles in split TF32 (16-row m-tiles dealt to the warps, the panel's 32 columns as 4 n-tiles),
// (ii) warp 0 factors the 32 x 32 diagonal block in the shared tile T (chol_tile) and writes it
// back with its reciprocal diagonal in T's column 32, (iii) every row below solves
// L[r, p] = A[r, p] L_pp^-T, one thread per row.  T: 32 x 36 + 32 floats of shared memory.
template <int NW>
__device__ __noinline__ void chol_cta(float* A, int ld, int n, float* T, int warp, int lane) {
  constexpr int TL = 36, kMt = 3;
  const int g = lane >> 2, t = lane & 3;
  for (int c0 = 0; c0 < n; c0 += 32) {
    const int pn = min(32, n - c0);
    if (c0 > 0) {
      const int nmt = (n - c0 + 15) >> 4;
      for (int mt0 = warp; mt0 < nmt; mt0 += NW * kMt) {
        float acc[kMt][4][4];
#pragma unroll
        for (int q = 0; q < kMt; q++)
#pragma unroll
          for (int nt = 0; nt < 4; nt++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[q][nt][e] = 0.f;
        // raw loads of chunk k0 + 8 are issued before chunk k0's splits and products
        float rb[4][2], ra[kMt][4];
        auto load = [&](int k0, float (&xb)[4][2], float (&xa)[kMt][4]) {
#pragma unroll
          for (int nt = 0; nt < 4; nt++) {  // B[k][j] = L[c0 + j][k0 + k], j = 8 nt + g
            const int r = c0 + 8 * nt + g;
            const float* Ar = A + size_t(r) * ld + k0;
            xb[nt][0] = r < n ? Ar[t] : 0.f;
            xb[nt][1] = r < n ? Ar[t + 4] : 0.f;
          }
#pragma unroll
          for (int q = 0; q < kMt; q++) {
            const int mt = mt0 + q * NW;
            const int r0 = c0 + 16 * mt + g, r1 = r0 + 8;
            const bool ok0 = mt < nmt && r0 < n, ok1 = mt < nmt && r1 < n;
            const float* A0 = A + size_t(r0) * ld + k0;
            const float* A1 = A + size_t(r1) * ld + k0;
            xa[q][0] = ok0 ? A0[t] : 0.f;
            xa[q][1] = ok1 ? A1[t] : 0.f;
            xa[q][2] = ok0 ? A0[t + 4] : 0.f;
            xa[q][3] = ok1 ? A1[t + 4] : 0.f;
          }
        };
        load(0, rb, ra);
        for (int k0 = 0; k0 < c0; k0 += 8) {
          float nb[4][2], na[kMt][4];
          if (k0 + 8 < c0) load(k0 + 8, nb, na);
          FragB b[4];
#pragma unroll
          for (int nt = 0; nt < 4; nt++) b[nt] = frag_b(rb[nt][0], rb[nt][1]);
#pragma unroll
          for (int q = 0; q < kMt; q++) {
            const int mt = mt0 + q * NW;
            if (mt < nmt) {
              const FragA a = frag_a(ra[q][0], ra[q][1], ra[q][2], ra[q][3]);
#pragma unroll
              for (int nt = 0; nt < 4; nt++) mma_3xtf32(acc[q][nt], a, b[nt]);
            }
          }
          if (k0 + 8 < c0) {
#pragma unroll
            for (int nt = 0; nt < 4; nt++) {
              rb[nt][0] = nb[nt][0];
              rb[nt][1] = nb[nt][1];
            }
#pragma unroll
            for (int q = 0; q < kMt; q++)
#pragma unroll
              for (int e = 0; e < 4; e++) ra[q][e] = na[q][e];
          }
        }
#pragma unroll
        for (int q = 0; q < kMt; q++) {
          const int mt = mt0 + q * NW;
          if (mt >= nmt) break;
          const int r0 = c0 + 16 * mt + g, r1 = r0 + 8;
#pragma unroll
          for (int nt = 0; nt < 4; nt++) {
            const int cc = c0 + 8 * nt + 2 * t;
#pragma unroll
            for (int e = 0; e < 2; e++) {
              if (cc + e < c0 + pn) {  // lower triangle only (the diagonal block's upper part
                                       // is not part of the factor)
                if (r0 < n && cc + e <= r0) A[size_t(r0) * ld + cc + e] -= acc[q][nt][e];
                if (r1 < n && cc + e <= r1) A[size_t(r1) * ld + cc + e] -= acc[q][nt][2 + e];
              }
            }
          }
        }
      }
    }
    __syncthreads();
    if (warp == 0) {  // (ii)
      for (int r = 0; r < pn; r++)
        if (lane < pn) T[r * TL + lane] = lane <= r ? A[size_t(c0 + r) * ld + c0 + lane] : 0.f;
      __syncwarp();
      chol_tile(T, TL, pn, lane);
      for (int r = 0; r < pn; r++)
        if (lane <= r) A[size_t(c0 + r) * ld + c0 + lane] = T[r * TL + lane];
      if (lane < pn) T[lane * TL + 32] = __frcp_rn(T[lane * TL + lane]);
    }
    __syncthreads();
    const bool vec = (ld & 3) == 0 && pn == 32 && aligned16(A);  // rows 16-byte aligned: float4 reads and writes
    for (int i = c0 + pn + int(threadIdx.x); i < n; i += NW * 32) {  // (iii)
      float* Ai = A + size_t(i) * ld + c0;
      float x[32];
      if (vec) {
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const float4 v = reinterpret_cast<const float4*>(Ai)[q];
          x[4 * q] = v.x;
          x[4 * q + 1] = v.y;
          x[4 * q + 2] = v.z;
          x[4 * q + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 32; c++) x[c] = c < pn ? Ai[c] : 0.f;
      }
#pragma unroll
      for (int c = 0; c < 32; c++) {
        if (c < pn) {
          float v = x[c];
#pragma unroll
          for (int q = 0; q < c; q++) v -= x[q] * T[c * TL + q];
          x[c] = v * T[c * TL + 32];
        }
      }
      if (vec) {
#pragma unroll
        for (int q = 0; q < 8; q++)
          reinterpret_cast<float4*>(Ai)[q] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
      } else {
#pragma unroll
        for (int c = 0; c < 32; c++)
          if (c < pn) Ai[c] = x[c];
      }
    }
    __syncthreads();
  }
}

// x = (L L^T)^-1 y by a CTA of NW warps for the n x n lower factor L in global memory (row stride
// ld), blocked by 32: forward, each block's partial y_b - L[b, :b] z[:b] is a row-per-warp dot
// product over the finished part (coalesced row reads, warp sums), then warp 0 solves the 32 x 32
// diagonal block with its rows in registers; backward, each block's partial
// z_b - L[b+:, b]^T x[b+:] is accumulated warp-per-row over the rows below (lane j reads the
// row's entry in column j of the block, coalesced), reduced across the warps in red, then warp 0
// solves L_bb^T.  z: n floats of shared memory (the intermediate vector); red: 32 NW floats.
// x and y are in global memory (x may alias y).
template <int NW>
__device__ __noinline__ void cho_solve_cta(const float* L, int ld, int n, float* x, const float* y,
                                           float* z, float* red, int warp, int lane) {
  for (int c0 = 0; c0 < n; c0 += 32) {  // L z = y
    const int pn = min(32, n - c0);
    for (int j = warp; j < pn; j += NW) {
      const float* Lr = L + size_t(c0 + j) * ld;
      float a = 0.f;
      for (int k = lane; k < c0; k += 32) a += Lr[k] * z[k];
      a = warp_sum(a);
      if (lane == 0) z[c0 + j] = y[c0 + j] - a;
    }
    __syncthreads();
    if (warp == 0) {
      float r[32];  // row `lane` of the diagonal block
      const float* Lr = L + size_t(c0 + min(lane, pn - 1)) * ld + c0;
#pragma unroll
      for (int q = 0; q < 32; q++) r[q] = (q < pn && q <= lane && lane < pn) ? Lr[q] : 1.f;
      float zi = lane < pn ? z[c0 + lane] : 0.f;
#pragma unroll
      for (int q = 0; q < 32; q++) {
        if (q < pn) {
          const float zq = __shfl_sync(WARP_FULL, zi, q) / __shfl_sync(WARP_FULL, r[q], q);
          if (lane == q) zi = zq;
          else if (lane > q && lane < pn) zi -= r[q] * zq;
        }
      }
      if (lane < pn) z[c0 + lane] = zi;
    }
    __syncthreads();
  }
  const int nb = (n + 31) / 32;
  for (int b = nb - 1; b >= 0; b--) {  // L^T x = z
    const int c0 = 32 * b, pn = min(32, n - c0);
    float acc = 0.f;  // lane j: sum over this warp's rows i below the block of L[i][c0 + j] x[i]
    for (int i = c0 + pn + warp; i < n; i += NW)
      if (lane < pn) acc += L[size_t(i) * ld + c0 + lane] * z[i];
    red[warp * 32 + lane] = acc;
    __syncthreads();
    if (warp == 0) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < NW; q++) t += red[q * 32 + lane];
      float xi = lane < pn ? z[c0 + lane] - t : 0.f;
      // back substitution with L_bb^T: column lane of L_bb is row lane of L_bb^T
      for (int q = pn - 1; q >= 0; q--) {
        const float lq = lane < q ? L[size_t(c0 + q) * ld + c0 + lane] : 0.f;
        const float xq = __shfl_sync(WARP_FULL, xi, q) / L[size_t(c0 + q) * ld + c0 + q];
        if (lane == q) xi = xq;
        else if (lane < q) xi -= lq * xq;
      }
      if (lane < pn) z[c0 + lane] = xi;
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += NW * 32) x[i] = z[i];
  __syncthreads();
}

// ------------------------------------------------------------------------------------------
// The world's sparsity.  A constraint row touches the dofs of at most two kinematic trees (the two
// bodies of a contact, one joint), and the mass matrix couples dofs within a tree only, so for a
// model of many trees most of H and of its factor is exactly zero (the 384-dof bin, 40 contacts
// per world: 5 % of L and 0.2 % of the dense factor's multiply-adds are nonzero).  One pass over
// the dense rows finds each row's trees; the trees' elimination fill follows in dof order as 64-bit
// masks; everything below then visits nonzero trees and tiles only.  A skipped term is a product
// with an exact zero, so every sum keeps its order and its bits.
//
// What bounds it: latency.  A world's solve is a chain of short dependent stages (12 panels or some
// ten levels per factorisation or substitution) on four warps, and the structure's 50 KB of shared
// memory lets four worlds run per SM.  Loops over the structure are kept rolled: unrolled, the code
// of one Newton iteration outgrew the instruction cache (no_instruction stalls 2.4 cycles per issue
// against 0.3, solver 21.1 against 13.0 ms).  Measured on the bin, Newton 10 iterations, whole step:
// 4096 worlds 83.2 -> 16.5 ms, 300 worlds with the sparse mass matrix 12.4 -> 4.7 ms.
constexpr int kSpTrees = 64;  // trees (bits of a mask)
// Capacities of the structure in shared memory, for models of up to kDofs dofs: kRows rows with
// their trees, kBlocks nonzero tree pairs of L, kSlots groups of up to 8 rows of a tree below a
// panel, kItems 8 x 8 tiles of L updated by earlier panels, kJ floats of staged nonzero row entries,
// kL floats of L.  Large: 4 worlds of the 384-dof bin per SM (57 KB each); Small: 9 worlds of up to
// 128 dofs (24 KB).
struct SparseLarge {
  static constexpr int kDofs = 512, kRows = 736, kBlocks = 512, kSlots = 512, kItems = 704, kJ = 2048, kL = 4096;
};
struct SparseSmall {
  static constexpr int kDofs = 128, kRows = 192, kBlocks = 160, kSlots = 160, kItems = 192, kJ = 4, kL = 2560;
};

// One direction's schedule of the triangular solves: the nodes by dependency level, eight lanes
// per node (32 for a node of more than 8 dofs), packed into warps.
template <int NODES>
struct SparseOrder {
  uint8_t slot[4 * NODES];   // node of each group of eight lanes, 255: none
  uint8_t start[NODES + 1];  // first warp of each level
  int levels;
};

template <class C>
struct SparseShape {
  static constexpr int kDofs = C::kDofs, kRows = C::kRows, kBlocks = C::kBlocks, kSlots = C::kSlots,
                       kItems = C::kItems, kJ = C::kJ, kL = C::kL, kPanels = C::kDofs / 32,
                       kNodes = kSpTrees + kPanels;  // nodes: a tree's dofs within one panel
  unsigned long long tmask[kSpTrees];      // trees u <= t with L(t, u) != 0, t itself among them
  unsigned long long tup[kSpTrees];        // trees t > u with L(t, u) != 0
  unsigned long long ptrees[kPanels];    // trees with dofs in each 32-column panel
  float cj[kJ];                          // staged row entries (tree u's, then tree t's)
  float cl[kL];                          // L, each tree's rows over its nonzero columns
  float sD[kRows];                       // D of the active rows, 0 elsewhere
  float sF[kRows];                       // the rows' forces
  float* L;                                // cl, or efc_h when L does not fit there
  int rbase[kSpTrees];                     // a tree's first row in L and its row stride
  uint32_t rlist[2 * kRows];             // each tree's rows, ascending: row | other tree << 16
  uint32_t group[kDofs];                 // dofs of the panel coupled (transitively) with a dof
  uint16_t rld[kSpTrees];
  uint16_t tadr[kSpTrees + 1];             // first dof of each tree
  uint16_t radr[kSpTrees + 1];             // first entry of each tree's rows in rlist
  uint16_t rtree[kRows];                 // a row's trees: u | t << 8, u <= t (u == t: one tree)
  uint16_t bst[kSpTrees + 1];              // a tree's first pair in blk / bcol
  uint16_t blk[kBlocks];                 // nonzero tree pairs t << 8 | u, u <= t
  uint16_t bcol[kBlocks];                // the pair's first column in its tree's rows of L
  uint16_t pslot[kSlots];                // each panel's rows below that are != 0 in it: tree | 8-row group << 8
  uint16_t padr[kPanels + 1];            // first entry of each panel in pslot
  uint16_t iadr[kPanels + 1];            // first entry of each panel in item
  uint32_t item[kItems];                 // a panel's updated 8 x 8 tiles: tree u | column group << 6 |
                                           // tree t << 11 | row group << 17, by u and column group
  uint16_t nadr[kNodes + 1];             // first dof of each node
  uint8_t ntree[kNodes];                 // its tree
  uint8_t dtree[kDofs];                  // tree of each dof
  SparseOrder<kNodes> fwd, bwd;
  int nblk;
  unsigned cnt[kSpTrees];

  // column of tree u's first dof in tree t's rows of L
  __device__ __forceinline__ int col(int t, int u) const {
    return bcol[bst[t] + __popcll(tmask[t] & ((1ull << u) - 1ull))];
  }
  __device__ __forceinline__ float* row(int i, int t) const { return L + rbase[t] + (i - tadr[t]) * rld[t]; }
};
template <int NW>
using SparseFor = SparseShape<std::conditional_t<NW == 1, SparseSmall, SparseLarge>>;
template <class SH>
constexpr int kSpFloats = int((sizeof(SH) + 15) / 16 * 4);

// the launches that look for a structure in each world, by the model and the Hessian's assembly; the
// others keep the dense forms' small part of shared memory
template <int NW>
__host__ __device__ __forceinline__ bool sparse_launch(const MjbModel& m, bool tc) {
  return !tc && m.nblock >= 2 && m.nblock <= kSpTrees && m.nv <= SparseFor<NW>::kDofs;
}

__device__ __forceinline__ unsigned long long bits_below(int b) {  // bits 0 .. b - 1
  return b >= 64 ? ~0ull : (1ull << b) - 1ull;
}
// the dofs of panel c0 .. c0 + pn - 1 that lie in tree u, as a mask
template <class SH>
__device__ __forceinline__ unsigned panel_bits(const SH& S, int u, int c0, int pn) {
  const int q0 = max(int(S.tadr[u]) - c0, 0), q1 = min(int(S.tadr[u + 1]) - c0, pn);
  return unsigned(bits_below(q1) & ~bits_below(q0));
}

// Finds the structure of a world's n rows (J: n x nv dense) by a CTA of NW warps; false (in every
// thread) when it does not fit the masks or lists, and the dense routines then run.  Whether it fits
// is decided by the reduction of a barrier: every warp returns from the same one.  cw: floats per
// row of cj (twice the largest tree), or 0 when the rows do not fit there.  H: the world's efc_h.
template <int NW, class SH>
__device__ __noinline__ bool sparse_shape(const MjbModel& m, const float* J, int n, float* H,
                                          SH& S, int& cw, int warp, int lane) {
  const int nv = m.nv, nt = m.nblock, tid = warp * 32 + lane;
  constexpr int NT = NW * 32;
  if (n > SH::kRows) return false;
  cw = 2 * m.block_max;
  if (n * cw > SH::kJ) cw = 0;
  bool bad = false;  // what this thread found does not fit
#pragma unroll 1
  for (int t = tid; t < nt; t += NT) {
    const int a = m.block_adr[t], z = m.block_size[t];
    S.tadr[t] = uint16_t(a);
    S.tmask[t] = 1ull << t;
    S.cnt[t] = 0u;
#pragma unroll 1
    for (int i = a; i < a + z; i++) S.dtree[i] = uint8_t(t);
  }
  if (tid == 0) S.tadr[nt] = uint16_t(nv);
  __syncthreads();
  // rows: a warp per four rows, four columns per lane of each loaded at once; the trees of the
  // nonzero entries
  const bool v4 = (nv & 3) == 0 && aligned16(J);
#pragma unroll 1
  for (int k0 = 4 * warp; k0 < n; k0 += 4 * NW) {
    unsigned lo[4] = {0u, 0u, 0u, 0u}, hi[4] = {0u, 0u, 0u, 0u};
#pragma unroll 1
    for (int base = 0; base < nv; base += 384) {
      float4 v[4][3];
#pragma unroll
      for (int h = 0; h < 4; h++)
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const int c = base + 128 * q + 4 * lane;
          const float* Jr = J + size_t(k0 + h) * nv + c;
          v[h][q] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (k0 + h < n) {
            if (v4) {
              if (c < nv) v[h][q] = *reinterpret_cast<const float4*>(Jr);
            } else {
              if (c < nv) v[h][q].x = Jr[0];
              if (c + 1 < nv) v[h][q].y = Jr[1];
              if (c + 2 < nv) v[h][q].z = Jr[2];
              if (c + 3 < nv) v[h][q].w = Jr[3];
            }
          }
        }
#pragma unroll
      for (int h = 0; h < 4; h++)
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const float e[4] = {v[h][q].x, v[h][q].y, v[h][q].z, v[h][q].w};
          if (e[0] != 0.f || e[1] != 0.f || e[2] != 0.f || e[3] != 0.f)
#pragma unroll
            for (int j = 0; j < 4; j++)
              if (e[j] != 0.f) {
                const int t = S.dtree[base + 128 * q + 4 * lane + j];
                if (t < 32) lo[h] |= 1u << t;
                else hi[h] |= 1u << (t - 32);
              }
        }
    }
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const int k = k0 + h;
      if (k >= n) break;
      const unsigned long long mk = (static_cast<unsigned long long>(__reduce_or_sync(WARP_FULL, hi[h])) << 32) |
                                    __reduce_or_sync(WARP_FULL, lo[h]);
      const int c = __popcll(mk);
      const int u = mk ? __ffsll(mk) - 1 : 0, t = mk ? 63 - __clzll(mk) : 0;
      if (lane == 0) {
        if (c > 2) bad = true;
        S.rtree[k] = uint16_t(u | (t << 8));
        atomicAdd(&S.cnt[t], 1u);
        if (u != t) {
          atomicAdd(&S.cnt[u], 1u);
          atomicOr(&S.tmask[t], 1ull << u);
        }
      }
      if (cw) {
        const float* Jr = J + size_t(k) * nv;
        const int au = S.tadr[u], nu = S.tadr[u + 1] - au, at = S.tadr[t], nn = S.tadr[t + 1] - at;
#pragma unroll 1
        for (int j = lane; j < nu + (u == t ? 0 : nn); j += 32)
          S.cj[k * cw + j] = Jr[j < nu ? au + j : at + j - nu];
      }
    }
  }
  if (__syncthreads_or(bad)) return false;
  if (warp == 0) {  // elimination fill, tree by tree; lane l holds trees l and l + 32
    unsigned long long m0 = lane < nt ? S.tmask[lane] : 0ull;
    unsigned long long m1 = lane + 32 < nt ? S.tmask[lane + 32] : 0ull;
#pragma unroll 1
    for (int k = 0; k < nt; k++) {
      const bool h0 = lane > k && ((m0 >> k) & 1ull), h1 = lane + 32 > k && ((m1 >> k) & 1ull);
      const unsigned long long R = __ballot_sync(WARP_FULL, h0) |
                                   (static_cast<unsigned long long>(__ballot_sync(WARP_FULL, h1)) << 32);
      if (h0) m0 |= R & bits_below(lane + 1);
      if (h1) m1 |= R & bits_below(lane + 33);
      if (lane == 0) S.tup[k] = R;
    }
    if (lane < nt) S.tmask[lane] = m0;
    if (lane + 32 < nt) S.tmask[lane + 32] = m1;
    // the pairs of L, its rows' columns and sizes, and the trees' row lists
    int tot0, tot1;
    const int e0 = warp_excl_scan(__popcll(m0), lane, &tot0);
    const int e1 = warp_excl_scan(__popcll(m1), lane, &tot1) + tot0;
    const bool fits = tot0 + tot1 <= SH::kBlocks;
    bad = !fits;
    // one warp: with over three quarters of the pairs nonzero the dense form is the faster one (forward of 2048
    // worlds of 14 capsules across one, all 120 pairs nonzero: 7.0 ms here, 3.9 in solve_generic)
    if (NW == 1) bad |= 8 * (tot0 + tot1) > 3 * nt * (nt + 1);
    if (lane == 0) S.nblk = tot0 + tot1;
    int w0 = 0, w1 = 0;  // columns of this lane's trees
    if (fits) {
      S.bst[lane] = uint16_t(e0);
      S.bst[lane + 32] = uint16_t(e1);
      int e = e0;
#pragma unroll 1
      for (unsigned long long q = m0; q; q &= q - 1ull) {
        const int u = __ffsll(q) - 1;
        S.blk[e] = uint16_t((lane << 8) | u);
        S.bcol[e++] = uint16_t(w0);
        w0 += S.tadr[u + 1] - S.tadr[u];
      }
      e = e1;
#pragma unroll 1
      for (unsigned long long q = m1; q; q &= q - 1ull) {
        const int u = __ffsll(q) - 1;
        S.blk[e] = uint16_t(((lane + 32) << 8) | u);
        S.bcol[e++] = uint16_t(w1);
        w1 += S.tadr[u + 1] - S.tadr[u];
      }
    }
    const int z0 = lane < nt ? S.tadr[lane + 1] - S.tadr[lane] : 0;
    const int z1 = lane + 32 < nt ? S.tadr[lane + 33] - S.tadr[lane + 32] : 0;
    int f0, f1;
    const int b0 = warp_excl_scan(w0 * z0, lane, &f0), b1 = warp_excl_scan(w1 * z1, lane, &f1) + f0;
    const bool compact = f0 + f1 <= SH::kL;
    if (lane == 0) S.L = compact ? S.cl : H;
    S.rbase[lane] = compact ? b0 : int(S.tadr[min(lane, nt)]) * nv;
    S.rld[lane] = uint16_t(compact ? w0 : nv);
    S.rbase[lane + 32] = compact ? b1 : int(S.tadr[min(lane + 32, nt)]) * nv;
    S.rld[lane + 32] = uint16_t(compact ? w1 : nv);
    if (fits && !compact) {
      __syncwarp();
#pragma unroll 1
      for (int e = lane; e < tot0 + tot1; e += 32) S.bcol[e] = S.tadr[S.blk[e] & 255];
    }
    const int r0 = lane < nt ? int(S.cnt[lane]) : 0, r1 = lane + 32 < nt ? int(S.cnt[lane + 32]) : 0;
    const int a0 = warp_excl_scan(r0, lane, &tot0), a1 = warp_excl_scan(r1, lane, &tot1) + tot0;
    S.radr[lane] = uint16_t(a0);
    S.radr[lane + 32] = uint16_t(a1);
    if (lane == 0) S.radr[kSpTrees] = uint16_t(tot0 + tot1);
  }
  if (__syncthreads_or(bad)) return false;
#pragma unroll 1
  for (int t = warp; t < nt; t += NW) {  // rows of each tree, ascending
    int e = S.radr[t];
#pragma unroll 1
    for (int k0 = 0; k0 < n && e < S.radr[t + 1]; k0 += 32) {
      const int k = k0 + lane, p = k < n ? S.rtree[k] : 0xffff, u = p & 255, v = p >> 8;
      const bool hit = u == t || v == t;
      const unsigned mk = __ballot_sync(WARP_FULL, hit);
      if (hit) S.rlist[e + __popc(mk & ((1u << lane) - 1u))] = unsigned(k) | (unsigned(u == t ? v : u) << 16);
      e += __popc(mk);
    }
  }
  const int n32 = (nv + 31) >> 5;
#pragma unroll 1
  for (int p = warp; p < n32; p += NW) {
    const int c0 = 32 * p, c1 = min(c0 + 32, nv), pn = c1 - c0;
    const int t0 = S.dtree[c0], t1 = S.dtree[c1 - 1];
    const unsigned long long in = bits_below(t1 + 1) & ~bits_below(t0);
    if (lane == 0) S.ptrees[p] = in;
    unsigned g = 0u;  // the panel's dofs coupled with this lane's, closed transitively
    if (lane < pn)
      for (unsigned long long q = S.tmask[S.dtree[c0 + lane]] & in; q; q &= q - 1ull)
        g |= panel_bits(S, __ffsll(q) - 1, c0, pn);
#pragma unroll 1
    for (;;) {
      const unsigned old = g;
#pragma unroll 1
      for (int q = 0; q < pn; q++) {
        const unsigned gq = __shfl_sync(WARP_FULL, g, q);
        if (gq & g) g |= gq;
      }
      if (!__any_sync(WARP_FULL, g != old)) break;
    }
    if (lane < pn) S.group[c0 + lane] = g;
  }
  __syncthreads();
  // nodes: in dof order, each tree's dofs within one panel
  if (warp == 0) {
    int tot0, tot1;
    const int s0 = lane < nt ? ((S.tadr[lane + 1] - 1) >> 5) - (S.tadr[lane] >> 5) + 1 : 0;
    const int s1 = lane + 32 < nt ? ((S.tadr[lane + 33] - 1) >> 5) - (S.tadr[lane + 32] >> 5) + 1 : 0;
    const int e0 = warp_excl_scan(s0, lane, &tot0), e1 = warp_excl_scan(s1, lane, &tot1) + tot0;
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      const int t = lane + 32 * h, e = h ? e1 : e0, z = h ? s1 : s0;
#pragma unroll 1
      for (int j = 0; j < z; j++) {
        S.nadr[e + j] = uint16_t(j ? ((S.tadr[t] >> 5) + j) << 5 : S.tadr[t]);
        S.ntree[e + j] = uint8_t(t);
      }
    }
    if (lane == 0) S.nadr[tot0 + tot1] = uint16_t(nv);
    // the rows below each panel, eight of a tree at a time
    int at = 0;
#pragma unroll 1
    for (int p = 0; p < n32; p++) {
      const int c1 = min(32 * p + 32, nv);
      if (lane == 0) S.padr[p] = uint16_t(min(at, SH::kSlots));
#pragma unroll 1
      for (int h = 0; h < 64; h += 32) {
        const int t = h + lane;
        const bool below = t < nt && S.tadr[t + 1] > c1 && (S.tmask[t] & S.ptrees[p]);
        const int z = below ? (S.tadr[t + 1] - max(int(S.tadr[t]), c1) + 7) >> 3 : 0;
        int tot;
        const int e = at + warp_excl_scan(z, lane, &tot);
#pragma unroll 1
        for (int j = 0; j < z; j++)
          if (e + j < SH::kSlots) S.pslot[e + j] = uint16_t(t | (j << 8));
        at += tot;
      }
    }
    if (lane == 0) S.padr[n32] = uint16_t(min(at, SH::kSlots));
    bad = at > SH::kSlots;
  }
  if (warp == NW - 1) {  // the tiles that earlier panels update: the pairs with a common earlier tree
    int at = 0;
#pragma unroll 1
    for (int p = 0; p < n32; p++) {
      const int c0 = 32 * p, c1 = min(c0 + 32, nv);
      if (lane == 0) S.iadr[p] = uint16_t(min(at, SH::kItems));
      if (p == 0) continue;
      const int tb = S.dtree[c0];
      const unsigned long long early = bits_below(tb + (S.tadr[tb] < c0 ? 1 : 0));
#pragma unroll 1
      for (unsigned long long b = S.ptrees[p]; b; b &= b - 1ull) {
        const int u = __ffsll(b) - 1, j0 = max(int(S.tadr[u]), c0), j1 = min(int(S.tadr[u + 1]), c1);
        const unsigned long long eu = S.tmask[u] & early;
        if (!eu) continue;
#pragma unroll 1
        for (int cg = 0; j0 + 8 * cg < j1; cg++)
#pragma unroll 1
          for (int h = 0; h < 64; h += 32) {
            const int t = h + lane;
            const bool hit = t >= u && t < nt && (S.tmask[t] & eu) && ((S.tmask[t] >> u) & 1ull);
            const int z = hit ? (S.tadr[t + 1] - max(int(S.tadr[t]), c0) + 7) >> 3 : 0;
            int tot;
            const int e = at + warp_excl_scan(z, lane, &tot);
#pragma unroll 1
            for (int j = 0; j < z; j++)
              if (e + j < SH::kItems) S.item[e + j] = unsigned(u) | (unsigned(cg) << 6) | (unsigned(t) << 11) | (unsigned(j) << 17);
            at += tot;
          }
      }
    }
    if (lane == 0) S.iadr[n32] = uint16_t(min(at, SH::kItems));
    bad |= at > SH::kItems;
  }
  if (__syncthreads_or(bad)) return false;
  // Levels: a node waits for every node of the trees its rows (forward) or columns (backward) couple
  // with, and for its own tree's previous node.  Warp 0 takes the forward order, warp 1 the other.
#pragma unroll 1
  for (int dir = warp; dir < 2; dir += NW) {
    const bool bw = dir == 1;
    auto& O = bw ? S.bwd : S.fwd;
    int last[2], first[2], len[2];  // levels of the trees' last and first nodes to be solved
    unsigned long long dep[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int t = lane + 32 * h;
      first[h] = 0;
      len[h] = t < nt ? ((S.tadr[t + 1] - 1) >> 5) - (S.tadr[t] >> 5) : 0;
      last[h] = len[h];
      dep[h] = t < nt ? (bw ? S.tup[t] : S.tmask[t] & ~(1ull << t)) : 0ull;
    }
#pragma unroll 1
    for (;;) {
      bool ch = false;
      int nf[2] = {0, 0};
      unsigned long long d0 = dep[0], d1 = dep[1];
#pragma unroll 1
      while (__any_sync(WARP_FULL, (d0 | d1) != 0ull)) {
        const int q0 = d0 ? __ffsll(d0) - 1 : 0, q1 = d1 ? __ffsll(d1) - 1 : 0;
        const int a0 = __shfl_sync(WARP_FULL, last[0], q0 & 31), b0 = __shfl_sync(WARP_FULL, last[1], q0 & 31);
        const int a1 = __shfl_sync(WARP_FULL, last[0], q1 & 31), b1 = __shfl_sync(WARP_FULL, last[1], q1 & 31);
        if (d0) nf[0] = max(nf[0], (q0 < 32 ? a0 : b0) + 1);
        if (d1) nf[1] = max(nf[1], (q1 < 32 ? a1 : b1) + 1);
        d0 &= d0 - 1ull;
        d1 &= d1 - 1ull;
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        ch |= nf[h] != first[h];
        first[h] = nf[h];
        last[h] = nf[h] + len[h];
      }
      if (!__any_sync(WARP_FULL, ch)) break;
    }
    const int top = __reduce_max_sync(WARP_FULL, max(lane < nt ? last[0] : 0, lane + 32 < nt ? last[1] : 0)) + 1;
    // node v of this lane (three passes of 32): its level
    int nn = 0;
#pragma unroll 1
    while (S.nadr[nn] < nv) nn++;
    int lv[3];
    bool big[3];
#pragma unroll
    for (int h = 0; h < 3; h++) {
      const int v = lane + 32 * h;
      const int t = v < nn ? S.ntree[v] : 0;
      const int f0 = __shfl_sync(WARP_FULL, first[0], t & 31), f1 = __shfl_sync(WARP_FULL, first[1], t & 31);
      const int seg = v < nn ? (S.nadr[v] >> 5) - (S.tadr[t] >> 5) : 0;
      const int z = v < nn ? ((S.tadr[t + 1] - 1) >> 5) - (S.tadr[t] >> 5) : 0;
      lv[h] = v < nn ? (t < 32 ? f0 : f1) + (bw ? z - seg : seg) : -1;
      big[h] = v < nn && S.nadr[v + 1] - S.nadr[v] > 8;
    }
    int at = 0;  // warps so far
#pragma unroll 1
    for (int l = 0; l < top; l++) {
      if (lane == 0) O.start[l] = uint8_t(at);
      int nb = 0, ns = 0;
#pragma unroll
      for (int h = 0; h < 3; h++) {
        nb += __popc(__ballot_sync(WARP_FULL, lv[h] == l && big[h]));
        ns += __popc(__ballot_sync(WARP_FULL, lv[h] == l && !big[h]));
      }
#pragma unroll 1
      for (int e = 4 * (at + nb) + ns + lane; e < 4 * (at + nb + ((ns + 3) >> 2)); e += 32) O.slot[e] = 255;
      int ib = 0, is = 0;
#pragma unroll
      for (int h = 0; h < 3; h++) {
        const unsigned mb = __ballot_sync(WARP_FULL, lv[h] == l && big[h]);
        const unsigned ms = __ballot_sync(WARP_FULL, lv[h] == l && !big[h]);
        const unsigned lt = (1u << lane) - 1u;
        if (lv[h] == l && big[h])
          for (int j = 0; j < 4; j++) O.slot[4 * (at + ib + __popc(mb & lt)) + j] = uint8_t(lane + 32 * h);
        if (lv[h] == l && !big[h]) O.slot[4 * (at + nb) + is + __popc(ms & lt)] = uint8_t(lane + 32 * h);
        ib += __popc(mb);
        is += __popc(ms);
      }
      at += nb + ((ns + 3) >> 2);
    }
    if (lane == 0) {
      O.start[top] = uint8_t(at);
      O.levels = top;
    }
  }
  __syncthreads();
  return true;
}

// chol_cta over the nonzero tiles of S, on S.L: the same panels, products and sums.
// (i) panel updates: a warp per two 8-row groups of trees t and one 8-column group of a panel's tree
// u, over the 8-column chunks that hold a tree both couple with (rows and columns of an mma tile are
// independent, so they are gathered; the chunks are those of the dense form); (ii) the diagonal
// block gathered into T, factored by warp 0 group by group; (iii) the rows below solve against it,
// a lane per row and up to eight columns of one tree in registers.
template <int NW, class SH>
__device__ __noinline__ void chol_cta_sparse(int n, float* T, const SH& S, int warp, int lane) {
  constexpr int TL = 36;
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll 1
  for (int c0 = 0; c0 < n; c0 += 32) {
    const int pn = min(32, n - c0), p = c0 >> 5;
    const int m0 = S.iadr[p], m1 = S.iadr[p + 1];
    if (NW == 1 && m1 > m0) {
      // chol_blocked's trailing updates, panel by panel: four partial sums by column mod 4.  Lane:
      // row g and columns t4, t4 + 4 of the tile.
      for (int e = m0; e < m1; e++) {
        const unsigned ia = S.item[e];
        const int u = ia & 63, ta = (ia >> 11) & 63;
        const int cb = max(int(S.tadr[u]), c0) + 8 * ((ia >> 6) & 31) + t4, ce = min(int(S.tadr[u + 1]), c0 + pn);
        const int r = max(int(S.tadr[ta]), c0) + 8 * (ia >> 17) + g;
        const bool kr = r < S.tadr[ta + 1], k0 = kr && cb < ce && cb <= r, k1 = kr && cb + 4 < ce && cb + 4 <= r;
        const float* Lr = S.row(kr ? r : S.tadr[ta], ta);
        const float* L0 = S.row(k0 ? cb : S.tadr[u], u);
        const float* L1 = S.row(k1 ? cb + 4 : S.tadr[u], u);
        float* C = const_cast<float*>(Lr) + S.col(ta, u) + cb - S.tadr[u];
        float a0 = k0 ? C[0] : 0.f, a1 = k1 ? C[4] : 0.f;
        float s[4] = {0.f, 0.f, 0.f, 0.f}, z[4] = {0.f, 0.f, 0.f, 0.f};
        int pv = -1;  // the earlier panel of the sums
        for (unsigned long long b = S.tmask[u] & S.tmask[ta]; b; b &= b - 1ull) {
          const int v = __ffsll(b) - 1, av = S.tadr[v], ev = min(int(S.tadr[v + 1]), c0);
          if (av >= c0) break;
          const int ct = S.col(ta, v) - av, cu = S.col(u, v) - av;
          for (int k = av & ~3; k < ev; k += 4) {
            if ((k >> 5) != pv) {
              a0 -= (s[0] + s[1]) + (s[2] + s[3]);
              a1 -= (z[0] + z[1]) + (z[2] + z[3]);
#pragma unroll
              for (int q = 0; q < 4; q++) s[q] = z[q] = 0.f;
              pv = k >> 5;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
              if (k + q >= av && k + q < ev) {
                const float x = Lr[ct + k + q];
                s[q] += x * L0[cu + k + q];
                z[q] += x * L1[cu + k + q];
              }
            }
          }
        }
        a0 -= (s[0] + s[1]) + (s[2] + s[3]);
        a1 -= (z[0] + z[1]) + (z[2] + z[3]);
        if (k0) C[0] = a0;
        if (k1) C[4] = a1;
      }
      __syncwarp();
    }
    if (NW > 1 && m1 > m0) {
      const unsigned long long low = bits_below(c0 >> 3);
#pragma unroll 1
      for (int e = m0 + 2 * warp; e < m1; e += 2 * NW) {
        // the second row group joins the first when it has the same columns, else runs by itself
        const unsigned it0 = S.item[e], it1 = S.item[min(e + 1, m1 - 1)];
        const bool pair = e + 1 < m1 && ((it0 ^ it1) & 2047u) == 0u;
#pragma unroll 1
        for (int half = 0; half < (pair || e + 1 >= m1 ? 1 : 2); half++) {
          const unsigned ia = half ? it1 : it0;
          const int u = ia & 63, ta = (ia >> 11) & 63, tb = (it1 >> 11) & 63;
          const int cb = max(int(S.tadr[u]), c0) + 8 * ((ia >> 6) & 31), ce = min(int(S.tadr[u + 1]), c0 + pn);
          const int ra = max(int(S.tadr[ta]), c0) + 8 * (ia >> 17) + g;
          const int rb = max(int(S.tadr[tb]), c0) + 8 * (it1 >> 17) + g;
          const bool ka = ra < S.tadr[ta + 1], kb = pair && rb < S.tadr[tb + 1], kc = cb + g < ce;
          const unsigned long long mu = S.tmask[u], ma = S.tmask[ta], mb = S.tmask[tb];
          const float* Ra = S.row(ka ? ra : S.tadr[ta], ta);
          const float* Rb = S.row(kb ? rb : S.tadr[tb], tb);
          const float* Rc = S.row(kc ? cb + g : S.tadr[u], u);
          const int ba = S.bst[ta], bb = S.bst[tb], bu = S.bst[u];
          unsigned long long km = 0ull;  // chunks of the common trees left of the panel
#pragma unroll 1
          for (unsigned long long b = mu & (pair ? ma | mb : ma); b; b &= b - 1ull) {
            const int v = __ffsll(b) - 1;
            km |= bits_below(((S.tadr[v + 1] - 1) >> 3) + 1) & ~bits_below(S.tadr[v] >> 3);
          }
          float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
          for (km &= low; km; km &= km - 1ull) {
            const int k0 = 8 * (__ffsll(km) - 1) + t4;
            float xa[2], xb[2], xc[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int k = k0 + 4 * h, v = S.dtree[k], o = k - S.tadr[v];
              const unsigned long long bit = 1ull << v, lw = bit - 1ull;
              xa[h] = ka && (ma & bit) ? Ra[S.bcol[ba + __popcll(ma & lw)] + o] : 0.f;
              xb[h] = kb && (mb & bit) ? Rb[S.bcol[bb + __popcll(mb & lw)] + o] : 0.f;
              xc[h] = kc && (mu & bit) ? Rc[S.bcol[bu + __popcll(mu & lw)] + o] : 0.f;
            }
            mma_3xtf32(acc, frag_a(xa[0], xb[0], xa[1], xb[1]), frag_b(xc[0], xc[1]));
          }
          float* Ca = const_cast<float*>(Ra) + S.bcol[ba + __popcll(ma & ((1ull << u) - 1ull))] - S.tadr[u];
          float* Cb = const_cast<float*>(Rb) + S.bcol[bb + __popcll(mb & ((1ull << u) - 1ull))] - S.tadr[u];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int c = cb + 2 * t4 + h;
            if (c < ce) {
              if (ka && c <= ra) Ca[c] -= acc[h];
              if (kb && c <= rb) Cb[c] -= acc[2 + h];
            }
          }
        }
      }
      __syncthreads();
    }
    const unsigned long long in = S.ptrees[p];
    const int cu = lane < pn ? S.dtree[c0 + lane] : 0, ca = c0 + lane - S.tadr[cu];  // this lane's column
    {  // the diagonal block, a warp per tree
      int turn = 0;
#pragma unroll 1
      for (unsigned long long b = in; b; b &= b - 1ull, turn++) {
        if ((turn & (NW - 1)) != warp) continue;
        const int tr = __ffsll(b) - 1, a = S.tadr[tr], ld = S.rld[tr];
        const int i0 = max(a, c0), i1 = min(int(S.tadr[tr + 1]), c0 + pn);
        const bool has = lane < pn && ((S.tmask[tr] >> cu) & 1ull);
        const float* L = S.L + S.rbase[tr] + (i0 - a) * ld + (has ? S.col(tr, cu) + ca : 0);
#pragma unroll 4
        for (int i = i0; i < i1; i++, L += ld) T[(i - c0) * TL + lane] = has && c0 + lane <= i ? *L : 0.f;
      }
    }
    __syncthreads();
    if (warp == 0) {
      chol_tile_groups(T, TL, pn, lane < pn ? S.group[c0 + lane] : 0u, lane);
      if (lane < pn) T[lane * TL + 32] = __frcp_rn(T[lane * TL + lane]);
    }
    __syncthreads();
    {  // the factored block back to L
      int turn = 0;
#pragma unroll 1
      for (unsigned long long b = in; b; b &= b - 1ull, turn++) {
        if ((turn & (NW - 1)) != warp) continue;
        const int tr = __ffsll(b) - 1, a = S.tadr[tr], ld = S.rld[tr];
        const int i0 = max(a, c0), i1 = min(int(S.tadr[tr + 1]), c0 + pn);
        const bool has = lane < pn && ((S.tmask[tr] >> cu) & 1ull);
        float* L = S.L + S.rbase[tr] + (i0 - a) * ld + (has ? S.col(tr, cu) + ca : 0);
#pragma unroll 4
        for (int i = i0; i < i1; i++, L += ld)
          if (has && c0 + lane <= i) *L = T[(i - c0) * TL + lane];
      }
    }
    const int s1 = S.padr[p + 1];
#pragma unroll 1
    for (int s0 = S.padr[p] + 4 * (NW - 1 - warp); s0 < s1; s0 += 4 * NW) {
      const int sl = s0 + (lane >> 3), ps = S.pslot[min(sl, s1 - 1)], tr = ps & 255;
      const int i = max(int(S.tadr[tr]), c0 + pn) + 8 * (ps >> 8) + (lane & 7);
      const bool own = sl < s1 && i < S.tadr[tr + 1];
      float* R = S.row(own ? i : S.tadr[tr], tr);
      const unsigned long long cp = S.tmask[tr] & in;  // the panel's trees, ascending
      unsigned long long b = own ? cp : 0ull;
      int j0 = 0, j1 = 0;  // the columns left of the current tree
      float* Ru = R;
#pragma unroll 1
      while (__any_sync(WARP_FULL, b != 0ull || j0 < j1)) {
        if (j0 >= j1 && b) {
          const int u = __ffsll(b) - 1;
          b &= b - 1ull;
          j0 = max(int(S.tadr[u]), c0);
          j1 = min(int(S.tadr[u + 1]), c0 + pn);
          Ru = R + S.col(tr, u) - S.tadr[u];
        }
        const int w = min(8, j1 - j0);  // <= 0: this lane is done
        const float* Tj = T + (j0 - c0) * TL - c0;
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = j < w ? Ru[j0 + j] : 0.f;
        if (w > 0)  // the panel's earlier columns
          for (unsigned long long q = cp; q; q &= q - 1ull) {
            const int u = __ffsll(q) - 1, k1 = min(int(S.tadr[u + 1]), j0);
            int k = max(int(S.tadr[u]), c0);
            if (k >= k1) break;
#pragma unroll 1
            for (const float* Rk = R + S.col(tr, u) - S.tadr[u]; k < k1; k++) {
              const float xk = Rk[k];
#pragma unroll
              for (int j = 0; j < 8; j++)
                if (j < w) x[j] -= xk * Tj[j * TL + k];
            }
          }
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (j < w) {
            x[j] *= T[(j0 - c0 + j) * TL + 32];
#pragma unroll
            for (int e = j + 1; e < 8; e++)
              if (e < w) x[e] -= x[j] * Tj[e * TL + j0 + j];
          }
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (j < w) Ru[j0 + j] = x[j];
        j0 += 8;
      }
    }
    __syncthreads();
  }
}

// cho_solve_cta on S.L, node by node in the order of S.fwd and S.bwd: a level's nodes do not depend
// on one another.  Lane = row (forward) or column (backward) of a node; each sum keeps the blocked
// solve's order: the part outside the 32-dof block first (forward: lane-strided partials added by
// a 32-lane butterfly, formed by eight lanes per row; backward: one partial per warp of that form),
// then the block's terms one by one.
template <int NW, class SH>
__device__ __noinline__ void cho_solve_cta_sparse(int n, float* x, const float* y, float* z,
                                                  const SH& S, int warp, int lane) {
  const int l8 = lane & 7;
#pragma unroll 1
  for (int lev = 0; lev < S.fwd.levels; lev++) {  // L z = y
#pragma unroll 1
    for (int q = S.fwd.start[lev] + warp; q < S.fwd.start[lev + 1]; q += NW) {
      const int v = S.fwd.slot[4 * q + (lane >> 3)];
      const bool any = v != 255;
      const int t = any ? S.ntree[v] : 0, i0 = any ? S.nadr[v] : 0, i1 = any ? S.nadr[v + 1] : 0;
      const bool big = i1 - i0 > 8;
      const int c0 = i0 & ~31, j0 = i0 + (big ? lane & 24 : 0), r = j0 + l8;
      const bool own = r < i1;
      const unsigned long long tm = any ? S.tmask[t] : 0ull;
      // trees with dofs before the block
      const int tb = S.dtree[c0];
      const unsigned long long before = NW == 1 ? 0ull : tm & bits_below(tb + (S.tadr[tb] < c0 ? 1 : 0));
      float a = 0.f;
      const float* Lr = S.row(own ? r : i0, t);
      if (own && before) {
        // column k's partial belongs to lane k mod 32: for each k mod 8 (taken in bit-reversed
        // order) its four lanes as (0 + 16) + (8 + 24), then the eight sums pairwise, as the
        // butterfly adds them
        float c1 = 0.f, c2 = 0.f, c4 = 0.f;
#pragma unroll 1
        for (int h = 0; h < 8; h++) {
          const int l = ((h & 1) << 2) | (h & 2) | (h >> 2);
          float p[4] = {0.f, 0.f, 0.f, 0.f};
          int e = S.bst[t];
#pragma unroll 1
          for (unsigned long long b = before; b; b &= b - 1ull, e++) {
            const int u = __ffsll(b) - 1, au = S.tadr[u], end = min(int(S.tadr[u + 1]), c0);
            const float* Lu = Lr + S.bcol[e] - au;
#pragma unroll 1
            for (int k = au + ((l - au) & 7); k < end; k += 8) {
              const float lk = Lu[k], zk = z[k];
              const int sl = (k >> 3) & 3;
#pragma unroll
              for (int q4 = 0; q4 < 4; q4++) p[q4] = sl == q4 ? fmaf(lk, zk, p[q4]) : p[q4];
            }
          }
          float f = (p[0] + p[2]) + (p[1] + p[3]);
          if (h & 1) {
            f = c1 + f;
            if (h & 2) {
              f = c2 + f;
              if (h & 4) a = c4 + f;
              else c4 = f;
            } else {
              c2 = f;
            }
          } else {
            c1 = f;
          }
        }
      }
      float zi = own ? y[r] - a : 0.f;
      if (own)
        for (unsigned long long b = NW == 1 ? tm : tm & S.ptrees[c0 >> 5] & ~(1ull << t); b; b &= b - 1ull) {
          const int u = __ffsll(b) - 1, au = S.tadr[u], end = min(int(S.tadr[u + 1]), i0);
          const float* Lu = Lr + S.col(t, u) - au;
#pragma unroll 1
          for (int k = NW == 1 ? au : max(au, c0); k < end; k++) zi -= Lu[k] * z[k];
        }
      const float* Lt = Lr + (any ? S.col(t, t) - S.tadr[t] : 0);
      const float diag = own ? Lt[r] : 1.f;
      const int steps = __reduce_max_sync(WARP_FULL, i1 - i0);
#pragma unroll 1
      for (int j = 0; j < steps; j++) {
        const int k = i0 + j;
        if (own && k == r) {
          zi /= diag;
          z[r] = zi;
        }
        __syncwarp();
        if (own && k < r) zi -= Lt[k] * z[k];
      }
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int lev = 0; lev < S.bwd.levels; lev++) {  // L^T x = z
#pragma unroll 1
    for (int q = S.bwd.start[lev] + warp; q < S.bwd.start[lev + 1]; q += NW) {
      const int v = S.bwd.slot[4 * q + (lane >> 3)];
      const bool any = v != 255;
      const int t = any ? S.ntree[v] : 0, i0 = any ? S.nadr[v] : 0, i1 = any ? S.nadr[v + 1] : 0;
      const bool big = i1 - i0 > 8;
      const int c1 = (i0 & ~31) + 32, r = i0 + (big ? lane & 24 : 0) + l8;
      const bool own = r < i1;
      const int ra = r - S.tadr[t];
      const unsigned long long up = own ? S.tup[t] : 0ull, in = S.ptrees[i0 >> 5];
      float s = 0.f;
      // rows outside the block: the node's own tree's (if it goes on) and the later trees'
      const unsigned long long out = NW == 1 ? 0ull : up | (own && S.tadr[t + 1] > c1 ? 1ull << t : 0ull);
      if (out) {
        float acc[NW];  // the partials of the blocked form's warps
#pragma unroll
        for (int h = 0; h < NW; h++) acc[h] = 0.f;
#pragma unroll 1
        for (unsigned long long b = out; b; b &= b - 1ull) {
          const int u = __ffsll(b) - 1, au = S.tadr[u], ld = S.rld[u], e = S.tadr[u + 1];
          int i = max(au, c1);
          const float* Lu = S.L + S.rbase[u] + S.col(u, t) + ra + (i - au) * ld;
#pragma unroll 1
          for (; i < e; i++, Lu += ld) {
            const float lk = *Lu, zk = z[i];
#pragma unroll
            for (int h = 0; h < NW; h++) acc[h] = (i & (NW - 1)) == h ? fmaf(lk, zk, acc[h]) : acc[h];
          }
        }
#pragma unroll
        for (int h = 0; h < NW; h++) s += acc[h];
      }
      float xi = own ? z[r] - s : 0.f;
      // the block's later trees (one warp: every later dof), from the last dof
      unsigned long long b = NW == 1 ? up | (own ? 1ull << t : 0ull) : up & in;
#pragma unroll 1
      while (b) {
        const int u = 63 - __clzll(b), au = S.tadr[u], ld = S.rld[u];
        b &= ~(1ull << u);
        const float* Lu = S.L + S.rbase[u] + S.col(u, t) + ra;
#pragma unroll 1
        for (int i = (NW == 1 ? int(S.tadr[u + 1]) : min(int(S.tadr[u + 1]), c1)) - 1; i >= max(au, i1); i--)
          xi -= Lu[(i - au) * ld] * z[i];
      }
      const int lt = any ? S.rld[t] : 0;
      const float* Lt = S.L + S.rbase[t] + (own ? S.col(t, t) + ra : 0) - int(S.tadr[t]) * lt;
      const float diag = own ? Lt[r * lt] : 1.f;
      const int steps = __reduce_max_sync(WARP_FULL, i1 - i0);
#pragma unroll 1
      for (int j = 1; j <= steps; j++) {
        const int k = i1 - j;
        if (own && k == r) {
          xi /= diag;
          z[r] = xi;
        }
        __syncwarp();
        if (own && k > r) xi -= Lt[k * lt] * z[k];
      }
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += NW * 32) x[i] = z[i];
  __syncthreads();
}

// Per-CTA shared memory of the solver (floats): reductions (16 NW, as doubles 32 NW), the
// diagonal tile (32 x 36 + 32), each warp's row-compaction scratch and the triangular solves'
// vector (nv); the precision form adds the FP64 Hessian factor, its lower triangle packed row by
// row (row i at i (i + 1) / 2), then the FP64 solve's vector and the factor's reciprocal
// diagonal (nv doubles each), 16-byte aligned after the floats.
__host__ __device__ __forceinline__ int tri(int i) { return i * (i + 1) / 2; }
// Each warp's row-compaction scratch (dense rows) or, with sparse (sparse_launch), the larger of it and
// the structure.  Dense launches without the structure's 50 KB: 2048 worlds of a 100-dof chain, two and
// four warps per world, forward 17.2 -> 15.3 and 11.8 -> 8.2 ms; of 66 free spheres (nv = 396) 39.7 -> 35.6.
__host__ __device__ __forceinline__ int cta_solver_union_floats(int nv, int nw, bool sparse) {
  const int sp = nw == 1 ? kSpFloats<SparseFor<1>> : kSpFloats<SparseFor<2>>;
  const int dense = nw == 1 ? generic_nz_floats(nv) : nw * 2 * round4i(nv);
  return sparse && sp > dense ? sp : dense;
}
__host__ __device__ __forceinline__ int cta_solver_smem_base(int nv, int nw, bool sparse) {
  return round4i(32 * nw + 32 * 36 + 32 + round4i(nv)) + cta_solver_union_floats(nv, nw, sparse);
}
__host__ __device__ __forceinline__ int cta_solver_smem_floats(int nv, int nw, bool prec, bool sparse) {
  const int base = cta_solver_smem_base(nv, nw, sparse);
  return prec ? base + 2 * (tri(nv) + 2 * nv + 1) : base;
}

// FP64 counterpart of chol_cta for the precision form, on the packed lower triangle P of an
// n x n SPD matrix in shared memory: per 32-column panel, (i) every entry (r, j) of the panel's
// rows r >= p subtracts its dot product over the finished columns (4 x 1 strips of entries per
// thread, so each loaded L[j][k] serves four rows); (ii) warp 0 factors the diagonal block in
// place, lane per row, with the pivot's reciprocal kept in rd; (iii) the rows below solve
// against it, one thread per row, multiplying by rd.
template <int NW>
__device__ __noinline__ void chol_cta_d(double* P, double* rd, int n, int warp, int lane) {
  constexpr int NT = NW * 32;
  for (int c0 = 0; c0 < n; c0 += 32) {
    const int pn = min(32, n - c0);
    if (c0 > 0) {
      const int nr4 = (n - c0 + 3) / 4;  // strips of four rows
      for (int e = int(threadIdx.x); e < nr4 * pn; e += NT) {
        const int r = c0 + 4 * (e / pn), j = c0 + e % pn;
        const double* Lj = P + tri(j);
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        const double* R0 = P + tri(r);
        const double* R1 = P + tri(min(r + 1, n - 1));
        const double* R2 = P + tri(min(r + 2, n - 1));
        const double* R3 = P + tri(min(r + 3, n - 1));
        for (int k = 0; k < c0; k++) {
          const double l = Lj[k];
          s0 += R0[k] * l;
          s1 += R1[k] * l;
          s2 += R2[k] * l;
          s3 += R3[k] * l;
        }
        if (j <= r) P[tri(r) + j] -= s0;
        if (r + 1 < n && j <= r + 1) P[tri(r + 1) + j] -= s1;
        if (r + 2 < n && j <= r + 2) P[tri(r + 2) + j] -= s2;
        if (r + 3 < n && j <= r + 3) P[tri(r + 3) + j] -= s3;
      }
      __syncthreads();
    }
    if (warp == 0) {  // (ii): column k of the block, lanes over its rows (left-looking)
      for (int k = 0; k < pn; k++) {
        const int i = c0 + k + lane;
        const double* Lk = P + tri(c0 + k) + c0;
        double s = 0.0;
        if (k + lane < pn) {
          const double* Li = P + tri(i) + c0;
          s = Li[k];
          for (int q = 0; q < k; q++) s -= Li[q] * Lk[q];
        }
        const double sk = __shfl_sync(WARP_FULL, s, 0);
        const double inv = rsqrt(sk);  // the pivot's reciprocal; L_kk = s_k rsqrt(s_k)
        const double lkk = sk * inv;
        __syncwarp();
        if (lane == 0) {
          P[tri(c0 + k) + c0 + k] = lkk;
          rd[c0 + k] = inv;
        } else if (k + lane < pn) {
          P[tri(i) + c0 + k] = s * inv;
        }
        __syncwarp();
      }
    }
    __syncthreads();
    for (int i = c0 + pn + int(threadIdx.x); i < n; i += NT) {  // (iii)
      double* Ai = P + tri(i) + c0;
      for (int c = 0; c < pn; c++) {
        double v = Ai[c];
        const double* Lc = P + tri(c0 + c) + c0;
        for (int q = 0; q < c; q++) v -= Ai[q] * Lc[q];
        Ai[c] = v * rd[c0 + c];
      }
    }
    __syncthreads();
  }
}

// x = (L L^T)^-1 y for the packed FP64 factor in shared memory, one warp, in FP64 with the
// intermediate vector in v (n doubles of shared memory) and the reciprocal diagonal rd; x and y
// are n floats in global memory (x may alias y).
static __device__ void cho_solve_d_warp(const double* P, const double* rd, int n, double* v, float* x,
                                 const float* y, int lane) {
  for (int i = lane; i < n; i += 32) v[i] = double(y[i]);
  __syncwarp();
  for (int k = 0; k < n; k++) {  // L z = y, a column at a time; lanes update the rows below
    const double zk = v[k] * rd[k];
    __syncwarp();
    if (lane == (k & 31)) v[k] = zk;
    for (int i = k + 1 + lane; i < n; i += 32) v[i] -= P[tri(i) + k] * zk;
    __syncwarp();
  }
  for (int k = n - 1; k >= 0; k--) {  // L^T x = z: row k of L is column k of L^T
    const double xk = v[k] * rd[k];
    __syncwarp();
    if (lane == (k & 31)) v[k] = xk;
    const double* Lk = P + tri(k);
    for (int i = lane; i < k; i += 32) v[i] -= Lk[i] * xk;
    __syncwarp();
  }
  for (int i = lane; i < n; i += 32) x[i] = float(v[i]);
  __syncwarp();
}

// cho_solve_d_warp for n <= 128: the vector in four registers per lane (entry i on lane i mod 32), each
// entry broadcast by a shuffle, instead of a column step through shared memory between two warp
// barriers: the same operations on every entry in the same order.
static __device__ __noinline__ void cho_solve_d_regs(const double* P, const double* rd, int n, float* x,
                                                     const float* y, int lane) {
  double v[4];
  const double* R[4];  // the lane's rows
#pragma unroll
  for (int t = 0; t < 4; t++) {
    const int i = lane + 32 * t;
    v[t] = i < n ? double(y[i]) : 0.0;
    R[t] = P + tri(min(i, n - 1));
  }
#pragma unroll
  for (int b = 0; b < 4; b++) {  // L z = y
#pragma unroll 1
    for (int k = 32 * b; k < min(n, 32 * b + 32); k++) {
      const double zk = __shfl_sync(WARP_FULL, v[b], k & 31) * rd[k];
      if (lane + 32 * b == k) v[b] = zk;
      else if (lane + 32 * b > k && lane + 32 * b < n) v[b] -= R[b][k] * zk;
#pragma unroll
      for (int t = b + 1; t < 4; t++)
        if (lane + 32 * t < n) v[t] -= R[t][k] * zk;
    }
  }
#pragma unroll
  for (int b = 3; b >= 0; b--) {  // L^T x = z
#pragma unroll 1
    for (int k = min(n, 32 * b + 32) - 1; k >= 32 * b; k--) {
      const double xk = __shfl_sync(WARP_FULL, v[b], k & 31) * rd[k];
      const double* Lk = P + tri(k) + lane;
      if (lane + 32 * b == k) v[b] = xk;
      else if (lane + 32 * b < k) v[b] -= Lk[32 * b] * xk;
#pragma unroll
      for (int t = 0; t < b; t++) v[t] -= Lk[32 * t] * xk;
    }
  }
#pragma unroll
  for (int t = 0; t < 4; t++)
    if (lane + 32 * t < n) x[lane + 32 * t] = float(v[t]);
  __syncwarp();
}

// A gradient with a NaN or an infinity in it (grad_dot alone may overflow): the dense substitution
// multiplies it with the zeros between the trees, so that every entry becomes NaN.  So it does here: no
// tree of a world that has gone wrong looks solved.
static __device__ __noinline__ void spread_nonfinite(const float* grad, float* Mgrad, int nv, int tid, int nt) {
  bool bad = false;
  for (int i = tid; i < nv; i += nt) bad |= !isfinite(grad[i]);
  if (!__syncthreads_or(bad)) return;
  for (int i = tid; i < nv; i += nt) Mgrad[i] = __int_as_float(0x7fffffff);
}

// the CG preconditioner, kept out of the Newton solver's code
static __device__ __noinline__ void cta_solve_m(const MjbModel& m, const MjbData& d, int w, float* x,
                                                const float* y, int lane) {
  solve_m_world(m, d, w, x, y, lane);
}

// TREES: worlds over nonzero trees and tiles (sparse_launch), the dense routines for those that do not
// fit; else the dense routines only, in kernels of their own, their loops left to the compiler: kept
// rolled, as the structure's kernels need them, they have fewer loads in flight (forward of 1024 worlds
// of a 140-dof chain 19.9 against 17.3 ms, of 2048 worlds of 66 free spheres 35.6 against 33.0).
template <int NW, bool PREC, bool TREES>
struct CtaSolver {
  const MjbModel& m;
  const MjbData& d;
  int w, tid, lane, warp, nv, adr, n;
  float *qacc, *Ma, *grad, *Mgrad, *search, *mv, *qfrc_constraint, *H;
  const float *qM, *qfrc_smooth, *qacc_smooth;
  float* red;    // 32 NW floats (cta sums of up to 9 values, as floats or doubles; the solves)
  float* T;      // chol_cta's diagonal tile
  float* nz;     // this warp's row compaction: round4(nv) ints, then round4(nv) floats
  float* zv;     // the triangular solves' intermediate vector (nv floats)
  double* Ld;    // precision form: the Hessian's FP64 factor, lower triangle packed by rows
  double* vd;    // precision form: the FP64 solve's vector (nv doubles)
  double* rdg;   // precision form: the factor's reciprocal diagonal (nv doubles)
  bool reuse = true, factored = false, changed = true;
  bool sp = false;      // the world's sparsity is in S: nonzero trees and tiles only
  bool cleared = false; // the zeros of efc_h's lower triangle are written
  int cw = 0;           // floats per staged row in S->cj, 0: entries read from efc_J
  using SH = SparseFor<NW>;
  SH* S;
  bool tc = false;  // FP32 form: the Hessian assembled on the tensor pipe (assemble_hessian_tc)
  float cost, prev_cost, gauss, grad_dot, search_dot, gtol, alpha, beta;
  float qg[3];
  static constexpr int NT = NW * 32;

  static constexpr int kU = TREES ? 1 : 0;  // loops that both forms run: rolled, or no pragma

  __device__ __forceinline__ bool sparse() const { return TREES && sp; }

  template <int K>
  __device__ __forceinline__ void sum(float (&v)[K]) { cta_sum<NW, K, float>(v, red, warp, lane); }
  // line-search coefficient sums: base + the CTA's sum of x, in FP64 in the precision form
  template <int K>
  __device__ __forceinline__ void ls_sums(const float (&base)[K], float (&x)[K]) {
    if (PREC) {
      double v[K];
#pragma unroll
      for (int k = 0; k < K; k++) v[k] = double(x[k]);
      cta_sum<NW, K, double>(v, reinterpret_cast<double*>(red), warp, lane);
#pragma unroll
      for (int k = 0; k < K; k++) x[k] = float(double(base[k]) + v[k]);
    } else {
      sum<K>(x);
#pragma unroll
      for (int k = 0; k < K; k++) x[k] = base[k] + x[k];
    }
  }

  // res = M vec (support.py:35-137): the dense mass matrix within each dof tree block, or the
  // sparse one's diagonal-plus-ancestor products, one tree per thread
  __device__ void mul_m(float* res, const float* vec) {
    if (m.is_sparse) {
#pragma unroll kU
      for (int blk = tid; blk < m.nblock; blk += NT) {
        const int a = m.block_adr[blk], size = m.block_size[blk];
#pragma unroll kU
        for (int i = a; i < a + size; i++) res[i] = qM[m.dof_Madr[i]] * vec[i];
#pragma unroll kU
        for (int i = a; i < a + size; i++) {
          int Mij = m.dof_Madr[i] + 1;
#pragma unroll 1
          for (int j = m.dof_parentid[i]; j >= 0; j = m.dof_parentid[j], Mij++) {
            res[i] += qM[Mij] * vec[j];
            res[j] += qM[Mij] * vec[i];
          }
        }
      }
      __syncthreads();
      return;
    }
#pragma unroll kU
    for (int i = tid; i < nv; i += NT) {
      int a, size;
      if (sparse()) {
        const int t = S->dtree[i];
        a = S->tadr[t];
        size = S->tadr[t + 1] - a;
      } else {
        dof_block(m, i, a, size);
      }
      const float* row = qM + size_t(i) * nv;
      float s = 0.f;
#pragma unroll kU
      for (int j = a; j < a + size; j++) s += row[j] * vec[j];
      res[i] = s;
    }
    __syncthreads();
  }

  // row k's entries in the columns of tree tr (one of its trees)
  __device__ __forceinline__ const float* row_entries(int k, int tr) const {
    if (!cw) return d.efc_J + size_t(adr + k) * nv + S->tadr[tr];
    const int u = S->rtree[k] & 255;
    return S->cj + k * cw + (tr == u ? 0 : S->tadr[u + 1] - S->tadr[u]);
  }

  // J_k . x in column order (solve_generic's sum)
  __device__ __forceinline__ float row_dot(int k, const float* x) const {
    const int pr = S->rtree[k], u = pr & 255, t = pr >> 8;
    float v = 0.f;
#pragma unroll 1
    for (int q = 0; q < (u == t ? 1 : 2); q++) {
      const int tr = q ? t : u, a = S->tadr[tr], z = S->tadr[tr + 1];
      const float* e = row_entries(k, tr);
#pragma unroll 2
      for (int c = a; c < z; c++) v += e[c - a] * x[c];
    }
    return v;
  }

  // out[r] = J_r . x - sub[r] for every row (warp per row); sub may be null
  __device__ void rows_dot(const float* x, float* out, const float* sub) {
    if (sparse() && NW == 1) {
#pragma unroll 1
      for (int k = lane; k < n; k += 32) {
        const float v = row_dot(k, x);
        out[adr + k] = sub ? v - sub[adr + k] : v;
      }
      __syncwarp();
      return;
    }
    if (sparse()) {
      // Eight lanes per row over its trees' columns.  The dense form sums lane-strided partials
      // by a 32-lane butterfly; column c's partial belongs to lane c mod 32, so lane l of the eight
      // keeps the four partials l, l + 8, l + 16, l + 24 and adds them as the butterfly does.
      const int l8 = lane & 7;
#pragma unroll 1
      for (int k0 = 4 * warp; k0 < n; k0 += 4 * NW) {
        const int k = k0 + (lane >> 3);
        float p[4] = {0.f, 0.f, 0.f, 0.f};
        if (cw && cw <= 16) {  // trees of up to 8 dofs: at most one column of each per lane
          if (k < n) {
            const int pr = S->rtree[k], u = pr & 255, t = pr >> 8;
            const int a0 = S->tadr[u], z0 = S->tadr[u + 1], a1 = S->tadr[t], z1 = u == t ? a1 : S->tadr[t + 1];
            const int e0 = (l8 - a0) & 7, e1 = (l8 - a1) & 7, c0 = a0 + e0, c1 = a1 + e1;
            const float* e = S->cj + k * cw;
            if (c0 < z0) p[0] = e[e0] * x[c0];
            if (c1 < z1) {
              const float J = e[z0 - a0 + e1], v = x[c1];
              p[0] = ((c0 ^ c1) & 24) ? __fadd_rn(p[0], __fmul_rn(J, v)) : fmaf(J, v, p[0]);
            }
          }
        } else if (k < n) {
          const int pr = S->rtree[k], u = pr & 255, t = pr >> 8;
#pragma unroll 1
          for (int q = 0; q < (u == t ? 1 : 2); q++) {
            const int tr = q ? t : u, a = S->tadr[tr], z = S->tadr[tr + 1];
            const float* e = row_entries(k, tr);
#pragma unroll 1
            for (int c = a + ((l8 - a) & 7); c < z; c += 8) {
              const float J = e[c - a], v = x[c];
              const int sl = (c >> 3) & 3;
#pragma unroll
              for (int j = 0; j < 4; j++) p[j] = sl == j ? fmaf(J, v, p[j]) : p[j];
            }
          }
        }
        float v = (p[0] + p[2]) + (p[1] + p[3]);
        v += __shfl_xor_sync(WARP_FULL, v, 4);
        v += __shfl_xor_sync(WARP_FULL, v, 2);
        v += __shfl_xor_sync(WARP_FULL, v, 1);
        if (l8 == 0 && k < n) out[adr + k] = sub ? v - sub[adr + k] : v;
      }
      __syncthreads();
      return;
    }
#pragma unroll kU
    for (int k = warp; k < n; k += NW) {
      const float* J = d.efc_J + size_t(adr + k) * nv;
      float v = 0.f;
#pragma unroll kU
      for (int i = lane; i < nv; i += 32) v += J[i] * x[i];
      v = warp_sum(v);
      if (lane == 0) out[adr + k] = sub ? v - sub[adr + k] : v;
    }
    __syncthreads();
  }

  // solver.py:75-173
  __device__ void update_constraint() {
    prev_cost = cost;
    float c[2] = {0.f, 0.f};
    bool ch = false;
#pragma unroll kU
    for (int k = tid; k < n; k += NT) {
      const int r = adr + k;
      const float Jaref = d.efc_Jaref[r], D = d.efc_D[r];
      const int active = Jaref < 0.f;
      ch |= d.efc_active[r] != active;
      d.efc_active[r] = active;
      if (sparse()) {
        S->sD[k] = active ? D : 0.f;
        S->sF[k] = active ? -1.f * D * Jaref : 0.f;
      }
      if (active) {
        d.efc_force[r] = -1.f * D * Jaref;
        c[0] += 0.5f * D * Jaref * Jaref;
      } else {
        d.efc_force[r] = 0.f;
      }
    }
    changed = __syncthreads_or(ch) != 0;
#pragma unroll kU
    for (int i = tid; i < nv; i += NT) {
      float f = 0.f;
      if (sparse()) {
        const int t = S->dtree[i], a = S->tadr[t];
#pragma unroll 1
        for (int e = S->radr[t]; e < S->radr[t + 1]; e++) {
          const int k = S->rlist[e] & 0xffff;
          const float fk = S->sF[k];
          if (fk != 0.f) f += row_entries(k, t)[i - a] * fk;
        }
      }
#pragma unroll kU
      for (int k = sparse() ? n : 0; k < n; k++) {
        const float fk = d.efc_force[adr + k];
        if (fk != 0.f) f += d.efc_J[size_t(adr + k) * nv + i] * fk;
      }
      qfrc_constraint[i] = f;
      c[1] += 0.5f * (Ma[i] - qfrc_smooth[i]) * (qacc[i] - qacc_smooth[i]);
    }
    sum<2>(c);
    gauss = c[1];
    cost = c[0] + c[1];
  }

  // H = tril(qM) + sum over active rows of D J'J in efc_h (update_gradient's Newton Hessian,
  // solver.py:249-276): warp q owns the H rows i with i % NW == q, and applies each row's outer
  // product over the row's nonzero columns to those rows in constraint order, so every entry sees
  // the reference's sequence of additions and no two warps write the same entry.
  // the lower triangle of the mass matrix into Out (row stride ldh, or packed by rows): the
  // dense qM a coalesced row per warp; the sparse one zeros, then each dof's row of its
  // ancestors (smooth.py:264-279's layout), one dof per thread
  template <typename TH, bool PACKED = false>
  __device__ void lower_mass(TH* Out, int ldh) {
    auto at = [&](int i) { return PACKED ? size_t(tri(i)) : size_t(i) * ldh; };
    if (!m.is_sparse) {
      for (int i = warp; i < nv; i += NW) {
        const float* Mi = qM + size_t(i) * nv;
        TH* Hi = Out + at(i);
        for (int j = lane; j <= i; j += 32) Hi[j] = TH(Mi[j]);
      }
      __syncthreads();
      return;
    }
    for (int i = warp; i < nv; i += NW) {
      TH* Hi = Out + at(i);
      for (int j = lane; j <= i; j += 32) Hi[j] = TH(0);
    }
    __syncthreads();
    for (int i = tid; i < nv; i += NT) {
      int a = m.dof_Madr[i];
      TH* Hi = Out + at(i);
      Hi[i] = TH(qM[a]);
      for (int j = m.dof_parentid[i]; j >= 0; j = m.dof_parentid[j]) Hi[j] = TH(qM[++a]);
    }
    __syncthreads();
  }

  // assemble_hessian over the nonzero tree pairs: a warp per pair, a lane per entry, the rows that
  // touch both trees in constraint order
  __device__ void assemble_hessian_sparse() {
    if (!cleared) {  // efc_h's lower triangle: zero outside the pairs
      for (int i = warp; i < nv; i += NW) {
        float* Hi = H + size_t(i) * nv;
        int j0 = 0;
        if ((nv & 3) == 0 && aligned16(H)) {
          j0 = (i + 1) & ~3;
#pragma unroll 1
          for (int j = 4 * lane; j < j0; j += 128) *reinterpret_cast<float4*>(Hi + j) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll 1
        for (int j = j0 + lane; j <= i; j += 32) Hi[j] = 0.f;
      }
      cleared = true;
      __syncthreads();
    }
    const bool msp = m.is_sparse;
    if (msp) {
#pragma unroll 1
      for (int i = tid; i < nv; i += NT) {
        const int t = S->dtree[i], t0 = S->tadr[t];
        float* Li = S->row(i, t) + S->col(t, t) - t0;
#pragma unroll 1
        for (int j = t0; j < i; j++) Li[j] = 0.f;
        int a = m.dof_Madr[i];
        Li[i] = qM[a];
#pragma unroll 1
        for (int j = m.dof_parentid[i]; j >= 0; j = m.dof_parentid[j]) Li[j] = qM[++a];
      }
      __syncthreads();
    }
    // lane = row i of the pair's tree t, eight columns of tree u in registers
#pragma unroll 1
    for (int b0 = 4 * warp; b0 < S->nblk; b0 += 4 * NW) {
      const int b = b0 + (lane >> 3);
      if (b >= S->nblk) continue;
      const int t = S->blk[b] >> 8, u = S->blk[b] & 255;
      const int at = S->tadr[t], au = S->tadr[u], st = S->tadr[t + 1] - at, su = S->tadr[u + 1] - au;
      const int r0 = S->radr[t], r1 = S->radr[t + 1], ld = S->rld[t];
      float* Lb = S->L + S->rbase[t] + S->bcol[b];
      const bool diag = t == u;
#pragma unroll 1
      for (int i = lane & 7; i < st; i += 8) {
#pragma unroll 1
        for (int j0 = 0; j0 < (diag ? i + 1 : su); j0 += 8) {
          const int jn = min(8, (diag ? i + 1 : su) - j0);
          float h[8];
#pragma unroll
          for (int j = 0; j < 8; j++)
            h[j] = j < jn && diag ? (msp ? Lb[i * ld + j0 + j] : qM[size_t(at + i) * nv + au + j0 + j]) : 0.f;
#pragma unroll 1
          for (int q = r0; q < r1; q++) {
            const unsigned e = S->rlist[q];
            const int k = e & 0xffff, o = e >> 16;
            const float D = S->sD[k];
            if (D == 0.f || (!diag && o != u)) continue;
            // the row's entries: its lower tree's, then the other's
            const float *Jt, *Ju;
            if (cw) {
              Jt = S->cj + k * cw;
              if (o < t) Jt += S->tadr[o + 1] - S->tadr[o];
              Ju = diag ? Jt : S->cj + k * cw;
            } else {
              Ju = d.efc_J + size_t(adr + k) * nv + au;
              Jt = d.efc_J + size_t(adr + k) * nv + at;
            }
            const float Ji = Jt[i];
            Ju += j0;
#pragma unroll
            for (int j = 0; j < 8; j++)
              if (j < jn) h[j] = fmaf(Ji * Ju[j], D, h[j]);
          }
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (j < jn) Lb[i * ld + j0 + j] = h[j];
        }
      }
    }
    __syncthreads();
  }

  // the factor's nonzero pairs into efc_h
  __device__ void store_factor() {
#pragma unroll 1
    for (int b = warp; b < S->nblk; b += NW) {
      const int t = S->blk[b] >> 8, u = S->blk[b] & 255;
      const int at = S->tadr[t], au = S->tadr[u], st = S->tadr[t + 1] - at, su = S->tadr[u + 1] - au;
      const float* Lb = S->L + S->rbase[t] + S->bcol[b];
#pragma unroll 1
      for (int e = lane; e < st * su; e += 32) {
        const int i = e / su, j = e - i * su;
        if (t != u || j <= i) H[size_t(at + i) * nv + au + j] = Lb[i * S->rld[t] + j];
      }
    }
  }

  __device__ void assemble_hessian() {
    lower_mass<float>(H, nv);
    int* nzi = reinterpret_cast<int*>(nz);
    float* nzv = nz + round4i(nv);
    for (int k = 0; k < n; k++) {
      const int r = adr + k;
      if (!d.efc_active[r]) continue;
      const float D = d.efc_D[r];
      if (D == 0.f) continue;
      const float* J = d.efc_J + size_t(r) * nv;
      int cnt = 0;
      for (int base = 0; base < nv; base += 256) {  // eight 32-column chunks loaded, then compacted
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const int c = base + 32 * q + lane;
          v[q] = c < nv ? J[c] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const unsigned mk = __ballot_sync(WARP_FULL, v[q] != 0.f);
          if (v[q] != 0.f) {
            const int p = cnt + __popc(mk & ((1u << lane) - 1u));
            nzi[p] = base + 32 * q + lane;
            nzv[p] = v[q];
          }
          cnt += __popc(mk);
        }
      }
      __syncwarp();
      for (int a = 0; a < cnt; a++) {
        const int i = nzi[a];
        if (i % NW != warp) continue;
        float* Hi = H + size_t(i) * nv;
        const float va = nzv[a];
        for (int b = lane; b <= a; b += 32) Hi[nzi[b]] += va * nzv[b] * D;
      }
      __syncwarp();
    }
    __syncthreads();
  }

  // H = tril(qM) + sum over active rows of D J'J on the tensor pipe in split TF32 (mjb_tc.cuh):
  // H = qM + A B with A = J^T (nv x n) and B = diag(c) J (n x nv), c = D on active rows and 0
  // elsewhere; warp q takes the 16-row m-tiles mt = q, q + NW, ... and, four at a time, the m16n8
  // tiles of that row band that touch the lower triangle; the k dimension runs over the world's
  // rows eight at a time, the accumulators start from qM; writes the lower triangle of Hout (row
  // stride ldh elements: efc_h; or, PACKED, the precision form's packed FP64 triangle).
  template <typename TH, bool PACKED = false>
  __device__ void assemble_hessian_tc(TH* Hout, int ldh) {
    const int g = lane >> 2, t = lane & 3;
    const int nmt = (nv + 15) >> 4, ncol8 = (nv + 7) >> 3;
    const float* J = d.efc_J + size_t(adr) * nv;
    // the accumulators start from the mass matrix: read from qM when dense; the sparse layout is
    // first expanded into Hout's lower triangle and read back from there
    const bool sparse = m.is_sparse;
    if (sparse) lower_mass<TH, PACKED>(Hout, ldh);
    auto mass = [&](int r, int c) -> float {
      if (r >= nv || c >= nv) return 0.f;
      if (!sparse) return qM[size_t(r) * nv + c];
      return c <= r ? float(Hout[(PACKED ? size_t(tri(r)) : size_t(r) * ldh) + c]) : 0.f;
    };
    for (int mt = warp; mt < nmt; mt += NW) {
      const int r0 = 16 * mt + g, r1 = r0 + 8;
      const int nnt = min((16 * mt + 15) / 8 + 1, ncol8);
      for (int nt0 = 0; nt0 < nnt; nt0 += 4) {
        float acc[4][4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int c = 8 * (nt0 + q) + 2 * t;
          acc[q][0] = mass(r0, c);
          acc[q][1] = mass(r0, c + 1);
          acc[q][2] = mass(r1, c);
          acc[q][3] = mass(r1, c + 1);
        }
        for (int k0 = 0; k0 < n; k0 += 8) {
          const int ka = k0 + t, kb = ka + 4;
          const bool va = ka < n, vb = kb < n;
          const float ca = (va && d.efc_active[adr + ka]) ? d.efc_D[adr + ka] : 0.f;
          const float cb = (vb && d.efc_active[adr + kb]) ? d.efc_D[adr + kb] : 0.f;
          const float* Ja = J + size_t(va ? ka : 0) * nv;
          const float* Jb = J + size_t(vb ? kb : 0) * nv;
          const FragA a = frag_a((va && r0 < nv) ? Ja[r0] : 0.f, (va && r1 < nv) ? Ja[r1] : 0.f,
                                 (vb && r0 < nv) ? Jb[r0] : 0.f, (vb && r1 < nv) ? Jb[r1] : 0.f);
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const int c = 8 * (nt0 + q) + g;
            if (nt0 + q < nnt) {
              const FragB b = frag_b((va && c < nv) ? ca * Ja[c] : 0.f, (vb && c < nv) ? cb * Jb[c] : 0.f);
              mma_3xtf32(acc[q], a, b);
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int c = 8 * (nt0 + q) + 2 * t;
#pragma unroll
          for (int e = 0; e < 2; e++) {
            if (r0 < nv && c + e <= r0)
              Hout[(PACKED ? size_t(tri(r0)) : size_t(r0) * ldh) + c + e] = TH(acc[q][e]);
            if (r1 < nv && c + e <= r1)
              Hout[(PACKED ? size_t(tri(r1)) : size_t(r1) * ldh) + c + e] = TH(acc[q][2 + e]);
          }
        }
      }
    }
    __syncthreads();
  }

  // solver.py:176-312
  __device__ void update_gradient() {
    float gd[1] = {0.f};
#pragma unroll kU
    for (int i = tid; i < nv; i += NT) {
      const float g = Ma[i] - qfrc_smooth[i] - qfrc_constraint[i];
      grad[i] = g;
      gd[0] += g * g;
    }
    sum<1>(gd);
    grad_dot = gd[0];
    if (m.solver == 1) {  // CG: Mgrad = M^-1 grad
      if (warp == 0) cta_solve_m(m, d, w, Mgrad, grad, lane);
      __syncthreads();
      return;
    }
    if (!(reuse && factored && !changed)) {
      if (PREC) {  // H in split TF32 straight into the FP64 tile, factored there in FP64
        assemble_hessian_tc<double, true>(Ld, 0);
        chol_cta_d<NW>(Ld, rdg, nv, warp, lane);
#pragma unroll kU
        for (int e = tid; e < nv * nv; e += NT) {  // efc_h keeps the factor (FP32-rounded)
          const int i = e / nv, j = e - i * nv;
          if (j <= i) H[e] = float(Ld[tri(i) + j]);
        }
      } else {
        if (sparse()) {
          assemble_hessian_sparse();
          chol_cta_sparse<NW, SH>(nv, T, *S, warp, lane);
        } else if constexpr (NW > 1) {
          if (!TREES && tc) assemble_hessian_tc(H, nv);
          else assemble_hessian();
          chol_cta<NW>(H, nv, nv, T, warp, lane);
        }
      }
      factored = true;
    }
    if (warp == 0) {
      if (PREC && nv <= 128) cho_solve_d_regs(Ld, rdg, nv, Mgrad, grad, lane);
      else if (PREC) cho_solve_d_warp(Ld, rdg, nv, vd, Mgrad, grad, lane);
    }
    if (sparse()) {
      cho_solve_cta_sparse<NW, SH>(nv, Mgrad, grad, zv, *S, warp, lane);
      if (!isfinite(grad_dot)) spread_nonfinite(grad, Mgrad, nv, tid, NT);
    } else if constexpr (!PREC && NW > 1) cho_solve_cta<NW>(H, nv, nv, Mgrad, grad, zv, red, warp, lane);
    __syncthreads();
  }

  // solver.py:737-869 with the iterative (:339-664) or parallel (:667-734) line search
  __device__ void linesearch() {
    if constexpr (NW == 1) {  // solve_generic's own search
      SolverCtx c{m, d, w, lane, nv, adr, n};
      c.qacc = qacc;
      c.Ma = Ma;
      c.search = search;
      c.mv = mv;
      c.qfrc_smooth = qfrc_smooth;
      c.gauss = gauss;
      c.search_dot = search_dot;
      c.alpha = alpha;
      c.gtol = gtol;
      // the smooth part as the compiler fuses it in solve_generic: the two give the same bits
      linesearch_with(c, [&]() { mul_m(mv, search); }, [&](int k) { return row_dot(k, search); },
                      [](const float* q, float a, float* out) { eval_pt3_fma(q, a, out); });
      alpha = c.alpha;
      gtol = c.gtol;
      for (int k = 0; k < 3; k++) qg[k] = c.qg[k];
    } else {
      linesearch_cta();
    }
  }
  __device__ void linesearch_cta() {
    mul_m(mv, search);
    {
      float q[3] = {0.f, 0.f, 0.f};
#pragma unroll kU
      for (int i = tid; i < nv; i += NT) {
        q[0] += gauss / float(nv);
        q[1] += search[i] * (Ma[i] - qfrc_smooth[i]);
        q[2] += 0.5f * search[i] * mv[i];
      }
      const float z[3] = {0.f, 0.f, 0.f};
      ls_sums<3>(z, q);
      qg[0] = q[0];
      qg[1] = q[1];
      qg[2] = q[2];
    }
    rows_dot(search, d.efc_jv, nullptr);
    // up to kRegRows rows per thread stay in registers through the line search
    constexpr int kRegRows = 3;
    const bool regs = n <= kRegRows * NT;
    float rJ[kRegRows], rv[kRegRows], rq[kRegRows][3];
#pragma unroll kU
    for (int k = tid, e = 0; k < n; k += NT, e++) {
      const int r = adr + k;
      const float jv = d.efc_jv[r], Jaref = d.efc_Jaref[r], D = d.efc_D[r];
      const float q0 = 0.5f * Jaref * Jaref * D, q1 = jv * Jaref * D, q2 = 0.5f * jv * jv * D;
      d.efc_quad[3 * r] = q0;
      d.efc_quad[3 * r + 1] = q1;
      d.efc_quad[3 * r + 2] = q2;
#pragma unroll
      for (int h = 0; h < kRegRows; h++)
        if (e == h) {
          rJ[h] = Jaref;
          rv[h] = jv;
          rq[h][0] = q0;
          rq[h][1] = q1;
          rq[h][2] = q2;
        }
    }
    // f(Jaref, jv, quad) for each of this thread's rows
    auto rows = [&](auto&& f) {
      if (regs) {
#pragma unroll
        for (int h = 0; h < kRegRows; h++)
          if (tid + h * NT < n) f(rJ[h], rv[h], rq[h]);
      } else {
#pragma unroll kU
        for (int k = tid; k < n; k += NT) {
          const int r = adr + k;
          f(d.efc_Jaref[r], d.efc_jv[r], d.efc_quad + 3 * r);
        }
      }
    };
    if (m.ls_parallel) {
      int best = 0;
      float bestc = 0.f;
#pragma unroll 1
      for (int c = 0; c < m.nlsp; c++) {
        const float a = m.alpha_candidate[c];
        float tt[3] = {0.f, 0.f, 0.f};
        rows([&](float jaref, float jv, const float* q) {
          if (jaref + a * jv < 0.f) {
            tt[0] += q[0];
            tt[1] += q[1];
            tt[2] += q[2];
          }
        });
        ls_sums<3>(qg, tt);
        const float cst = a * a * tt[2] + a * tt[1] + tt[0];
        if (c == 0 || cst < bestc) {
          bestc = cst;
          best = c;
        }
      }
      alpha = m.alpha_candidate[best];
    } else {
      const float scale = m.meaninertia * float(max(1, nv));
      gtol = m.tolerance * m.ls_tolerance * sqrtf(search_dot) * scale;
      float p0[3] = {0.f, 0.f, 0.f};
      rows([&](float jaref, float, const float* q) {
        if (jaref >= 0.f) return;
        p0[0] += q[0];
        p0[1] += q[1];
        p0[2] += 2.f * q[2];
      });
      {
        const float base[3] = {qg[0], qg[1], 2.f * qg[2]};
        ls_sums<3>(base, p0);
      }
      // the total cost polynomial's value and derivatives at up to three step sizes at once
      auto totals = [&](int na, const float* al, float (*out)[3]) {
        float acc[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        rows([&](float jaref, float jv, const float* q) {
#pragma unroll
          for (int t = 0; t < 3; t++) {
            if (t < na && jaref + al[t] * jv < 0.f) {
              float p[3];
              eval_pt3(q, al[t], p);
              acc[3 * t] += p[0];
              acc[3 * t + 1] += p[1];
              acc[3 * t + 2] += p[2];
            }
          }
        });
        float base[9];
#pragma unroll
        for (int t = 0; t < 3; t++) {
          float gq[3] = {0.f, 0.f, 0.f};
          if (t < na) eval_pt3(qg, al[t], gq);
          base[3 * t] = gq[0];
          base[3 * t + 1] = gq[1];
          base[3 * t + 2] = gq[2];
        }
        ls_sums<9>(base, acc);
#pragma unroll
        for (int t = 0; t < 3; t++) {
          out[t][0] = acc[3 * t];
          out[t][1] = acc[3 * t + 1];
          out[t][2] = acc[3 * t + 2];
        }
      };
      float lo_alpha = -safe_div(p0[1], p0[2]), hi_alpha = 0.f;
      float lo[3], hi[3];
      bool done = false;
#pragma unroll 1
      for (int it = -1; it < m.ls_iterations && !done; it++) {
        float al[3] = {lo_alpha, 0.f, 0.f};
        if (it >= 0) {
          al[0] = lo_alpha - safe_div(lo[1], lo[2]);
          al[1] = hi_alpha - safe_div(hi[1], hi[2]);
          al[2] = 0.5f * (lo_alpha + hi_alpha);
        }
        float o[3][3];
        totals(it < 0 ? 1 : 3, al, o);
        if (it < 0) {  // the bracket: the start and the Newton step
          if (o[0][1] < p0[1]) {
#pragma unroll
            for (int e = 0; e < 3; e++) {
              lo[e] = o[0][e];
              hi[e] = p0[e];
            }
            hi_alpha = 0.f;
          } else {
#pragma unroll
            for (int e = 0; e < 3; e++) {
              hi[e] = o[0][e];
              lo[e] = p0[e];
            }
            hi_alpha = lo_alpha;
            lo_alpha = 0.f;
          }
          continue;
        }
        float *lon = o[0], *hin = o[1], *mid = o[2];
        // _swap (solver.py:537-617)
        const bool s1 = in_bracket(lo, lon);
        if (s1) { lo[0] = lon[0]; lo[1] = lon[1]; lo[2] = lon[2]; lo_alpha = al[0]; }
        const bool s2 = in_bracket(lo, mid);
        if (s2) { lo[0] = mid[0]; lo[1] = mid[1]; lo[2] = mid[2]; lo_alpha = al[2]; }
        const bool s3 = in_bracket(lo, hin);
        if (s3) { lo[0] = hin[0]; lo[1] = hin[1]; lo[2] = hin[2]; lo_alpha = al[1]; }
        const bool t1 = in_bracket(hi, hin);
        if (t1) { hi[0] = hin[0]; hi[1] = hin[1]; hi[2] = hin[2]; hi_alpha = al[1]; }
        const bool t2 = in_bracket(hi, mid);
        if (t2) { hi[0] = mid[0]; hi[1] = mid[1]; hi[2] = mid[2]; hi_alpha = al[2]; }
        const bool t3 = in_bracket(hi, lon);
        if (t3) { hi[0] = lon[0]; hi[1] = lon[1]; hi[2] = lon[2]; hi_alpha = al[0]; }
        done = (!(s1 || s2 || s3) && !(t1 || t2 || t3)) || (lo[1] < 0.f && lo[1] > -gtol) ||
               (hi[1] > 0.f && hi[1] < gtol);
        float a = 0.f;
        const bool improved = lo[0] < p0[0] || hi[0] < p0[0];
        const bool lo_better = lo[0] < hi[0];
        if (improved && lo_better) a = lo_alpha;
        if (improved && !lo_better) a = hi_alpha;
        alpha = a;
      }
    }
    // solver.py:816-841
#pragma unroll kU
    for (int i = tid; i < nv; i += NT) {
      qacc[i] += alpha * search[i];
      Ma[i] += alpha * mv[i];
    }
#pragma unroll kU
    for (int k = tid; k < n; k += NT) d.efc_Jaref[adr + k] += alpha * d.efc_jv[adr + k];
    __syncthreads();
  }

  // search = -Mgrad (+ beta search for CG); returns search . search
  __device__ void new_search() {
    float sd[1] = {0.f};
#pragma unroll kU
    for (int i = tid; i < nv; i += NT) {
      float v = -Mgrad[i];
      if (m.solver == 1) v += beta * search[i];
      search[i] = v;
      sd[0] += v * v;
    }
    sum<1>(sd);
    search_dot = sd[0];
  }

  __device__ void run() {
    const float* ws = d.qacc_warmstart + W(w, nv);
    if constexpr (NW == 1) {  // solve_generic's arithmetic, which takes the worlds that do not fit
      if (n > SH::kRows) return;  // k_solve_many_rows's
      sp = sparse_shape<NW, SH>(m, d.efc_J + size_t(adr) * nv, n, H, *S, cw, warp, lane);
      if (!sp) {
        solve_generic(m, d, w, lane, H, nz, true);
        return;
      }
    } else if constexpr (TREES)
      sp = sparse_shape<NW, SH>(m, d.efc_J + size_t(adr) * nv, n, H, *S, cw, warp, lane);
#pragma unroll kU
    for (int i = tid; i < nv; i += NT) qacc[i] = ws[i];
    __syncthreads();
    // _create_context (solver.py:26-72)
    cost = __int_as_float(0x7f800000);
    search_dot = 0.f;
    alpha = 0.f;
    gtol = 0.f;
    beta = 0.f;
    qg[0] = qg[1] = qg[2] = 0.f;
    rows_dot(qacc, d.efc_Jaref, d.efc_aref);
    mul_m(Ma, qacc);
    float* prev_grad = d.efc_prev_grad ? d.efc_prev_grad + W(w, nv) : nullptr;
    float* prev_Mgrad = d.efc_prev_Mgrad ? d.efc_prev_Mgrad + W(w, nv) : nullptr;
    bool done = false;
#pragma unroll 1
    for (int it = -1; it < m.iterations && !done; it++) {  // it = -1: the start
      if (it >= 0) {
        linesearch();
        if (m.solver == 1) {
#pragma unroll kU
          for (int i = tid; i < nv; i += NT) {
            prev_grad[i] = grad[i];
            prev_Mgrad[i] = Mgrad[i];
          }
          __syncthreads();
        }
      }
      update_constraint();
      update_gradient();
      if (it >= 0 && m.solver == 1) {  // Polak-Ribiere (solver.py:918-970)
        float nd[2] = {0.f, 0.f};
#pragma unroll kU
        for (int i = tid; i < nv; i += NT) {
          nd[0] += grad[i] * (Mgrad[i] - prev_Mgrad[i]);
          nd[1] += prev_grad[i] * prev_Mgrad[i];
        }
        sum<2>(nd);
        beta = fmaxf(0.f, nd[0] / fmaxf(kMinVal, nd[1]));
      }
      new_search();
      const float scale = m.meaninertia * float(max(1, nv));
      done = it >= 0 && ((prev_cost - cost) / scale < m.tolerance || sqrtf(grad_dot) / scale < m.tolerance);
    }
    if (sparse() && factored && S->L != H) store_factor();
    float* wsw = d.qacc_warmstart + W(w, nv);
#pragma unroll kU
    for (int i = tid; i < nv; i += NT) wsw[i] = qacc[i];
    if (tid == 0) {
      if (d.efc_cost) d.efc_cost[w] = cost;
      if (d.efc_prev_cost) d.efc_prev_cost[w] = prev_cost;
      if (d.efc_gauss) d.efc_gauss[w] = gauss;
      if (d.efc_grad_dot) d.efc_grad_dot[w] = grad_dot;
      if (d.efc_search_dot) d.efc_search_dot[w] = search_dot;
      if (d.efc_gtol) d.efc_gtol[w] = gtol;
      if (d.efc_alpha) d.efc_alpha[w] = alpha;
      if (d.efc_beta) d.efc_beta[w] = beta;
      if (d.efc_done) d.efc_done[w] = done ? 1 : 0;
      if (d.efc_solver_niter) d.efc_solver_niter[w] = 0;  // never advanced by the reference
      if (d.efc_quad_gauss) {
        d.efc_quad_gauss[3 * w] = qg[0];
        d.efc_quad_gauss[3 * w + 1] = qg[1];
        d.efc_quad_gauss[3 * w + 2] = qg[2];
      }
    }
    __syncthreads();
  }
};

// One world's solve by the whole CTA; smem: cta_solver_smem_floats(nv, NW, PREC, TREES) floats
template <int NW, bool PREC, bool TREES>
__device__ void solve_cta(const MjbModel& m, const MjbData& d, int w, float* smem, bool tc) {
  const int nv = m.nv;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  CtaSolver<NW, PREC, TREES> s{m, d, w, tid, lane, warp, nv, d.world_efcadr[w], d.world_nefc[w]};
  s.qacc = d.qacc + W(w, nv);
  s.Ma = d.efc_Ma + W(w, nv);
  s.grad = d.efc_grad + W(w, nv);
  s.Mgrad = d.efc_Mgrad + W(w, nv);
  s.search = d.efc_search + W(w, nv);
  s.mv = d.efc_mv + W(w, nv);
  s.qfrc_constraint = d.qfrc_constraint + W(w, nv);
  s.H = d.efc_h + W(w, nv * nv);
  s.qM = d.qM + (m.is_sparse ? W(w, m.nM) : W(w, nv * nv));
  s.qfrc_smooth = d.qfrc_smooth + W(w, nv);
  s.qacc_smooth = d.qacc_smooth + W(w, nv);
  s.red = smem;
  s.T = smem + 32 * NW;
  s.zv = smem + 32 * NW + 32 * 36 + 32;
  float* part = smem + round4i(32 * NW + 32 * 36 + 32 + round4i(nv));  // structure or scratch
  s.nz = part + warp * 2 * round4i(nv);
  s.S = reinterpret_cast<SparseFor<NW>*>(part);
  s.Ld = PREC ? reinterpret_cast<double*>(smem + cta_solver_smem_base(nv, NW, false)) : nullptr;
  s.vd = PREC ? s.Ld + tri(nv) : nullptr;
  s.rdg = PREC ? s.vd + nv : nullptr;
  s.tc = tc;
  s.run();
}

}  // namespace mjb
