// Device kernels of the HIF factor / apply path (sm_100a, FP64).
//
// The reference performs these steps with LAPACK/BLAS on one CPU core
// (arbenson/HIFDE3D src/Factor.cpp, include/Schur.hpp, src/InterpDecomp.cpp).
// Here each level phase is a handful of batched launches over every cell or
// face of the level:
//   gather      dense blocks from the 7-point stencil plus the live Schur
//               complement blocks (replaces DenseSubmatrix over std::map and
//               UpdateMatrixAndDOFs, src/Factor.cpp:262-311);
//   sweep       in-place Gauss-Jordan elimination of the redundant DOFs of a
//               block [A22 A21; A12 A11]: yields A22^{-1}, X = A22^{-1} A21 and
//               A11 - A12 X in one pass (Schur.hpp:72-100);
//   dgemm       batched FP64 GEMM (rank-128 sweep updates, the QR by phases, ID
//               rotations);
//   id          column-pivoted QR (narrow faces Householder, wide ones by phases of
//               pivoted Cholesky), rank test and interpolation matrix
//               (InterpDecomp.cpp:86-138);
//   gemv        gather / multiply / scatter sweeps of Apply (Factor.cpp:992-1081).
#include "hif_kernels.cuh"

#include <cooperative_groups.h>

#include <cfloat>
#include <climits>
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>

namespace hif {

namespace {

// Kernel attributes are per device (cudaFuncSetAttribute acts on the current
// device) and launchers run on several host threads at once (the serving
// loop's factor workers): every one-time setting goes through this table,
// keyed by (device, kernel), under one mutex.
std::mutex g_attr_mu;
std::map<std::pair<int, const void*>, size_t> g_attr_smem;

// Multiprocessor count of the current device (cached per device).
int sm_count() {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_attr_mu);
  static std::map<int, int> sms;
  auto it = sms.find(dev);
  if (it != sms.end()) return it->second;
  int n = 0;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  if (n <= 0) n = 1;
  sms[dev] = n;
  return n;
}

// Raises `fn`'s dynamic shared-memory limit on the current device to at least
// `bytes` (never lowers it).
void ensure_smem(const void* fn, size_t bytes) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_attr_mu);
  size_t& cur = g_attr_smem[{dev, fn}];
  if (bytes > cur) {
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    cur = bytes;
  }
}

__device__ __forceinline__ int find_desc(const int* __restrict__ off, int nd, int t) {
  int lo = 0, hi = nd - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum; every thread gets the result. scratch: >= 32 doubles.
__device__ double block_sum(double v, double* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  double t = (threadIdx.x < nw) ? scratch[threadIdx.x] : 0.0;
  if (warp == 0) t = warp_sum(t);
  if (threadIdx.x == 0) scratch[32] = t;
  __syncthreads();
  double r = scratch[32];
  __syncthreads();
  return r;
}

}  // namespace

// ===========================================================================
// Gather / assembly
// ===========================================================================
// Tiles of 32 rows x 64 columns: lane x of warp w assembles row x of columns
// w, w + 8, ..., w + 56, so a thread's row, its stencil row and its row covers
// (up to three sources and positions) stay in registers, and a column's covers (each
// turned into a pointer to the source's column) are warp-uniform shared-memory reads.
constexpr int kGTM = 32, kGTN = 64;

int gather_tiles(int m, int n) {
  return ((m + kGTM - 1) / kGTM) * ((n + kGTN - 1) / kGTN);
}

__device__ __forceinline__ void resolve_cover(const GatherTarget& g, int p,
                                              const int* __restrict__ dof_src,
                                              const int* __restrict__ src_owner,
                                              long long ncell3, CoverEntry* out) {
#pragma unroll
  for (int c = 0; c < kCover; ++c) {
    CoverEntry ce{-1, 0};
    if (p >= 0 && g.mode != 2) {
      const int s = dof_src[(2 * c) * ncell3 + p];
      if (s >= 0) {
        const bool ok = (g.mode == 0) ? (src_owner[s] == g.owner)
                                      : (s == g.allowA || s == g.allowB);
        if (ok) ce = CoverEntry{s, dof_src[(2 * c + 1) * ncell3 + p]};
      }
    }
    out[c] = ce;
  }
}

// Persistent over the tile list: CTA b assembles the contiguous tiles
// [b chunk, (b + 1) chunk), so the target of its first tile is found once by
// binary search and the rest by stepping through tile_off (a per-tile search
// costs ~log2(targets) dependent loads, more than a small tile's own work).
__global__ void __launch_bounds__(256) k_gather(const GatherTarget* __restrict__ tg,
                                                const int* __restrict__ tile_off, int ntg,
                                                int total_tiles,
                                                const SourceDesc* __restrict__ src,
                                                const int* __restrict__ src_owner,
                                                const int* __restrict__ dof_src,
                                                const double* __restrict__ band,
                                                long long ncell3, int NC) {
  const int chunk = (total_tiles + gridDim.x - 1) / gridDim.x;
  const int t0 = blockIdx.x * chunk, t1 = min(total_tiles, t0 + chunk);
  if (t0 >= t1) return;
  int d = find_desc(tile_off, ntg, t0);
  int dbeg = tile_off[d], dend = tile_off[d + 1];
  __shared__ int s_col[kGTN];
  __shared__ int s_src[kGTN][kCover];             // a column's sources, -2: none
  __shared__ const double* s_base[kGTN][kCover];  // their columns
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int NC2 = NC * NC;
  for (int t = t0; t < t1; ++t) {
    while (t >= dend) {
      ++d;
      dbeg = dend;
      dend = tile_off[d + 1];
    }
    const GatherTarget g = tg[d];
    const int local = t - dbeg;
    const int tiles_m = (g.m + kGTM - 1) / kGTM;
    const int i0 = (local % tiles_m) * kGTM, j0 = (local / tiles_m) * kGTN;
    __syncthreads();  // the previous tile's readers of the column tables are done
    if (threadIdx.x < kGTN) {
      const int j = j0 + threadIdx.x;
      const int q = (j < g.n) ? g.cols[j] : -1;
      s_col[threadIdx.x] = q;
      CoverEntry cc[kCover];
      resolve_cover(g, q, dof_src, src_owner, ncell3, cc);
#pragma unroll
      for (int c = 0; c < kCover; ++c) {
        const bool has = cc[c].src >= 0;
        s_src[threadIdx.x][c] = has ? cc[c].src : -2;
        if (has) {
          const SourceDesc sd = src[cc[c].src];
          s_base[threadIdx.x][c] = sd.ptr + (long long)cc[c].pos * sd.ld;
        } else {
          s_base[threadIdx.x][c] = nullptr;
        }
      }
    }
    // this thread's row: DOF, stencil row, sources and its positions in them
    const int i = i0 + lane;
    const int p = (i < g.m) ? g.rows[i] : -1;
    CoverEntry rc[kCover];
    resolve_cover(g, p, dof_src, src_owner, ncell3, rc);
    __syncthreads();
    if (i < g.m) {
      const bool row_a0 = i < g.a0_skip;
      const bool row_a22 = g.a22_out != nullptr && i < g.r;
      const int ld = (int)g.ld;
      double* orow = g.out + i;
#pragma unroll 4
      for (int cc = warp; cc < kGTN; cc += 8) {
        const int j = j0 + cc;
        if (j >= g.n) break;
        // sources holding both DOFs, in the column's cover order: a row is in a source
        // at most once, so its position is selected and one load is issued per column
        // source (a column's sources are warp-uniform shared-memory reads)
        double tv[kCover];
#pragma unroll
        for (int c = 0; c < kCover; ++c) {
          const int sc = s_src[cc][c];
          int pos = -1;
#pragma unroll
          for (int a = kCover - 1; a >= 0; --a) pos = rc[a].src == sc ? rc[a].pos : pos;
          tv[c] = pos >= 0 ? __ldg(s_base[cc][c] + pos) : 0.0;
        }
        double v = 0.0;
        if (row_a0 || j < g.a0_skip) {
          // stencil term: q - p in {0, -1, 1, -NC, NC, -NC^2, NC^2} -> bands 0..6
          const int dd = s_col[cc] - p, ad = abs(dd);
          if (ad == 0 || ad == 1 || ad == NC || ad == NC2) {
            const int b = (ad == 0 ? 0 : (ad == 1 ? 1 : (ad == NC ? 3 : 5))) + (dd > 0 ? 1 : 0);
            v = band[b * ncell3 + p];
          }
        }
#pragma unroll
        for (int c = 0; c < kCover; ++c) v += tv[c];
        orow[(long long)j * ld] = v;
        if (row_a22 && j < g.r) g.a22_out[i + (long long)j * g.r] = v;
      }
    }
  }
}

void launch_gather(const GatherTarget* d_tg, const int* d_tile_off, int ntg, int total_tiles,
                   const SourceDesc* d_src, const int* d_src_owner, const int* d_dof_src,
                   const double* d_band, long long ncell3, int NC, cudaStream_t s) {
  if (total_tiles <= 0) return;
  // 8 resident CTAs of 256 threads per SM, several waves' worth of
  // chunks so that uneven tiles even out
  const int grid = std::min(total_tiles, sm_count() * 8 * 4);
  k_gather<<<grid, 256, 0, s>>>(d_tg, d_tile_off, ntg, total_tiles, d_src, d_src_owner,
                                d_dof_src, d_band, ncell3, NC);
}

// ===========================================================================
// Batched FP64 GEMM on the FP64 tensor cores (DMMA, mma.sync m8n8k4), 64 x 64 x 16
// tiles by 4 warps (32 x 32 each), four CTAs per SM; and 128 x 128 x 16 tiles by 16
// warps, for products that need one tile along a dimension (in-place panels) and as
// the tuner's other candidate. Operands go through a cp.async pipeline (8-byte
// copies: sub-matrix views are only 8-byte aligned; out-of-range elements are
// zero-filled by the copy).
//
// Bound: the DMMA pipe. What kept it idle was the work between two stages' products:
// recomputing every copy's address and bounds (~15 instructions a copy) right after
// the barrier, with all 16 warps of one CTA at the same point. So a thread's copies
// are one pointer plus constant strides, the next stage's copies are issued a quarter
// after each k-step of 4, and four independent CTAs fill each other's barriers,
// fragment loads and epilogues. 8000 x 8000 (odd sizes), TF/s before -> after, at
// k = 2050: 23.8 -> 31.4, transposed A with beta = 1: 23.2 -> 31.1, k = 128 with
// beta = 1: 18.2 -> 28.0 (cuBLAS, aligned: 34.6 at k = 2050); the 128 x 128 form 30.8,
// 30.3 and 22.1. Stage rows are padded to 4 mod 16 doubles: a fragment load (8 rows x
// 4 k) then touches each bank pair once per half warp.
// ===========================================================================
int dgemm_tiles(int m, int n, int tile) {
  if (m <= 0 || n <= 0) return 0;
  return ((m + tile - 1) / tile) * ((n + tile - 1) / tile);
}

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem, bool valid) {
  const unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
  const int bytes = valid ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(gmem),
               "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

constexpr int kGBK = 16;  // k per stage
template <int BM, int BN, int ST>
constexpr int dgemm_smem() {
  return ST * kGBK * (BM + 4 + BN + 4) * (int)sizeof(double);
}

// Warp tile 32 x 32 = 4 x 4 MMA tiles. Fragments (PTX ISA, m8n8k4 .f64): with
// g = lane / 4, t = lane % 4, A holds (row g, k t), B holds (k t, col g), C holds
// (row g, cols 2t and 2t + 1).
template <int BM, int BN, int ST, int MINB>
__global__ void __launch_bounds__(BM * BN / 32, MINB)
    k_dgemm(const GemmDesc* __restrict__ descs, const int* __restrict__ tile_off, int nd) {
  constexpr int T = BM * BN / 32;  // threads
  constexpr int SA = BM + 4, SB = BN + 4;
  constexpr int QA = BM * kGBK / T, QB = BN * kGBK / T;  // copies of a thread per stage
  constexpr int KS = kGBK / 4;
  static_assert(T % BM == 0 && T % BN == 0 && T % kGBK == 0 && QA % KS == 0 && QB % KS == 0,
                "a thread's copies differ by constant strides, an equal share per k-step");
  extern __shared__ double lsm[];
  double* As = lsm;                   // [stage][k][SA]
  double* Bs = lsm + ST * kGBK * SA;  // [stage][k][SB]
  const int di = find_desc(tile_off, nd, blockIdx.x);
  const GemmDesc g = descs[di];
  const int local = blockIdx.x - tile_off[di];
  const int tiles_m = (g.m + BM - 1) / BM;
  const int m0 = (local % tiles_m) * BM, n0 = (local / tiles_m) * BN;
  // lower: 1 skips the 128 x 128 blocks above the diagonal, 2 the tiles above it
  if (g.lower == 1 && m0 / 128 < n0 / 128) return;
  if (g.lower == 2 && m0 < n0) return;
  if (g.skip && *g.skip) return;
  const int kend = g.a_lower ? min(g.k, m0 + BM) : g.k;
  const int kbeg = g.b_lower ? min(kend, n0) : 0;  // n0: a multiple of kGBK
  const int nk = (kend - kbeg + kGBK - 1) / kGBK;
  const int tid = threadIdx.x;
  const bool ta = g.transA != 0, tb = g.transB != 0;
  // copy q of a thread: A row amm (+ q T / BK if transposed), k akk (+ q T / BM if not)
  const int amm = ta ? tid / kGBK : tid % BM, akk = ta ? tid % kGBK : tid / BM;
  const int bnn = tb ? tid % BN : tid / kGBK, bkk = tb ? tid / BN : tid % kGBK;
  const long long astep = (long long)(ta ? T / kGBK : T / BM) * g.lda;
  const long long bstep = (long long)(tb ? T / BN : T / kGBK) * g.ldb;
  const long long aadv = ta ? kGBK : (long long)kGBK * g.lda;
  const long long badv = tb ? (long long)kGBK * g.ldb : kGBK;
  const int ak = kbeg + akk, bk = kbeg + bkk;
  const double* ap = ta ? g.A + ak + (long long)(m0 + amm) * g.lda
                        : g.A + (m0 + amm) + (long long)ak * g.lda;
  const double* bp = tb ? g.B + (n0 + bnn) + (long long)bk * g.ldb
                        : g.B + bk + (long long)(n0 + bnn) * g.ldb;
  const int as0 = akk * SA + amm, bs0 = bkk * SB + bnn;
  const int asq = ta ? T / kGBK : (T / BM) * SA, bsq = tb ? (T / BN) * SB : T / kGBK;
  unsigned amask = 0, bmask = 0;  // copies whose row / column is in range
#pragma unroll
  for (int q = 0; q < QA; ++q)
    if (m0 + amm + (ta ? (T / kGBK) * q : 0) < g.m) amask |= 1u << q;
#pragma unroll
  for (int q = 0; q < QB; ++q)
    if (n0 + bnn + (tb ? 0 : (T / kGBK) * q) < g.n) bmask |= 1u << q;
  // copies [q0, q1) of the stage whose first k is k0; ap / bp point at that stage
  auto issue = [&](int stage, int k0, int part, int parts) {
    double* as = As + stage * kGBK * SA + as0;
    double* bs = Bs + stage * kGBK * SB + bs0;
#pragma unroll
    for (int q = 0; q < QA; ++q)
      if (q >= QA / parts * part && q < QA / parts * (part + 1)) {
        const bool ok = (amask >> q & 1) && k0 + akk + (ta ? 0 : (T / BM) * q) < kend;
        cp_async8(as + q * asq, ok ? ap + q * astep : g.A, ok);
      }
#pragma unroll
    for (int q = 0; q < QB; ++q)
      if (q >= QB / parts * part && q < QB / parts * (part + 1)) {
        const bool ok = (bmask >> q & 1) && k0 + bkk + (tb ? (T / BN) * q : 0) < kend;
        cp_async8(bs + q * bsq, ok ? bp + q * bstep : g.B, ok);
      }
  };

  const int lane = tid & 31, warp = tid >> 5;
  const int wm = (warp % (BM / 32)) * 32, wn = (warp / (BM / 32)) * 32;
  const int gq = lane >> 2, tq = lane & 3;
  double acc[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;

#pragma unroll
  for (int st = 0; st < ST - 1; ++st) {
    if (st < nk) {
      issue(st, kbeg + st * kGBK, 0, 1);
      ap += aadv;
      bp += badv;
    }
    cp_async_commit();
  }
  for (int t = 0; t < nk; ++t) {
    cp_async_wait<ST - 2>();
    __syncthreads();
    const int nt = t + ST - 1;
    const double* as = As + (t % ST) * kGBK * SA + tq * SA + wm + gq;
    const double* bs = Bs + (t % ST) * kGBK * SB + tq * SB + wn + gq;
#pragma unroll
    for (int k4 = 0; k4 < KS; ++k4) {
      double af[4], bf[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) af[a] = as[k4 * 4 * SA + a * 8];
#pragma unroll
      for (int b = 0; b < 4; ++b) bf[b] = bs[k4 * 4 * SB + b * 8];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
          asm volatile(
              "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
              : "+d"(acc[a][b][0]), "+d"(acc[a][b][1])
              : "d"(af[a]), "d"(bf[b]));
      if (nt < nk) issue(nt % ST, kbeg + nt * kGBK, k4, KS);
    }
    cp_async_commit();
    ap += aadv;
    bp += badv;
  }
  cp_async_wait<0>();
  // with beta != 0 a column group's C entries are loaded before its first store, so
  // that the loads are in flight together
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    double cv[4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int gm = m0 + wm + a * 8 + gq, gn = n0 + wn + b * 8 + tq * 2 + c;
        cv[a][c] =
            (g.beta != 0.0 && gm < g.m && gn < g.n) ? g.C[gm + (long long)gn * g.ldc] : 0.0;
      }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int gm = m0 + wm + a * 8 + gq, gn = n0 + wn + b * 8 + tq * 2 + c;
        if (gm >= g.m || gn >= g.n) continue;
        const double v = g.alpha * acc[a][b][c];
        g.C[gm + (long long)gn * g.ldc] = (g.beta == 0.0) ? v : fma(g.beta, cv[a][c], v);
      }
  }
}

void launch_dgemm(const GemmDesc* d_desc, const int* d_tile_off, int nd, int total_tiles,
                  cudaStream_t s, int tile) {
  if (total_tiles <= 0) return;
  if (tile == 128) {
    constexpr int smem = dgemm_smem<128, 128, 4>();
    ensure_smem((const void*)k_dgemm<128, 128, 4, 1>, smem);
    k_dgemm<128, 128, 4, 1><<<total_tiles, 512, smem, s>>>(d_desc, d_tile_off, nd);
  } else {
    constexpr int smem = dgemm_smem<64, 64, 3>();
    ensure_smem((const void*)k_dgemm<64, 64, 3, 4>, smem);
    k_dgemm<64, 64, 3, 4><<<total_tiles, 128, smem, s>>>(d_desc, d_tile_off, nd);
  }
}

__global__ void k_splitk_reduce(const SplitKDesc* __restrict__ descs) {
  const SplitKDesc d = descs[blockIdx.y];
  const long long mn = (long long)d.m * d.n;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < mn;
       e += (long long)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int q = 0; q < d.S; ++q) acc += d.P[e + q * mn];
    const int i = (int)(e % d.m), j = (int)(e / d.m);
    double* c = d.C + i + (long long)j * d.ldc;
    *c = (d.beta == 0.0) ? d.alpha * acc : fma(d.beta, *c, d.alpha * acc);
  }
}

void launch_splitk_reduce(const SplitKDesc* d_desc, int nd, cudaStream_t s) {
  if (nd <= 0) return;
  dim3 grid(64, nd);
  k_splitk_reduce<<<grid, 256, 0, s>>>(d_desc);
}

// TF32 rounding of an FP32 value (round to nearest, ties away), as a 32-bit container.
__device__ __forceinline__ unsigned tf32_of(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return r;
}

// ===========================================================================
// Split-TF32 GEMM on the 5th-generation tensor cores (tcgen05).
//
// 1. k_tc_convert splits every FP64 operand value into a TF32 pair
//    (hi = rn(x), lo = rn(x - hi)) and stores the pairs as tiles of 128 rows
//    x 32 values of k in the K-major canonical layout without swizzle that the
//    tensor cores read from shared memory: 8-row x 16-byte core matrices of
//    128 bytes, K-adjacent ones 128 bytes apart (LBO), 8-row groups 1024 bytes
//    apart (SBO); a tile is 16 KB of hi followed by 16 KB of lo.
// 2. k_gemm_tc computes one 128 x 128 tile of C per CTA with warp roles:
//    one thread of warp 0 brings the A and B tiles of each k step into a
//    3-stage ring with bulk asynchronous copies (cp.async.bulk, completion
//    counted in bytes on the stage's mbarrier); one thread of warp 1 issues,
//    per k-step of 8, the products lo*hi, hi*lo, hi*hi (M = N = 128, K = 8,
//    FP32 accumulation in tensor memory) and releases the stage with
//    tcgen05.commit; warps 4-7 read the accumulator (warp w: lanes
//    32 (w - 4) .. + 31) every 256 values of k and add it to an FP64
//    accumulator that also lives in tensor memory (two 32-bit columns per
//    value), so no FP32 sum runs over more than 256 terms and C is read and
//    written once (alpha acc + beta C). Two FP32 accumulators alternate, so
//    the products of the next chunk proceed while one is read; the CTA holds
//    all 512 tensor-memory columns (one CTA per SM by its shared memory).
// Every mbarrier wait is bounded (globaltimer, 2 s); a wait that runs out
// marks the CTA aborted (every role stops waiting), records kStatusTimeout and
// leaves the tile unwritten; the CTA still frees its tensor memory.
// ===========================================================================
constexpr int kTcM = 128, kTcN = 128, kTcK = 32, kTcStages = 3, kTcChunk = 256;
constexpr int kTcPart = kTcM * kTcK * 4;             // bytes of one operand part (hi or lo)
constexpr int kTcTile = 2 * kTcPart;                 // one converted operand tile (hi, lo)
constexpr int kTcStage = 2 * kTcTile;                // A tile, B tile
constexpr int kTcSmem = kTcStages * kTcStage + 256;  // + mbarriers, tensor memory address
constexpr unsigned long long kTcWaitNs = 2000000000ull;

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait for the completion of the mbarrier phase with the given parity;
// gives up at once when *abort is set, and sets it when the time runs out.
__device__ __forceinline__ bool mbar_wait(unsigned addr, unsigned parity,
                                          volatile int* abort = nullptr) {
  const unsigned long long t0 = global_ns();
  for (;;) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (abort && *abort) return false;
    if (global_ns() - t0 > kTcWaitNs) {
      if (abort) *abort = 1;
      return false;
    }
  }
}

// Shared-memory matrix descriptor: K-major, no swizzle, LBO 128 B, SBO 1024 B,
// descriptor version 1 (sm_100).
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr) {
  unsigned long long d = (unsigned long long)((addr >> 4) & 0x3FFF);
  d |= (unsigned long long)(128 >> 4) << 16;
  d |= (unsigned long long)(1024 >> 4) << 32;
  d |= 1ull << 46;
  return d;
}

// Instruction descriptor, kind::tf32: D F32 (bits 4-5 = 1), A and B TF32
// (bits 7-9, 10-12 = 2), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
constexpr unsigned kTcIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(kTcN >> 3) << 17) |
                              ((unsigned)(kTcM >> 4) << 24);

// Byte offset of element (row, k) of one 128 x 32 operand part.
__device__ __forceinline__ int tc_off(int row, int kc) {
  return (((row >> 3) * (kTcK / 4) + kc) << 7) + ((row & 7) << 4);
}

__global__ void __launch_bounds__(256) k_tc_convert(const TcOperand* __restrict__ ops,
                                                    const int* __restrict__ tile_off, int nops) {
  const int oi = find_desc(tile_off, nops, blockIdx.x);
  const TcOperand o = ops[oi];
  const int local = blockIdx.x - tile_off[oi];
  const int kt_n = (o.kdim + kTcK - 1) / kTcK;
  const int rt = local / kt_n, kt = local % kt_n;
  unsigned char* dst = o.out + (size_t)local * kTcTile;
  const int row = threadIdx.x & 127, half = threadIdx.x >> 7;
  const int gi = rt * kTcM + row;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int kc = half + 2 * i;
    uint4 h, l;
    unsigned* ph = &h.x;
    unsigned* pl = &l.x;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int gk = kt * kTcK + 4 * kc + e;
      const double x = (gi < o.rows && gk < o.kdim)
                           ? (o.trans ? o.X[gk + (long long)gi * o.ld] : o.X[gi + (long long)gk * o.ld])
                           : 0.0;
      const float f = (float)x;
      const unsigned fh = tf32_of(f);
      ph[e] = fh;
      pl[e] = tf32_of(f - __uint_as_float(fh));
    }
    const int off = tc_off(row, kc);
    *reinterpret_cast<uint4*>(dst + off) = h;
    *reinterpret_cast<uint4*>(dst + kTcPart + off) = l;
  }
}

void launch_tc_convert(const TcOperand* d_ops, const int* d_tile_off, int nops, int total_tiles,
                       cudaStream_t s) {
  if (total_tiles <= 0) return;
  k_tc_convert<<<total_tiles, 256, 0, s>>>(d_ops, d_tile_off, nops);
}

__global__ void __launch_bounds__(256, 1) k_gemm_tc(const TcGemm* __restrict__ descs,
                                                    const int* __restrict__ tile_off, int nd,
                                                    int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(tc_smem + kTcStages * kTcStage);
  unsigned long long* full = bars;                  // [kTcStages]
  unsigned long long* empty = bars + kTcStages;     // [kTcStages]
  unsigned long long* tfull = bars + 2 * kTcStages;  // [2]
  unsigned long long* tempty = tfull + 2;            // [2]
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(tempty + 2);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int di = find_desc(tile_off, nd, blockIdx.x);
  const TcGemm g = descs[di];
  const int local = blockIdx.x - tile_off[di];
  const int tiles_m = (g.m + kTcM - 1) / kTcM;
  const int mt = local % tiles_m, nt = local / tiles_m;
  if (g.lower && mt < nt) return;  // whole CTA, before any barrier or allocation
  const int m0 = mt * kTcM, n0 = nt * kTcN;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kt_n = (g.k + kTcK - 1) / kTcK;
  constexpr int spc = kTcChunk / kTcK;  // k steps per chunk
  const int nchunk = (kt_n + spc - 1) / spc;

  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(4 * kTcN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int q = 0; q < kTcStages; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[q])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[q])) : "memory");
    }
    for (int q = 0; q < 2; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&tfull[q])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(smem_u32(&tempty[q])) : "memory");
    }
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // producer: bulk copies of the converted A and B tiles
    const unsigned char* a_src = g.A + (size_t)mt * kt_n * kTcTile;
    const unsigned char* b_src = g.B + (size_t)nt * kt_n * kTcTile;
    for (int kt = 0; kt < kt_n; ++kt) {
      const int s = kt % kTcStages;
      if (kt >= kTcStages &&
          !mbar_wait(smem_u32(&empty[s]), (unsigned)((kt / kTcStages - 1) & 1), abort))
        break;
      const unsigned fb = smem_u32(&full[s]);
      const unsigned dst = smem_u32(tc_smem + s * kTcStage);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                   "r"(kTcStage)
                   : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
          "[%3];" ::"r"(dst),
          "l"(a_src + (size_t)kt * kTcTile), "r"(kTcTile), "r"(fb)
          : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
          "[%3];" ::"r"(dst + kTcTile),
          "l"(b_src + (size_t)kt * kTcTile), "r"(kTcTile), "r"(fb)
          : "memory");
    }
  } else if (warp == 1 && lane == 0) {
    // tensor-core issue
    for (int kt = 0; kt < kt_n; ++kt) {
      const int s = kt % kTcStages, c = kt / spc, buf = c & 1;
      if (kt % spc == 0 && c >= 2 &&
          !mbar_wait(smem_u32(&tempty[buf]), (unsigned)((c / 2 - 1) & 1), abort))
        break;
      if (!mbar_wait(smem_u32(&full[s]), (unsigned)((kt / kTcStages) & 1), abort)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned base = smem_u32(tc_smem + s * kTcStage);
      const unsigned dacc = tmem + (unsigned)(buf * kTcN);
#pragma unroll
      for (int j = 0; j < kTcK / 8; ++j) {
        const unsigned long long dah = tc_desc(base + 0 * kTcPart + 256 * j);
        const unsigned long long dal = tc_desc(base + 1 * kTcPart + 256 * j);
        const unsigned long long dbh = tc_desc(base + 2 * kTcPart + 256 * j);
        const unsigned long long dbl = tc_desc(base + 3 * kTcPart + 256 * j);
        const unsigned long long da[3] = {dal, dah, dah}, db[3] = {dbh, dbl, dbh};
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          const unsigned acc = (kt % spc > 0 || j > 0 || p > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred q;\n\t"
              "setp.ne.b32 q, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, q;\n\t}\n" ::"r"(dacc),
              "l"(da[p]), "l"(db[p]), "r"(kTcIdesc), "r"(acc)
              : "memory");
        }
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              smem_u32(&empty[s]))
          : "memory");
      if (kt % spc == spc - 1 || kt == kt_n - 1)
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(&tfull[buf]))
            : "memory");
    }
  } else if (warp >= 4) {
    // epilogue: every chunk's FP32 sums are added to an FP64 accumulator kept
    // in tensor memory (columns 2 kTcN + 2 j, + 1: low and high words of
    // column j's value); C is read and written once, after the last chunk
    const int q = warp - 4;
    const int gm = m0 + 32 * q + lane;
    const unsigned lanes = (unsigned)(32 * q) << 16;
    for (int c = 0; c < nchunk; ++c) {
      const int buf = c & 1;
      const bool last = c == nchunk - 1;
      if (!mbar_wait(smem_u32(&tfull[buf]), (unsigned)((c / 2) & 1), abort)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int cc = 0; cc < kTcN / 16; ++cc) {
        unsigned v[16], w[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
            "%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(tmem + lanes + (unsigned)(buf * kTcN + 16 * cc))
            : "memory");
        const unsigned a64 = tmem + lanes + (unsigned)(2 * kTcN + 32 * cc);
        if (c > 0) {
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
              "%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, "
              "[%32];"
              : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]),
                "=r"(w[6]), "=r"(w[7]), "=r"(w[8]), "=r"(w[9]), "=r"(w[10]), "=r"(w[11]),
                "=r"(w[12]), "=r"(w[13]), "=r"(w[14]), "=r"(w[15]), "=r"(w[16]), "=r"(w[17]),
                "=r"(w[18]), "=r"(w[19]), "=r"(w[20]), "=r"(w[21]), "=r"(w[22]), "=r"(w[23]),
                "=r"(w[24]), "=r"(w[25]), "=r"(w[26]), "=r"(w[27]), "=r"(w[28]), "=r"(w[29]),
                "=r"(w[30]), "=r"(w[31])
              : "r"(a64)
              : "memory");
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        double acc[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const double x = (double)__uint_as_float(v[e]);
          acc[e] = (c > 0) ? __hiloint2double((int)w[2 * e + 1], (int)w[2 * e]) + x : x;
        }
        if (!last) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            w[2 * e] = (unsigned)__double2loint(acc[e]);
            w[2 * e + 1] = (unsigned)__double2hiint(acc[e]);
          }
          asm volatile(
              "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
              "%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
              "%32};" ::"r"(a64),
              "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]),
              "r"(w[7]), "r"(w[8]), "r"(w[9]), "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]),
              "r"(w[14]), "r"(w[15]), "r"(w[16]), "r"(w[17]), "r"(w[18]), "r"(w[19]),
              "r"(w[20]), "r"(w[21]), "r"(w[22]), "r"(w[23]), "r"(w[24]), "r"(w[25]),
              "r"(w[26]), "r"(w[27]), "r"(w[28]), "r"(w[29]), "r"(w[30]), "r"(w[31])
              : "memory");
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        } else if (gm < g.m) {
          // the 16 C entries loaded before the first store (in flight together)
          double cv[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int gn = n0 + 16 * cc + e;
            cv[e] = (g.beta != 0.0 && gn < g.n) ? g.C[gm + (long long)gn * g.ldc] : 0.0;
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int gn = n0 + 16 * cc + e;
            if (gn < g.n) {
              const double val = g.alpha * acc[e];
              g.C[gm + (long long)gn * g.ldc] = (g.beta == 0.0) ? val : fma(g.beta, cv[e], val);
            }
          }
        }
      }
      // this chunk's accumulator has been read: release it to the next chunk but one
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[buf]))
                     : "memory");
    }
    if (kt_n == 0 && gm < g.m) {
      for (int e = 0; e < kTcN; ++e) {
        const int gn = n0 + e;
        if (gn < g.n) {
          double* cp = g.C + gm + (long long)gn * g.ldc;
          *cp = (g.beta == 0.0) ? 0.0 : g.beta * *cp;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && *abort) atomicOr(status, kStatusTimeout);
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(4 * kTcN)
                 : "memory");
  }
}

void launch_gemm_tc(const TcGemm* d_desc, const int* d_tile_off, int nd, int total_tiles,
                    int* d_status, cudaStream_t s) {
  if (total_tiles <= 0) return;
  ensure_smem((const void*)k_gemm_tc, kTcSmem);
  k_gemm_tc<<<total_tiles, 256, kTcSmem, s>>>(d_desc, d_tile_off, nd, d_status);
}

// ===========================================================================
// FP64 products on the int8 tensor cores (Ozaki scheme).
//
// C = op(A) op(B) is computed from exact integer pieces of the operands.
// Every operand row (row i of op(A), column j of op(B)) is scaled by a power
// of two into (-1, 1) and cut into S signed 7-bit slices by truncation
// (v <- 128 v; q = trunc(v); v <- v - q, exact in FP64):
//   x_ik = 2^{e_i} sum_{s<S} q_s(i, k) 2^{-7(s+1)} + r_ik,  |r_ik| < 2^{e_i - 7S}.
// Then
//   C_ij = 2^{e_i + f_j - 14} sum_{d<S} 2^{-7d} P_d(i, j),  P_d = sum_{s+t=d} Q_s R_t^T,
// the slice pairs with s + t >= S being dropped (they weigh less than the
// representation error). |P_d| <= (d + 1) k 127^2 < 2^31 for k <= kOzMaxK, so
// each diagonal sum is exact in int32 and accumulates over the whole k range
// in its own tensor-memory accumulator (tcgen05.mma kind::i8, M = 128,
// N = BN, K = 32); the epilogue reads each once, sums them in FP64 (Horner in
// 2^-7) and scales by 2^{e_i + f_j - 14}. Integer accumulation makes the
// result independent of the order of the products. The error is of order
// k 2^{-7S} max_k |a_ik| max_k |b_kj| (an FP64 product's scales with
// u sum_k |a_ik| |b_kj|).
// A converted tile holds S slices of 128 rows x 64 bytes, each in the K-major
// canonical layout without swizzle: 8-row x 16-byte core matrices of 128 B,
// K-adjacent ones 128 B apart (LBO), 8-row groups 512 B apart (SBO), so rows
// 64..127 of a slice are its second 4 KB and a 64-row B tile is a contiguous
// half of each slice.
// Roles as in k_gemm_tc: one thread of warp 0 streams the A and B tiles of
// every 64-k step into a ring of stages (cp.async.bulk, completion counted in
// bytes on the stage's mbarrier); one thread of warp 1 issues the
// S (S + 1) / 2 slice products of each 32-k half and releases the stage with
// tcgen05.commit; warps 4-7 wait for the last products and write C. Waits are
// bounded as in k_gemm_tc.
// ===========================================================================
// Tile (128 rows x 64 k) of an operand into shared memory, read along the
// operand's contiguous dimension: for trans = 0 lanes run over rows, for
// trans = 1 over k, so that both layouts are read in whole cache lines. Each
// thread issues its 32 loads before the first store, so that they are in
// flight together. T[i * kOzTs + k]; entries past the operand are zero.
constexpr int kOzTs = kOzK + 1;
constexpr size_t kOzConvSmem = (size_t)128 * kOzTs * sizeof(double);
static_assert(128 * kOzK == 256 * 32, "tile loader: 256 threads x 32 elements");
__device__ __forceinline__ void oz_load_tile(const OzOperand& o, int rt, int kt, double* T) {
  const int r0 = rt * 128, k0 = kt * kOzK;
  double v[32];
  if (o.trans == 0) {
    // thread: row i = tid & 127, k = (tid >> 7) + 2 j
    const int i = threadIdx.x & 127, kb = threadIdx.x >> 7;
    const int gi = r0 + i;
    const double* src = o.X + gi;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int gk = k0 + kb + 2 * j;
      v[j] = (gi < o.rows && gk < o.kdim) ? __ldg(src + (long long)gk * o.ld) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) T[i * kOzTs + kb + 2 * j] = v[j];
  } else {
    // thread: k = tid & 63, row i = (tid >> 6) + 4 j
    const int k = threadIdx.x & (kOzK - 1), ib = threadIdx.x >> 6;
    const int gk = k0 + k;
    const double* src = o.X + gk;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int gi = r0 + ib + 4 * j;
      v[j] = (gi < o.rows && gk < o.kdim) ? __ldg(src + (long long)gi * o.ld) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) T[(ib + 4 * j) * kOzTs + k] = v[j];
  }
}

// Tiles of a triangular operand that no product reads (all above the diagonal).
__device__ __forceinline__ bool oz_unread(const OzOperand& o, int rt, int kt) {
  return (o.tri == 1 && kt * kOzK > rt * 128 + 127) || (o.tri == 2 && kt * kOzK + 63 < rt * 128);
}

// Row exponents, read in place along the operand's contiguous dimension:
// trans = 0, two threads per row (lanes over consecutive rows), 32 k each;
// trans = 1, a warp per row (lanes over consecutive k), 16 rows per warp. The
// 32 loads of a thread are issued before the first maximum, which is taken over the
// high words (an exponent needs no more). Rows of subnormals take the exact way, and rows
// that hold a NaN, which is left out of the maximum and has no digits.
__device__ __forceinline__ int oz_exponent(int hi) {  // m < 2^e, m >= 2^(e - 1)
  return (hi >> 20) - 1022;
}
__global__ void __launch_bounds__(256) k_oz_exp(const OzOperand* __restrict__ ops,
                                                const int* __restrict__ tile_off, int nops) {
  const int oi = find_desc(tile_off, nops, blockIdx.x);
  const OzOperand o = ops[oi];
  const int local = blockIdx.x - tile_off[oi];
  const int kt_n = (o.kdim + kOzK - 1) / kOzK;
  const int rt = local / kt_n, kt = local % kt_n;
  if (oz_unread(o, rt, kt)) return;
  const int k0 = kt * kOzK;
  double v[32];
  if (o.trans == 0) {
    const int row = threadIdx.x & 127, half = threadIdx.x >> 7;
    const int gi = rt * 128 + row;
    if (gi >= o.rows) return;
    const double* src = o.X + gi;
#pragma unroll
    for (int e = 0; e < 32; ++e) {
      const int gk = k0 + 32 * half + e;
      v[e] = gk < o.kdim ? __ldg(src + (long long)gk * o.ld) : 0.0;
    }
    int h = 0;
#pragma unroll
    for (int e = 0; e < 32; ++e) h = max(h, __double2hiint(v[e]) & 0x7fffffff);
    if (h >= 0x00100000 && h < 0x7ff00000) {
      atomicMax(&o.rexp[gi], oz_exponent(h));
    } else {
      double m = 0.0;
#pragma unroll
      for (int e = 0; e < 32; ++e) m = fmax(m, fabs(v[e]));
      int ex;
      frexp(m, &ex);
      if (m > 0.0) atomicMax(&o.rexp[gi], ex);
    }
  } else {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gk0 = k0 + lane, gk1 = k0 + 32 + lane;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int gi = rt * 128 + warp + 8 * j;
      const double* src = o.X + (long long)gi * o.ld;
      v[2 * j] = (gi < o.rows && gk0 < o.kdim) ? __ldg(src + gk0) : 0.0;
      v[2 * j + 1] = (gi < o.rows && gk1 < o.kdim) ? __ldg(src + gk1) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int gi = rt * 128 + warp + 8 * j;
      const int h = __reduce_max_sync(
          0xffffffffu, max(__double2hiint(v[2 * j]) & 0x7fffffff,
                           __double2hiint(v[2 * j + 1]) & 0x7fffffff));
      if (gi >= o.rows) continue;
      if (h >= 0x00100000 && h < 0x7ff00000) {
        if (lane == 0) atomicMax(&o.rexp[gi], oz_exponent(h));
      } else {
        double m = fmax(fabs(v[2 * j]), fabs(v[2 * j + 1]));
        int ex;
        frexp(m, &ex);
        if (m > 0.0) atomicMax(&o.rexp[gi], ex);
      }
    }
  }
}

// The seven-bit digits of 28 bits, the lowest in byte 0; negated bytewise if neg.
__device__ __forceinline__ unsigned oz_digits(unsigned x, bool neg) {
  const unsigned d = (x & 0x7fu) | ((x << 1) & 0x7f00u) | ((x << 2) & 0x7f0000u) |
                     ((x << 3) & 0x7f000000u);
  return neg ? (0x80808080u - d) ^ 0x80808080u : d;  // digits below 128: no borrow
}

// |x| 2^{7S - e} truncated to an integer of 7S bits, cut into S digits with x's sign:
// what truncating v <- 128 v digit by digit gives, from the bits of x. Done in FP64 the
// S roundings and conversions per entry (a quarter of the FP64 rate or less) set the
// pace: 2.7 TB/s. n = 128 mixed: 25.1 ms of slicing then, 17.7 ms now, the triangular
// operands' unread tiles left out.
template <int S>
__global__ void __launch_bounds__(256) k_oz_slice(const OzOperand* __restrict__ ops,
                                                  const int* __restrict__ tile_off, int nops) {
  extern __shared__ double oz_t[];
  const int oi = find_desc(tile_off, nops, blockIdx.x);
  const OzOperand o = ops[oi];
  const int local = blockIdx.x - tile_off[oi];
  const int kt_n = (o.kdim + kOzK - 1) / kOzK;
  const int rt = local / kt_n, kt = local % kt_n;
  if (oz_unread(o, rt, kt)) return;
  oz_load_tile(o, rt, kt, oz_t);
  __syncthreads();
  const int row = threadIdx.x & 127, half = threadIdx.x >> 7;
  const int gi = rt * 128 + row;
  // rows without a nonzero keep the cleared exponent; their slices are zero
  const int ex = gi < o.rows ? max(o.rexp[gi], -4096) : 0;
  signed char* dst = o.out + (size_t)local * S * kOzPart;
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    const int kc = 2 * half + c;  // 16-byte chunk of the row's 64 bytes
    unsigned w[8][4];             // slice S - 1 - s of the chunk's entries, four a word
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      unsigned lo[4], hi[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const double x = oz_t[row * kOzTs + 16 * kc + 4 * q + b];
        const int xh = __double2hiint(x), e = (xh >> 20) & 0x7ff;
        const unsigned mh = (unsigned)(xh & 0xfffff) | (e ? 0x100000u : 0u);
        const unsigned long long m =
            e == 0x7ff ? 0ull : ((unsigned long long)mh << 32) | (unsigned)__double2loint(x);
        const int t = max(e, 1) - 1075 + 7 * S - ex;  // at most 7 S - 53 <= 3
        const unsigned long long f = t >= 0 ? m << t : (t > -64 ? m >> -t : 0ull);
        lo[b] = oz_digits((unsigned)f & 0xfffffffu, xh < 0);
        hi[b] = S > 4 ? oz_digits((unsigned)(f >> 28) & 0xfffffffu, xh < 0) : 0u;
      }
      // 4 x 4 byte transpose: entries within a word, slices across words
      auto words = [&](const unsigned (&v)[4], int s0) {
        const unsigned t0 = __byte_perm(v[0], v[1], 0x5140), t1 = __byte_perm(v[2], v[3], 0x5140);
        const unsigned t2 = __byte_perm(v[0], v[1], 0x7362), t3 = __byte_perm(v[2], v[3], 0x7362);
        w[s0][q] = __byte_perm(t0, t1, 0x5410);
        w[s0 + 1][q] = __byte_perm(t0, t1, 0x7632);
        w[s0 + 2][q] = __byte_perm(t2, t3, 0x5410);
        w[s0 + 3][q] = __byte_perm(t2, t3, 0x7632);
      };
      words(lo, 0);
      if (S > 4) words(hi, 4);
    }
    const int off = ((row >> 3) * 4 + kc) * 128 + (row & 7) * 16;
#pragma unroll
    for (int s = 0; s < S; ++s)
      *reinterpret_cast<uint4*>(dst + (size_t)(S - 1 - s) * kOzPart + off) =
          make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
  }
}

template <int S>
static void launch_oz_slice(const OzOperand* d_ops, const int* d_tile_off, int nops,
                            int total_tiles, cudaStream_t s) {
  ensure_smem((const void*)k_oz_slice<S>, kOzConvSmem);
  k_oz_slice<S><<<total_tiles, 256, kOzConvSmem, s>>>(d_ops, d_tile_off, nops);
}

void launch_oz_convert(const OzOperand* d_ops, const int* d_tile_off, int nops, int total_tiles,
                       int slices, int* d_rexp, long long n_rexp, cudaStream_t s) {
  if (total_tiles <= 0) return;
  // 0x80808080: below every exponent a double can have
  cudaMemsetAsync(d_rexp, 0x80, (size_t)n_rexp * sizeof(int), s);
  k_oz_exp<<<total_tiles, 256, 0, s>>>(d_ops, d_tile_off, nops);
  switch (slices) {
    case 2: launch_oz_slice<2>(d_ops, d_tile_off, nops, total_tiles, s); break;
    case 3: launch_oz_slice<3>(d_ops, d_tile_off, nops, total_tiles, s); break;
    case 4: launch_oz_slice<4>(d_ops, d_tile_off, nops, total_tiles, s); break;
    case 5: launch_oz_slice<5>(d_ops, d_tile_off, nops, total_tiles, s); break;
    case 6: launch_oz_slice<6>(d_ops, d_tile_off, nops, total_tiles, s); break;
    case 7: launch_oz_slice<7>(d_ops, d_tile_off, nops, total_tiles, s); break;
    case 8: launch_oz_slice<8>(d_ops, d_tile_off, nops, total_tiles, s); break;
    default: break;
  }
}

// Shared-memory matrix descriptor: K-major, no swizzle, LBO 128 B, SBO 512 B.
__device__ __forceinline__ unsigned long long oz_desc(unsigned addr) {
  unsigned long long d = (unsigned long long)((addr >> 4) & 0x3FFF);
  d |= (unsigned long long)(128 >> 4) << 16;
  d |= (unsigned long long)(512 >> 4) << 32;
  d |= 1ull << 46;
  return d;
}

template <int S, int BN>
struct OzCfg {
  static constexpr int kA = S * kOzPart;   // A bytes of one stage
  static constexpr int kB = S * BN * kOzK;  // B bytes of one stage
  static constexpr int kStage = kA + kB;
  static constexpr int kStages = (200 * 1024) / kStage > 4 ? 4 : (200 * 1024) / kStage;
  static constexpr int kSmem = kStages * kStage + 256;
  static constexpr int kCols = S * BN <= 256 ? 256 : 512;  // tensor-memory columns
  // Instruction descriptor, kind::i8: D S32 (bits 4-5 = 2), A and B signed
  // 8-bit (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at 24.
  static constexpr unsigned kIdesc = (2u << 4) | (1u << 7) | (1u << 10) |
                                     ((unsigned)(BN >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
  static_assert(S * BN <= 512, "diagonal accumulators exceed tensor memory");
  static_assert(kStages >= 2, "stage ring");
};

__device__ __forceinline__ void bulk_g2s(unsigned dst, const void* src, int bytes, unsigned bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// One int8 slice product; U selects the A collector buffer's use: 0 read A
// from shared memory only, 1 read it and keep it (fill), 2 reuse the kept A,
// 3 reuse it for the last time.
template <int U>
__device__ __forceinline__ void oz_mma(unsigned d, unsigned long long da, unsigned long long db,
                                       unsigned idesc, unsigned acc) {
  if (U == 0)
    asm volatile(
        "{\n\t.reg .pred r;\n\tsetp.ne.b32 r, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, r;\n\t}\n" ::"r"(d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
  else if (U == 1)
    asm volatile(
        "{\n\t.reg .pred r;\n\tsetp.ne.b32 r, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8.collector::a::fill [%0], %1, %2, %3, r;\n\t}\n" ::"r"(
            d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
  else if (U == 2)
    asm volatile(
        "{\n\t.reg .pred r;\n\tsetp.ne.b32 r, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8.collector::a::use [%0], %1, %2, %3, r;\n\t}\n" ::"r"(d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred r;\n\tsetp.ne.b32 r, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8.collector::a::lastuse [%0], %1, %2, %3, r;\n\t}\n" ::"r"(
            d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}

// Persistent: one CTA per SM walks the launch's tiles t = blockIdx.x,
// blockIdx.x + gridDim.x, ...; the tensor memory is allocated and the barriers
// set up once. The stage ring runs on across tiles. The accumulators of a tile
// are released (tempty) as soon as the epilogue warps have read them, so its
// C writes overlap the next tile's products.
template <int S, int BN>
__global__ void __launch_bounds__(256, 1) k_gemm_oz(const OzGemm* __restrict__ descs,
                                                    const int* __restrict__ tile_off, int nd,
                                                    int total_tiles, int* __restrict__ status) {
  using Cfg = OzCfg<S, BN>;
  constexpr int NS = Cfg::kStages;
  extern __shared__ __align__(1024) unsigned char oz_smem[];
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(oz_smem + NS * Cfg::kStage);
  unsigned long long* full = bars;        // [NS]
  unsigned long long* empty = bars + NS;  // [NS]
  unsigned long long* tfull = bars + 2 * NS;
  unsigned long long* tempty = tfull + 1;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(tempty + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // tile decode shared by the roles
  // k tiles [kf, kt_cnt) of the launch's range run: with a lower-triangular A
  // none past the tile's last row, with a lower-triangular B none before its
  // first column
  auto tile = [&](int t, OzGemm& g, int& mt, int& nt, int& kf, int& kt_cnt) -> bool {
    const int di = find_desc(tile_off, nd, t);
    g = descs[di];
    const int local = t - tile_off[di];
    const int tiles_m = (g.m + 127) / 128;
    mt = local % tiles_m;
    nt = local / tiles_m;
    const int m0 = mt * 128, n0 = nt * BN;
    if (g.lower && n0 >= m0 + 128) return false;
    kt_cnt = g.a_lower ? min(g.kt_cnt, max(0, (m0 + 128 + kOzK - 1) / kOzK - g.kt0)) : g.kt_cnt;
    kf = g.b_lower ? min(kt_cnt, max(0, n0 / kOzK - g.kt0)) : 0;
    return true;
  };

  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(Cfg::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int q = 0; q < NS; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[q])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[q])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(tfull)) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(smem_u32(tempty)) : "memory");
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // producer: per k tile, the S slices of the A tile, then those of the B tile
    int it = 0;
    for (int t = blockIdx.x; t < total_tiles && !*abort; t += gridDim.x) {
      OzGemm g;
      int mt, nt, kf, kt_cnt;
      if (!tile(t, g, mt, nt, kf, kt_cnt)) continue;
      const int n0 = nt * BN, bt = n0 / 128, bhalf = (n0 / 64) & 1;
      bool ok = true;
      for (int i = kf; i < kt_cnt; ++i, ++it) {
        const int kt = g.kt0 + i, s = it % NS;
        if (it >= NS && !mbar_wait(smem_u32(&empty[s]), (unsigned)((it / NS - 1) & 1), abort)) {
          ok = false;
          break;
        }
        const unsigned fb = smem_u32(&full[s]);
        const unsigned dst = smem_u32(oz_smem + s * Cfg::kStage);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                     "r"(Cfg::kStage)
                     : "memory");
        bulk_g2s(dst, g.A + ((size_t)mt * g.kt_total + kt) * S * kOzPart, Cfg::kA, fb);
        const signed char* b = g.B + ((size_t)bt * g.kt_total + kt) * S * kOzPart;
        if (BN == 128) {
          bulk_g2s(dst + Cfg::kA, b, Cfg::kB, fb);
        } else {
#pragma unroll
          for (int q = 0; q < S; ++q)
            bulk_g2s(dst + Cfg::kA + q * BN * kOzK, b + (size_t)q * kOzPart + bhalf * BN * kOzK,
                     BN * kOzK, fb);
        }
      }
      if (!ok) break;
    }
  } else if (warp == 1 && lane == 0) {
    // tensor-core issue: slice pair (p, q) adds into the accumulator of diagonal p + q
    int it = 0, a = 0;
    for (int t = blockIdx.x; t < total_tiles && !*abort; t += gridDim.x) {
      OzGemm g;
      int mt, nt, kf, kt_cnt;
      if (!tile(t, g, mt, nt, kf, kt_cnt) || kt_cnt <= kf) continue;
      // the previous tile's accumulators have been read
      if (a > 0 && !mbar_wait(smem_u32(tempty), (unsigned)((a - 1) & 1), abort)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      bool ok = true;
      for (int i = kf; i < kt_cnt; ++i, ++it) {
        const int s = it % NS;
        if (!mbar_wait(smem_u32(&full[s]), (unsigned)((it / NS) & 1), abort)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned base = smem_u32(oz_smem + s * Cfg::kStage);
#pragma unroll
        for (int j = 0; j < kOzK / 32; ++j) {
#pragma unroll
          for (int p = 0; p < S; ++p) {
            const unsigned long long da = oz_desc(base + p * kOzPart + 256 * j);
#pragma unroll
            for (int q = 0; p + q < S; ++q) {
              const unsigned long long db = oz_desc(base + Cfg::kA + q * BN * kOzK + 256 * j);
              const unsigned acc = (i > kf || j > 0 || p > 0) ? 1u : 0u;
              const unsigned d = tmem + (unsigned)((p + q) * BN);
              // A slice p is read from shared memory once per 32-k step and kept
              // in the collector buffer for its other slice pairs
              if (p == S - 1)
                oz_mma<0>(d, da, db, Cfg::kIdesc, acc);
              else if (q == 0)
                oz_mma<1>(d, da, db, Cfg::kIdesc, acc);
              else if (p + q < S - 1)
                oz_mma<2>(d, da, db, Cfg::kIdesc, acc);
              else
                oz_mma<3>(d, da, db, Cfg::kIdesc, acc);
            }
          }
        }
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(&empty[s]))
            : "memory");
      }
      if (!ok) break;
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              smem_u32(tfull))
          : "memory");
      ++a;
    }
  } else if (warp >= 4) {
    // epilogue: C = alpha 2^{e_i + f_j - 14} sum_d 2^{-7d} P_d + beta C, the
    // diagonals combined 64 columns at a time in registers
    const int q4 = warp - 4;
    const unsigned lanes = (unsigned)(32 * q4) << 16;
    int a = 0;
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
      OzGemm g;
      int mt, nt, kf, kt_cnt;
      if (!tile(t, g, mt, nt, kf, kt_cnt)) continue;
      kt_cnt -= kf;  // k tiles run
      const int gm = mt * 128 + 32 * q4 + lane, n0 = nt * BN;
      bool ok = true;
      if (kt_cnt > 0) {
        ok = mbar_wait(smem_u32(tfull), (unsigned)(a & 1), abort) && !*abort;
        if (ok) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      if (!ok) break;
      const int ea = gm < g.m ? max(g.ea[gm], -4096) : 0;
#pragma unroll
      for (int half = 0; half < BN / 64; ++half) {
        double h[64];
#pragma unroll
        for (int e = 0; e < 64; ++e) h[e] = 0.0;
        if (kt_cnt > 0) {
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
#pragma unroll
            for (int d = S - 1; d >= 0; --d) {
              unsigned v[16];
              asm volatile(
                  "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,"
                  "%11,%12,%13,%14,%15}, [%16];"
                  : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                    "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
                    "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                  : "r"(tmem + lanes + (unsigned)(d * BN + 64 * half + 16 * cc))
                  : "memory");
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int e = 0; e < 16; ++e)
                h[16 * cc + e] = fma(h[16 * cc + e], 0.0078125, (double)(int)v[e]);
            }
          }
          if (half == BN / 64 - 1) {
            // every accumulator of the tile is read: release them to the next tile
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(tempty))
                           : "memory");
          }
        }
        if (gm < g.m) {
          // 16 columns at a time: their C entries and column exponents are
          // loaded before any store, so the loads are in flight together (a
          // load after a store to C would wait for it: the compiler cannot rule
          // out aliasing)
          double* crow = g.C + gm;
#pragma unroll
          for (int e0 = 0; e0 < 64; e0 += 16) {
            double cv[16];
            int fe[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const int gn = n0 + 64 * half + e0 + e;
              const bool in = gn < g.n;
              fe[e] = in ? g.eb[gn] : 0;
              cv[e] = (in && g.beta != 0.0) ? crow[(long long)gn * g.ldc] : 0.0;
            }
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const int gn = n0 + 64 * half + e0 + e;
              if (gn < g.n) {
                const double val = g.alpha * ldexp(h[e0 + e], ea + max(fe[e], -4096) - 14);
                crow[(long long)gn * g.ldc] = (g.beta == 0.0) ? val : fma(g.beta, cv[e], val);
              }
            }
          }
        }
      }
      if (kt_cnt > 0) ++a;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && *abort) atomicOr(status, kStatusTimeout);
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(Cfg::kCols)
                 : "memory");
  }
}

int oz_tile_n(int slices) { return slices <= 4 ? 128 : 64; }

template <int S, int BN>
static void launch_gemm_oz_t(const OzGemm* d_desc, const int* d_tile_off, int nd, int total_tiles,
                             int* d_status, cudaStream_t s) {
  ensure_smem((const void*)k_gemm_oz<S, BN>, OzCfg<S, BN>::kSmem);
  const int grid = std::min(total_tiles, sm_count());
  k_gemm_oz<S, BN><<<grid, 256, OzCfg<S, BN>::kSmem, s>>>(d_desc, d_tile_off, nd, total_tiles,
                                                           d_status);
}

void launch_gemm_oz(const OzGemm* d_desc, const int* d_tile_off, int nd, int total_tiles,
                    int slices, int* d_status, cudaStream_t s) {
  if (total_tiles <= 0) return;
  switch (slices) {
    case 2: launch_gemm_oz_t<2, 128>(d_desc, d_tile_off, nd, total_tiles, d_status, s); break;
    case 3: launch_gemm_oz_t<3, 128>(d_desc, d_tile_off, nd, total_tiles, d_status, s); break;
    case 4: launch_gemm_oz_t<4, 128>(d_desc, d_tile_off, nd, total_tiles, d_status, s); break;
    case 5: launch_gemm_oz_t<5, 64>(d_desc, d_tile_off, nd, total_tiles, d_status, s); break;
    case 6: launch_gemm_oz_t<6, 64>(d_desc, d_tile_off, nd, total_tiles, d_status, s); break;
    case 7: launch_gemm_oz_t<7, 64>(d_desc, d_tile_off, nd, total_tiles, d_status, s); break;
    case 8: launch_gemm_oz_t<8, 64>(d_desc, d_tile_off, nd, total_tiles, d_status, s); break;
    default: break;
  }
}

// ===========================================================================
// Cholesky elimination (symmetric positive definite interiors; the lower
// triangle of every block is the one read and written).
//   [A22 A12^T; A12 A11] = [L 0; Y^T I] [I 0; 0 S] [L^T Y; 0 I],
//   A22 = L L^T, Y = L^{-1} A12^T, S = A11 - Y^T Y.
// The factor keeps L (for F u), L^{-1} and Y (for F^{-1} u): in exact
// arithmetic X = L^{-T} Y and A22^{-1} = L^{-T} L^{-1}, the reference's
// Schur() outputs (include/Schur.hpp:72-100).
// ===========================================================================

// ===========================================================================
// Gauss-Jordan sweep. For B = [A22 A21; A12 A11] (red first), eliminating
// pivots 0..r-1 in place gives [A22^{-1} X; * A11 - A12 X] with
// X = A22^{-1} A21: the three outputs of the reference's Schur().
// Entries of the bottom-left block whose column is already pivoted are never
// read again and are not updated.
// ===========================================================================
//
// Small blocks (n <= kSmallSweepN), a CTA each, by Gauss-Jordan or (CHOL) Cholesky: the
// block lives in registers, thread (tx, ty) of a 16 x 16 grid holding rows tx + 16a and
// columns ty + 16b, and a pivot is one barrier: the owners of row and column k publish
// them (two buffers, alternating) and every thread updates its TS x TS entries.
//   Gauss-Jordan, p = a_kk: row k * (1 / p); column k * (-1 / p); the rest a - a_ik r_j.
//   Cholesky, t = 1 / sqrt(a_kk), l = t a_ik (i > k): column k of [L; Y^T] is l, kept in
//   shared memory; row k * t (left of k: L^{-1}; its diagonal t); rows below: a - l_i r_j,
//   with -l_i t in column k.
// Bound by the barrier and the publish of a pivot. In shared memory, with four barriers
// and an integer division per entry, level 0's 27-of-81 blocks of n = 128 took 7.8 ms
// (Cholesky 6.5 ms), 2.8 ms (3.3 ms) here; reading and writing them takes 0.5 ms.
template <int TS, bool CHOL>
__global__ void __launch_bounds__(256, TS == 6 ? 2 : 1) k_elim_small(const SweepDesc* __restrict__ descs,
                                                    int* __restrict__ status) {
  const SweepDesc d = descs[blockIdx.x];
  const int n = d.n, r = d.r, s = n - r;
  extern __shared__ double S[];  // n x n, ld n: staging
  __shared__ double rowk[2][16 * TS], colk[2][16 * TS];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31, warp = tid >> 5;
  const int nn = n * n;
#pragma unroll 8
  for (int e = tid; e < nn; e += 256) S[e] = d.B[e];
  __syncthreads();
  double a[TS][TS];
#pragma unroll
  for (int u = 0; u < TS; ++u)
#pragma unroll
    for (int v = 0; v < TS; ++v) {
      const int i = tx + 16 * u, j = ty + 16 * v;
      // Cholesky: the lower triangle, mirrored
      a[u][v] = (i < n && j < n) ? ((CHOL && i < j) ? S[j + i * n] : S[i + j * n]) : 0.0;
    }
  int bad = 0;
#pragma unroll
  for (int kb = 0; kb < TS; ++kb) {
    for (int kk = 0; kk < 16; ++kk) {
      const int k = kb * 16 + kk, buf = k & 1;
      if (k >= r) break;
      if (tx == kk) {
#pragma unroll
        for (int v = 0; v < TS; ++v) rowk[buf][ty + 16 * v] = a[kb][v];
      }
      if (ty == kk) {
#pragma unroll
        for (int u = 0; u < TS; ++u) colk[buf][tx + 16 * u] = a[u][kb];
      }
      __syncthreads();
      const double p = rowk[buf][k];
      double t;
      if (CHOL) {
        if (!(p > 1e-300) || !isfinite(p)) bad = 1;
        t = rsqrt(fabs(p) > 1e-300 ? fabs(p) : 1.0);
      } else {
        if (!(fabs(p) > 1e-300) || !isfinite(p)) bad = 1;
        t = 1.0 / p;
      }
      double rj[TS], ci[TS];
#pragma unroll
      for (int v = 0; v < TS; ++v)
        rj[v] = (ty + 16 * v == k) ? t : rowk[buf][ty + 16 * v] * t;
#pragma unroll
      for (int u = 0; u < TS; ++u) {
        const int i = tx + 16 * u;
        ci[u] = colk[buf][i];
        if (CHOL) ci[u] = i > k ? ci[u] * t : 0.0;
      }
      // column k restarts from zero (Cholesky: below the diagonal)
      if (ty == kk) {
#pragma unroll
        for (int u = 0; u < TS; ++u)
          if (!CHOL || tx + 16 * u > k) a[u][kb] = 0.0;
      }
#pragma unroll
      for (int u = 0; u < TS; ++u)
#pragma unroll
        for (int v = 0; v < TS; ++v) a[u][v] = fma(-ci[u], rj[v], a[u][v]);
      if (tx == kk) {
#pragma unroll
        for (int v = 0; v < TS; ++v) a[kb][v] = rj[v];
      }
      if (CHOL && ty == kk) {
        // column k of [L; Y^T], zero above the diagonal
        const double q = fabs(p) > 1e-300 ? fabs(p) : 1.0;
#pragma unroll
        for (int u = 0; u < TS; ++u) {
          const int i = tx + 16 * u;
          if (i < n) S[i + k * n] = i == k ? q * t : ci[u];
        }
      }
    }
  }
  if (bad && tid == 0) atomicOr(status, kStatusTinyPivot);
  __syncthreads();
  // compact outputs: A22^{-1} or L^{-1} (r x r), X or Y (r x s), L; A11 - A12 X stays
  // in B
#pragma unroll
  for (int u = 0; u < TS; ++u)
#pragma unroll
    for (int v = 0; v < TS; ++v) {
      const int i = tx + 16 * u, j = ty + 16 * v;
      if (i >= n || j >= n) continue;
      if (i < r && j < r) d.a22inv[i + (long long)j * r] = (CHOL && i < j) ? 0.0 : a[u][v];
      else if (!CHOL && i < r) d.X[i + (long long)(j - r) * r] = a[u][v];
      else if (i >= r && j >= r) d.B[i + (long long)j * n] = a[u][v];
    }
  if (CHOL) {
    for (int j = warp; j < r; j += 8)
      for (int i = lane; i < r; i += 32) d.L[i + (long long)j * r] = S[i + j * n];
    for (int j = warp; j < s; j += 8)
      for (int i = lane; i < r; i += 32) d.X[i + (long long)j * r] = S[(r + j) + i * n];
  }
}

template <bool CHOL>
void launch_elim_small(const SweepDesc* d_desc, int nd, int max_n, int* d_status,
                       cudaStream_t s) {
  if (nd <= 0) return;
  const size_t smem = (size_t)max_n * max_n * sizeof(double);
  if (max_n <= 96) {
    ensure_smem((const void*)k_elim_small<6, CHOL>, 96 * 96 * sizeof(double));
    k_elim_small<6, CHOL><<<nd, 256, smem, s>>>(d_desc, d_status);
  } else {
    ensure_smem((const void*)k_elim_small<10, CHOL>,
                kSmallSweepN * kSmallSweepN * sizeof(double));
    k_elim_small<10, CHOL><<<nd, 256, smem, s>>>(d_desc, d_status);
  }
}
void launch_sweep_small(const SweepDesc* d_desc, int nd, int max_n, int* d_status,
                        cudaStream_t s) {
  launch_elim_small<false>(d_desc, nd, max_n, d_status, s);
}
void launch_chol_small(const SweepDesc* d_desc, int nd, int max_n, int* d_status,
                       cudaStream_t s) {
  launch_elim_small<true>(d_desc, nd, max_n, d_status, s);
}

// --- blocked sweep ---------------------------------------------------------
// Step for pivot block K = [k0, k1) of A22: Dinv = B[K, K]^{-1}, also over B[K, K]
// (k_pivot_block); the row / column panels and the rank-128 update are batched GEMMs
// issued by the host.
// The pivot block of both eliminations, 128 x 128, by 16-wide block steps: one CTA
// per block, and on the critical path of the top levels, where one or a few blocks
// remain, so it is built for latency. 16 worker warps hold the block as DMMA
// accumulators (32 x 32 a warp); step K reads the panels of block K from the owners
// through shared memory and updates everything by one rank-16 product:
//   Gauss-Jordan: with D = LU = block KK, G = L^{-1} (row panel) and H = (column panel)
//     U^{-1}: rows K := U^{-1} G, columns K := -H L^{-1}, the rest A - H G: with the K
//     rows and columns of the accumulators zeroed, G[:, K] = L^{-1} and H[K, :] = -U^{-1}
//     it is A - H G throughout;
//   Cholesky: l = chol(D); L_iK = A_iK l^{-T} below, the finished part of
//     L^{-1} left of K gets X_K = l^{-1} X_K; R = [X_K | l^{-1} | L_jK^T], rows K := R and
//     rows below K := A - L_iK R. The lower triangle only; L goes straight to its place.
// The panels are substituted, a column or row a thread, not multiplied by inverses of D
// or of its factors: that keeps the errors of single pivots (a few u times the scaled
// condition number), where products with D^{-1} were 20 to 100 times that for the wide
// faces of a field of contrast 10^6, and costs fewer multiply-adds.
// The serial part is four more warps', which hold no accumulators: the factors of D one
// warp's, the substitutions all four's. The owner of the next diagonal block updates
// that block first and hands it over, so its factors run beside the rest of the update.
// Of a step's 9.7 k cycles the factors take 7.8 k (16 dependent reciprocals, beside the
// update's 4.1 k cycles of DMMA; 5 k alone), the substitutions 1.7 k. A block takes 61 us
// (Cholesky 48 us); one pivot and one barrier at a time over registers took 200 us, the
// Cholesky factor 32-wide by one warp 150 us, explicit inverses in the 16-wide steps 62 us.
constexpr int kPbW = 16;                  // block step
constexpr int kPbLd = kSweepNB + 4;       // panel rows: 4 mod 16 doubles, conflict-free fragments
constexpr int kPbSt = kSweepNB + 1;       // staging
constexpr int kPbD = kPbW + 1;
constexpr int kPbThreads = 20 * 32;
constexpr int kPbSmem =
    (kSweepNB * kPbSt + 4 * kPbW * kPbLd + 2 * kPbW * kPbW + 3 * kPbW * kPbD) * (int)sizeof(double);

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// The factors of a 16 x 16 pivot D by one warp: lane = (row i, half h), columns
// 8h .. 8h + 7 in registers. D = LU: F0[k][i] = L_ik below a diagonal of ones,
// F1[k][i] = U_ki right of a diagonal of reciprocal pivots. CHOL, D = l l^T: F0[k][i] =
// l_ik below a diagonal of reciprocals, l itself to Ls[k][i].
template <bool CHOL>
__device__ __forceinline__ void pivot16(const double* Dn, double* F0, double* F1, double* Ls,
                                        int live, int& bad) {
  const int lane = threadIdx.x & 31, i = lane & 15, h = lane >> 4;
  double a[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) a[c] = Dn[i * kPbD + 8 * h + c];
#pragma unroll
  for (int k = 0; k < kPbW; ++k) {
    const int kh = k >> 3, kc = k & 7;
    const double p = __shfl_sync(0xffffffffu, a[kc], k + 16 * kh);
    const double cik = __shfl_sync(0xffffffffu, a[kc], i + 16 * kh);
    double rj[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) rj[c] = __shfl_sync(0xffffffffu, a[c], k + 16 * h);
    double li;
    if (CHOL) {
      if (k < live && (!(p > 1e-300) || !isfinite(p))) bad = 1;
      const double q = fabs(p) > 1e-300 ? fabs(p) : 1.0, rk = rsqrt(q);
      li = cik * rk;
      if (h == 0) {
        Ls[k * kPbD + i] = i > k ? li : (i == k ? q * rk : 0.0);
        F0[k * kPbW + i] = i == k ? rk : li;
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) rj[c] *= rk;
    } else {
      if (k < live && (!(fabs(p) > 1e-300) || !isfinite(p))) bad = 1;
      const double ip = 1.0 / p;
      li = cik * ip;
      if (h == 0) F0[k * kPbW + i] = i == k ? 1.0 : li;
      if (i == k) {
#pragma unroll
        for (int c = 0; c < 8; ++c) F1[k * kPbW + 8 * h + c] = 8 * h + c == k ? ip : a[c];
      }
    }
    if (i > k) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (8 * h + c > k) a[c] = fma(-li, rj[c], a[c]);
    }
  }
}

// y := the solution of the triangle of F (its column k below the diagonal, its diagonal
// inverted), y's entries in registers
template <bool UNIT>
__device__ __forceinline__ void substitute16(double (&y)[kPbW], const double* F) {
#pragma unroll
  for (int k = 0; k < kPbW; ++k) {
    double f[kPbW];
#pragma unroll
    for (int i = k & ~1; i < kPbW; i += 2) {
      const double2 v = *reinterpret_cast<const double2*>(F + k * kPbW + i);
      f[i] = v.x;
      f[i + 1] = v.y;
    }
    if (!UNIT) y[k] *= f[k];
#pragma unroll
    for (int i = k + 1; i < kPbW; ++i) y[i] = fma(-f[i], y[k], y[i]);
  }
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// sym (always with CHOL): the block is taken from its lower triangle (mirrored), so
// that the inverse of a symmetric elimination stays consistent when the input carries
// an asymmetric rounding error.
template <bool CHOL>
__global__ void __launch_bounds__(kPbThreads, 1)
    k_pivot_block(const SweepDesc* __restrict__ descs, const int* __restrict__ active, int k0,
                  double* __restrict__ dinv, int* __restrict__ status, int sym) {
  constexpr int NBLK = kSweepNB / kPbW;
  const int di = active[blockIdx.x];
  const SweepDesc d = descs[di];
  const int nb = min(kSweepNB, d.r - k0);
  extern __shared__ double pb_sm[];
  double* St = pb_sm;                      // [col][row], staging
  double* Rowp = St + kSweepNB * kPbSt;    // [k][col]: rows K
  double* Colp = Rowp + kPbW * kPbLd;      // [k][row]: columns K
  double* Rn = Colp + kPbW * kPbLd;        // [k][col]: G (Cholesky: R)
  double* An = Rn + kPbW * kPbLd;          // [k][row]: -H (Cholesky: -L_iK, I at K)
  double* F0 = An + kPbW * kPbLd;          // the factors of the diagonal block
  double* F1 = F0 + kPbW * kPbW;
  double* Dn = F1 + kPbW * kPbW;           // the next diagonal block
  double* Ls = Dn + kPbW * kPbD;           // 2 x the Cholesky factor, [k][row]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  {
    const double* Bk = d.B + k0 + (long long)k0 * d.n;
#pragma unroll 8
    for (int e = tid; e < kSweepNB * kSweepNB; e += kPbThreads) {
      const int i = e & (kSweepNB - 1), j = e / kSweepNB;
      const int ii = (sym && i < j) ? j : i, jj = (sym && i < j) ? i : j;
      // past nb: the identity, which the elimination leaves alone
      St[i + j * kPbSt] =
          (i < nb && j < nb) ? Bk[ii + (long long)jj * d.n] : (i == j ? 1.0 : 0.0);
    }
  }
  __syncthreads();
  if (warp >= 16) {
    int bad = 0;
    if (warp == 16) {
      for (int e = lane; e < kPbW * kPbW; e += 32)
        Dn[(e & 15) * kPbD + (e >> 4)] = St[(e & 15) + (e >> 4) * kPbSt];
      __syncwarp();
      pivot16<CHOL>(Dn, F0, F1, Ls, nb, bad);
    }
    const int j = tid - 512;
    for (int kb = 0; kb < NBLK; ++kb) {
      const int K = kb * kPbW;
      const bool own = (unsigned)(j - K) < kPbW;
      bar_sync(1, kPbThreads);
      // G and H (Cholesky: R), a column and a row a thread
      const double* src = (CHOL && j > K) ? Colp : Rowp;
      double y[kPbW], z[kPbW];
#pragma unroll
      for (int k = 0; k < kPbW; ++k) {
        y[k] = own ? (j - K == k ? 1.0 : 0.0) : src[k * kPbLd + j];
        if (!CHOL) z[k] = own ? (j - K == k ? 1.0 : 0.0) : -Colp[k * kPbLd + j];
      }
      substitute16<!CHOL>(y, F0);
      if (!CHOL) substitute16<false>(z, F1);
#pragma unroll
      for (int k = 0; k < kPbW; ++k) {
        Rn[k * kPbLd + j] = y[k];
        An[k * kPbLd + j] =
            !CHOL ? z[k] : (own ? (j - K == k ? 1.0 : 0.0) : (j > K ? -y[k] : 0.0));
      }
      bar_arrive(2, kPbThreads);
      if (warp == 16 && kb + 1 < NBLK) {
        bar_sync(3, 64);
        pivot16<CHOL>(Dn, F0, F1, Ls + ((kb + 1) & 1) * kPbW * kPbD, nb - (kb + 1) * kPbW, bad);
      }
    }
    if (bad) atomicOr(status, kStatusTinyPivot);
  } else {
    const int wr = warp & 3, wc = warp >> 2, wm = wr * 32, wn = wc * 32;
    double acc[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          acc[a][b][c] = St[(wm + a * 8 + gq) + (wn + b * 8 + tq * 2 + c) * kPbSt];
    auto step = [&](auto par_, int kb) {
      constexpr int P = decltype(par_)::value;  // kb & 1: the K rows are MMA tiles 2P, 2P + 1
      const int K = kb * kPbW;
      if (wr == kb >> 1 && (!CHOL || wc <= wr)) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 2; ++c)
              Rowp[(a * 8 + gq) * kPbLd + wn + b * 8 + tq * 2 + c] = acc[2 * P + a][b][c];
      }
      if (wc == kb >> 1 && (!CHOL || wc <= wr)) {
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int i = wm + a * 8 + gq, k = b * 8 + tq * 2 + c;
              Colp[k * kPbLd + i] = acc[a][2 * P + b][c];
            }
      }
      // rows and columns K are replaced (Cholesky keeps columns K of the rows above)
      if (wr == kb >> 1) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) acc[2 * P + a][b][0] = acc[2 * P + a][b][1] = 0.0;
      }
      if (wc == kb >> 1) {
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 2; ++b)
            if (!CHOL || wm + a * 8 >= K) acc[a][2 * P + b][0] = acc[a][2 * P + b][1] = 0.0;
      }
      bar_sync(1, kPbThreads);
      bar_sync(2, kPbThreads);
      // A += An Rn, the quadrant that holds the next diagonal block first
      const bool run = !CHOL || (wc <= wr && wm + 32 > K);
      if (run) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int qa = (q & 1) ? P : 1 - P, qb = (q & 2) ? P : 1 - P;
#pragma unroll
          for (int k4 = 0; k4 < kPbW; k4 += 4) {
            double af[2], bf[2];
#pragma unroll
            for (int a = 0; a < 2; ++a)
              af[a] = An[(k4 + tq) * kPbLd + wm + (2 * qa + a) * 8 + gq];
#pragma unroll
            for (int b = 0; b < 2; ++b)
              bf[b] = Rn[(k4 + tq) * kPbLd + wn + (2 * qb + b) * 8 + gq];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
              for (int b = 0; b < 2; ++b) dmma(acc[2 * qa + a][2 * qb + b], af[a], bf[b]);
          }
          if (q == 0 && kb + 1 < NBLK && wr == wc && wr == (kb + 1) >> 1) {
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
              for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                  Dn[(a * 8 + gq) * kPbD + b * 8 + tq * 2 + c] =
                      acc[2 * qa + a][2 * qb + b][c];
            bar_arrive(3, 64);
          }
        }
      }
      if (CHOL) {
        // columns K of L: zeros above, l, L_iK
        const double* L = Ls + (kb & 1) * kPbW * kPbD;
        for (int e = tid; e < kPbW * kSweepNB; e += 512) {
          const int i = e & (kSweepNB - 1), k = e / kSweepNB, r = i - K;
          if (i < nb && K + k < nb)
            d.L[(k0 + i) + (long long)(k0 + K + k) * d.r] =
                r < 0 ? 0.0 : (r < kPbW ? L[k * kPbD + r] : Rn[k * kPbLd + i]);
        }
      }
    };
    for (int kb = 0; kb < NBLK; kb += 2) {
      step(std::integral_constant<int, 0>{}, kb);
      step(std::integral_constant<int, 1>{}, kb + 1);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          St[(wm + a * 8 + gq) + (wn + b * 8 + tq * 2 + c) * kPbSt] = acc[a][b][c];
  }
  __syncthreads();
  double* out = dinv + (long long)di * kSweepNB * kSweepNB;
  for (int e = tid; e < nb * nb; e += kPbThreads) {
    const int i = e % nb, j = e / nb;
    const double v = (CHOL && i < j) ? 0.0 : St[i + j * kPbSt];
    out[e] = v;
    // Gauss-Jordan: the step's panels and updates leave block KK alone; Cholesky:
    // diagonal block K of L^{-1}
    if (!CHOL) d.B[(k0 + i) + (long long)(k0 + j) * d.n] = v;
    else d.a22inv[(k0 + i) + (long long)(k0 + j) * d.r] = v;
  }
}

void launch_sweep_diag(const SweepDesc* d_desc, const int* d_active, int nact, int k0,
                       double* d_dinv, int* d_status, cudaStream_t s, int sym) {
  if (nact <= 0) return;
  ensure_smem((const void*)k_pivot_block<false>, kPbSmem);
  k_pivot_block<false><<<nact, kPbThreads, kPbSmem, s>>>(d_desc, d_active, k0, d_dinv, d_status,
                                                         sym);
}

void launch_chol_diag(const SweepDesc* d_desc, const int* d_active, int nact, int k0,
                      double* d_dinv, int* d_status, cudaStream_t s) {
  if (nact <= 0) return;
  ensure_smem((const void*)k_pivot_block<true>, kPbSmem);
  k_pivot_block<true><<<nact, kPbThreads, kPbSmem, s>>>(d_desc, d_active, k0, d_dinv, d_status,
                                                        1);
}

// ===========================================================================
// Interpolative decomposition (one CTA per face).
//
// Column-pivoted Householder QR (Businger-Golub greedy pivoting on partial
// column norms, with the norm-downdating safeguard of Drmac and Bujanovic:
// recompute a norm when the downdated value lost more than half its digits),
// the reference's per-diagonal skeleton test |R_ii| > eps |R_00|
// (InterpDecomp.cpp:101-110) and W = R11^{-1} R12 restricted to the redundant
// columns, computed with the reference's construction of W_full and R_skel
// (InterpDecomp.cpp:115-137).
// ===========================================================================
// stage_ld > 0: the face matrix is copied into shared memory (after the
// work arrays, at offset stage_off doubles) and the QR runs there; it is
// copied back at the end, so M ends overwritten as without staging.
__global__ void __launch_bounds__(512) k_id(const IdDesc* __restrict__ descs, double eps,
                                            int* __restrict__ status, int stage_off) {
  const IdDesc d = descs[blockIdx.x];
  const int m = d.m, n = d.n;
  extern __shared__ double sm[];
  double* vn1 = sm;
  double* vn2 = vn1 + n;
  double* scratch = vn2 + n;             // 64 doubles
  int* jp = reinterpret_cast<int*>(scratch + 64);
  int* flag = jp + n;                    // n
  int* pos = flag + n;                   // n (skeleton positions, then redundant)
  int* iscratch = pos + n;               // 32 (per-warp argmax indices)
  __shared__ int s_pvt;
  __shared__ int s_k;
  double* M = d.M;
  if (stage_off > 0) {
    M = sm + stage_off;
    for (long long e = threadIdx.x; e < (long long)m * n; e += blockDim.x) M[e] = d.M[e];
    __syncthreads();
  }

  const int tid = threadIdx.x, nthr = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nthr >> 5;
  const double tol3z = sqrt(DBL_EPSILON * 0.5);

  for (int j = tid; j < n; j += nthr) jp[j] = j;
  for (int j = warp; j < n; j += nw) {
    double s = 0.0;
    for (int i = lane; i < m; i += 32) {
      const double v = M[i + (long long)j * m];
      s = fma(v, v, s);
    }
    s = warp_sum(s);
    if (lane == 0) { vn1[j] = sqrt(s); vn2[j] = vn1[j]; }
  }
  __syncthreads();

  const int steps = min(m, n);
  for (int i = 0; i < steps; ++i) {
    // ---- pivot choice
    if (d.order != nullptr) {
      if (tid == 0) s_pvt = i;
      __syncthreads();
      const int want = d.order[i];
      for (int j = i + tid; j < n; j += nthr)
        if (jp[j] == want) s_pvt = j;
      __syncthreads();
    } else {
      // first index of the maximum of vn1[i..n)
      double best = -1.0;
      int bi = INT_MAX;
      for (int j = i + tid; j < n; j += nthr) {
        const double v = vn1[j];
        if (v > best || (v == best && j < bi)) { best = v; bi = j; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      __syncthreads();
      if (lane == 0) { scratch[warp] = best; iscratch[warp] = bi; }
      __syncthreads();
      if (tid == 0) {
        double b = scratch[0];
        int bb = iscratch[0];
        for (int w = 1; w < nw; ++w)
          if (scratch[w] > b || (scratch[w] == b && iscratch[w] < bb)) {
            b = scratch[w];
            bb = iscratch[w];
          }
        s_pvt = (bb == INT_MAX) ? i : bb;
      }
      __syncthreads();
    }
    const int pvt = s_pvt;
    if (pvt != i) {
      for (int r = tid; r < m; r += nthr) {
        const double a = M[r + (long long)i * m];
        M[r + (long long)i * m] = M[r + (long long)pvt * m];
        M[r + (long long)pvt * m] = a;
      }
      if (tid == 0) {
        const int t = jp[pvt];
        jp[pvt] = jp[i];
        jp[i] = t;
        vn1[pvt] = vn1[i];
        vn2[pvt] = vn2[i];
      }
    }
    __syncthreads();
    // ---- Householder reflector for column i, rows i..m-1
    double xs = 0.0;
    for (int r = i + 1 + tid; r < m; r += nthr) {
      const double v = M[r + (long long)i * m];
      xs = fma(v, v, xs);
    }
    const double xnorm = sqrt(block_sum(xs, scratch));
    const double alpha = M[i + (long long)i * m];
    double tau = 0.0, beta = alpha;
    if (xnorm != 0.0) {
      beta = -copysign(hypot(alpha, xnorm), alpha);
      tau = (beta - alpha) / beta;
      const double scal = 1.0 / (alpha - beta);
      for (int r = i + 1 + tid; r < m; r += nthr) M[r + (long long)i * m] *= scal;
    }
    __syncthreads();
    if (tid == 0) {
      M[i + (long long)i * m] = beta;
      d.rdiag[i] = beta;
    }
    __syncthreads();
    // ---- apply H = I - tau [1; v][1; v]^T to columns i+1..n-1
    if (tau != 0.0) {
      for (int j = i + 1 + warp; j < n; j += nw) {
        double* cj = M + (long long)j * m;
        const double* ci = M + (long long)i * m;
        double w = (lane == 0) ? cj[i] : 0.0;
        for (int r = i + 1 + lane; r < m; r += 32) w = fma(ci[r], cj[r], w);
        w = warp_sum(w) * tau;
        if (lane == 0) cj[i] -= w;
        for (int r = i + 1 + lane; r < m; r += 32) cj[r] = fma(-w, ci[r], cj[r]);
      }
    }
    __syncthreads();
    // ---- partial norm downdate
    for (int j = i + 1 + tid; j < n; j += nthr) {
      flag[j] = 0;
      if (vn1[j] != 0.0) {
        double temp = fabs(M[i + (long long)j * m]) / vn1[j];
        temp = fmax(1.0 - temp * temp, 0.0);
        const double q = vn1[j] / vn2[j];
        const double temp2 = temp * q * q;
        if (temp2 <= tol3z) flag[j] = 1;
        else vn1[j] *= sqrt(temp);
      }
    }
    __syncthreads();
    for (int j = i + 1 + warp; j < n; j += nw) {
      if (!flag[j]) continue;
      double s = 0.0;
      for (int r = i + 1 + lane; r < m; r += 32) {
        const double v = M[r + (long long)j * m];
        s = fma(v, v, s);
      }
      s = warp_sum(s);
      if (lane == 0) {
        vn1[j] = (i + 1 < m) ? sqrt(s) : 0.0;
        vn2[j] = vn1[j];
      }
    }
    __syncthreads();
  }

  // ---- rank test
  const double r00 = fabs(M[0]);
  const double tol = r00 * eps;
  if (tid == 0) {
    int k = 0;
    for (int i = 0; i < n; ++i) {
      const int kp = fabs(M[i + (long long)i * m]) > tol;
      flag[i] = kp;
      if (kp) pos[k++] = i;
    }
    int rr = k;
    for (int i = 0; i < n; ++i)
      if (!flag[i]) pos[rr++] = i;
    s_k = k;
    *d.rank = k;
    if (r00 == 0.0) atomicOr(status, kStatusIdZero);
  }
  __syncthreads();
  const int k = s_k;
  for (int j = tid; j < n; j += nthr) {
    d.jpvt[j] = jp[j];
    d.keep[j] = flag[j];
  }
  // ---- W (k x (n-k)): back substitution with R_skel, one redundant column per thread
  //   W_full(a, c) = R(pos[a], c) if c >= a else 0;  R_skel = W_full(:, 0:k)
  const int nred = n - k;
  for (int b = tid; b < nred; b += nthr) {
    const int c = pos[k + b];
    double* x = d.W + (long long)b * k;
    for (int a = 0; a < k; ++a) x[a] = (c >= a) ? M[pos[a] + (long long)c * m] : 0.0;
    for (int a = k - 1; a >= 0; --a) {
      const double xa = x[a] / M[pos[a] + (long long)a * m];
      x[a] = xa;
      for (int t = 0; t < a; ++t) x[t] = fma(-M[pos[t] + (long long)a * m], xa, x[t]);
    }
  }
  if (stage_off > 0)
    for (long long e = threadIdx.x; e < (long long)m * n; e += blockDim.x) d.M[e] = M[e];
}

// The same for narrow faces (n <= 64 columns, m <= 32 RPL rows), NW warps a face, the
// face in shared memory for good. A step is one barrier: every warp finds the pivot and
// forms the reflector itself (columns are swapped by index only, the reflector is
// applied unscaled), then takes its columns through registers: product, update, norm
// downdate or recomputation. The index and norm arrays alternate between two buffers.
// Bound by a step's instructions and latency (every warp's reflector among them).
// k_id's step has about ten barriers: level 1's 11520 faces of 49 columns of n = 128
// took 20.6 ms there, 15.2 ms here; 12 such faces 0.36 and 0.19 ms.
template <int NW, int RPL>
__global__ void __launch_bounds__(NW == 1 ? 128 : NW * 32)
    k_id_small(const IdDesc* __restrict__ descs, int nd, double eps, int* __restrict__ status,
               int max_mn, int max_n) {
  const int lane = threadIdx.x & 31, wi = NW == 1 ? 0 : threadIdx.x >> 5;
  const int slot = NW == 1 ? threadIdx.x >> 5 : 0;
  const int fi = NW == 1 ? blockIdx.x * 4 + slot : blockIdx.x;
  if (fi >= nd) return;
  const IdDesc d = descs[fi];
  const int m = d.m, n = d.n;
  extern __shared__ double is_sm[];
  double* S = is_sm + (size_t)slot * (max_mn + 8 * max_n);
  double* vn1 = S + max_mn;        // 2 x n
  double* vn2 = vn1 + 2 * max_n;   // 2 x n
  double* rd = vn2 + 2 * max_n;    // R's diagonal
  double* sc = rd + max_n;         // scale of the reflector below it
  int* cof = reinterpret_cast<int*>(sc + max_n);  // 2 x n: column at each position
  int* jp = cof + 2 * max_n;
  int* pos = jp + max_n;
  auto sync = [&] {
    if (NW == 1) __syncwarp();
    else __syncthreads();
  };
  const double tol3z = sqrt(DBL_EPSILON * 0.5);
  for (int e = (wi << 5) + lane; e < m * n; e += NW * 32) S[e] = d.M[e];
  sync();
  for (int j = wi; j < n; j += NW) {
    double t = 0.0;
    for (int r = lane; r < m; r += 32) t = fma(S[r + j * m], S[r + j * m], t);
    t = sqrt(warp_sum(t));
    if (lane == 0) {
      vn1[j] = vn2[j] = t;
      cof[j] = j;
    }
  }
  sync();
  const int steps = min(m, n);
  for (int i = 0; i < steps; ++i) {
    const int b = (i & 1) * max_n, nb = max_n - b;
    // pivot: first position of the largest norm (or the prescribed column)
    double best = -1.0;
    int pvt = INT_MAX;
    const int want = d.order ? d.order[i] : -1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = i + lane + 32 * h;
      if (j >= n) continue;
      const double v = d.order ? (cof[b + j] == want ? 1.0 : -1.0) : vn1[b + j];
      if (v > best) {
        best = v;
        pvt = j;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, pvt, o);
      if (ob > best || (ob == best && oi < pvt)) {
        best = ob;
        pvt = oi;
      }
    }
    if (pvt == INT_MAX) pvt = i;
    const int ci = cof[b + pvt];
    const double* x = S + ci * m;
    const double alpha = x[i];
    double xr[RPL], xs[2] = {0.0, 0.0};
#pragma unroll
    for (int u = 0; u < RPL; ++u) {
      const int r = lane + 32 * u;
      xr[u] = (r > i && r < m) ? x[r] : 0.0;
      xs[u & 1] = fma(xr[u], xr[u], xs[u & 1]);
    }
    const double x2 = warp_sum(xs[0] + xs[1]);
    double tau = 0.0, beta = alpha, scal = 1.0;
    if (x2 != 0.0) {
      beta = -copysign(sqrt(fma(alpha, alpha, x2)), alpha);
      tau = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    if (wi == 0 && lane == 0) {
      rd[i] = beta;
      sc[i] = scal;
      jp[i] = ci;
    }
    for (int j = i + 1 + wi; j < n; j += NW) {
      const int from = j == pvt ? i : j;  // position pvt takes over position i's column
      const int cj = cof[b + from];
      double v1 = vn1[b + from], v2 = vn2[b + from];
      double* c = S + cj * m;
      double ar[RPL], ws[2] = {0.0, 0.0};
#pragma unroll
      for (int u = 0; u < RPL; ++u) {
        const int r = lane + 32 * u;
        ar[u] = (r > i && r < m) ? c[r] : 0.0;
        ws[u & 1] = fma(xr[u], ar[u], ws[u & 1]);
      }
      double aij = c[i];
      double w = tau * fma(scal, warp_sum(ws[0] + ws[1]), aij);
      aij -= w;
      w *= scal;
      double ns[2] = {0.0, 0.0};
#pragma unroll
      for (int u = 0; u < RPL; ++u) {
        const int r = lane + 32 * u;
        ar[u] = fma(-w, xr[u], ar[u]);
        ns[u & 1] = fma(ar[u], ar[u], ns[u & 1]);
        if (r > i && r < m) c[r] = ar[u];
      }
      // partial norm downdate, recomputed on cancellation
      if (v1 != 0.0) {
        double temp = fabs(aij) / v1;
        temp = fmax(1.0 - temp * temp, 0.0);
        const double q = v1 / v2;
        if (temp * q * q <= tol3z) v1 = v2 = (i + 1 < m) ? sqrt(warp_sum(ns[0] + ns[1])) : 0.0;
        else v1 *= sqrt(temp);
      }
      __syncwarp();  // every lane has read c[i]
      if (lane == 0) {
        c[i] = aij;
        vn1[nb + j] = v1;
        vn2[nb + j] = v2;
        cof[nb + j] = cj;
      }
    }
    sync();
  }
  // rank test on every diagonal entry
  const double r00 = fabs(rd[0]), tol = r00 * eps;
  const bool k0 = lane < n && fabs(rd[min(lane, n - 1)]) > tol;
  const bool k1 = lane + 32 < n && fabs(rd[min(lane + 32, n - 1)]) > tol;
  const unsigned m0 = __ballot_sync(0xffffffffu, k0), m1 = __ballot_sync(0xffffffffu, k1);
  const int k = __popc(m0) + __popc(m1);
  if (wi == 0) {
    const unsigned below = (1u << lane) - 1u;
    const int q0 = __popc(m0 & below), q1 = __popc(m0) + __popc(m1 & below);
    if (lane < n) pos[k0 ? q0 : k + lane - q0] = lane;
    if (lane + 32 < n) pos[k1 ? q1 : k + lane + 32 - q1] = lane + 32;
    if (lane == 0) {
      *d.rank = k;
      if (r00 == 0.0) atomicOr(status, kStatusIdZero);
    }
    for (int h = 0; h < 2; ++h) {
      const int j = lane + 32 * h;
      if (j >= n) continue;
      d.jpvt[j] = jp[j];
      d.keep[j] = h ? k1 : k0;
      d.rdiag[j] = rd[j];
    }
  }
  sync();
  // W = R_skel^{-1} W_full, a warp per redundant column, lanes over the rows. at(r, c):
  // the QR array as geqp3 leaves it (R, and the scaled reflectors below)
  auto at = [&](int r, int c) {
    const double v = S[r + jp[c] * m];
    return r < c ? v : (r == c ? rd[c] : v * sc[c]);
  };
  for (int q = wi; q < n - k; q += NW) {
    const int c = pos[k + q];
    double x[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int a = lane + 32 * h;
      x[h] = (a < k && c >= a) ? at(pos[a], c) : 0.0;
    }
    for (int a = k - 1; a >= 0; --a) {
      const double xa =
          __shfl_sync(0xffffffffu, a < 32 ? x[0] : x[1], a & 31) / at(pos[a], a);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = lane + 32 * h;
        if (t == a) x[h] = xa;
        else if (t < a) x[h] = fma(-at(pos[t], a), xa, x[h]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (lane + 32 * h < k) d.W[(long long)q * k + lane + 32 * h] = x[h];
  }
}

// ---------------------------------------------------------------------------
// Grouped ID (see hif_kernels.cuh).
// ---------------------------------------------------------------------------
namespace {

// Barrier of the `group` CTAs of one face: arrival counter sync[0], generation
// sync[1]. Bounded spin; on timeout the status word records kStatusTimeout and
// *ok turns false (every CTA then skips to the end).
__device__ void group_barrier(int* sync, int group, int* status, bool* ok) {
  __syncthreads();
  if (group > 1 && threadIdx.x == 0) {
    volatile int* gen = sync + 1;
    const int g0 = *gen;
    __threadfence();
    if (atomicAdd(sync, 1) == group - 1) {
      atomicExch(sync, 0);
      __threadfence();
      atomicAdd(sync + 1, 1);
    } else {
      long long spins = 0;
      while (*gen == g0) {
        if (++spins > (1LL << 28)) {
          atomicOr(status, kStatusTimeout);
          *ok = false;
          break;
        }
      }
    }
    __threadfence();
  }
  __syncthreads();
}

}  // namespace

__global__ void __launch_bounds__(512) k_id_group(const IdGroupDesc* __restrict__ descs,
                                                  int group, double eps,
                                                  int* __restrict__ status) {
  const int face = blockIdx.x / group, me = blockIdx.x % group;
  const IdGroupDesc gd = descs[face];
  const IdDesc d = gd.id;
  const int m = d.m, n = d.n;
  double* M = d.M;
  double* vn1 = gd.norms;
  double* vn2 = gd.norms + n;
  int* jp = d.jpvt;
  extern __shared__ double gsm[];
  double* vsh = gsm;          // reflector rows i..m-1 (m doubles)
  __shared__ double scratch[64];
  __shared__ int iscr[32];
  __shared__ int s_pvt;
  __shared__ bool s_ok;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nthr >> 5;
  const double tol3z = sqrt(DBL_EPSILON * 0.5);
  if (tid == 0) s_ok = true;
  __syncthreads();

  // own columns: j = me, me + group, ...
  for (int j = me + warp * group; j < n; j += nw * group) {
    double sacc = 0.0;
    for (int r = lane; r < m; r += 32) {
      const double v = __ldcg(M + r + (long long)j * m);
      sacc = fma(v, v, sacc);
    }
    sacc = warp_sum(sacc);
    if (lane == 0) {
      __stcg(vn1 + j, sqrt(sacc));
      __stcg(vn2 + j, sqrt(sacc));
      __stcg(jp + j, j);
    }
  }
  group_barrier(gd.sync, group, status, &s_ok);

  const int steps = min(m, n);
  for (int i = 0; i < steps && s_ok; ++i) {
    // ---- candidates over own columns >= i
    double best = -1.0;
    int bi = INT_MAX;
    if (d.order != nullptr) {
      const int want = d.order[i];
      for (int j = i + ((me - i % group + group) % group) + tid * group; j < n; j += nthr * group)
        if (__ldcg(jp + j) == want) { best = 1.0; bi = j; }
    } else {
      for (int j = i + ((me - i % group + group) % group) + tid * group; j < n; j += nthr * group) {
        const double v = __ldcg(vn1 + j);
        if (v > best || (v == best && j < bi)) { best = v; bi = j; }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { scratch[warp] = best; iscr[warp] = bi; }
    __syncthreads();
    if (tid == 0) {
      double b = scratch[0];
      int bb = iscr[0];
      for (int w = 1; w < nw; ++w)
        if (scratch[w] > b || (scratch[w] == b && iscr[w] < bb)) { b = scratch[w]; bb = iscr[w]; }
      __stcg(gd.cand + me, b);
      __stcg(gd.sync + 32 + me, bb);
    }
    group_barrier(gd.sync, group, status, &s_ok);
    if (!s_ok) break;
    if (tid == 0) {
      double b = -1.0;
      int bb = INT_MAX;
      for (int c = 0; c < group; ++c) {
        const double cb = __ldcg(gd.cand + c);
        const int ci = __ldcg(gd.sync + 32 + c);
        if (cb > b || (cb == b && ci < bb)) { b = cb; bb = ci; }
      }
      s_pvt = (bb == INT_MAX) ? i : bb;
    }
    __syncthreads();
    const int pvt = s_pvt;
    // ---- owner of column i: swap, reflector
    if (i % group == me) {
      if (pvt != i) {
        for (int r = tid; r < m; r += nthr) {
          const double a = __ldcg(M + r + (long long)i * m);
          const double b = __ldcg(M + r + (long long)pvt * m);
          __stcg(M + r + (long long)i * m, b);
          __stcg(M + r + (long long)pvt * m, a);
        }
        if (tid == 0) {
          const int t = __ldcg(jp + pvt);
          __stcg(jp + pvt, __ldcg(jp + i));
          __stcg(jp + i, t);
          __stcg(vn1 + pvt, __ldcg(vn1 + i));
          __stcg(vn2 + pvt, __ldcg(vn2 + i));
        }
      }
      __syncthreads();
      double xs = 0.0;
      for (int r = i + 1 + tid; r < m; r += nthr) {
        const double v = __ldcg(M + r + (long long)i * m);
        xs = fma(v, v, xs);
      }
      const double xnorm = sqrt(block_sum(xs, scratch));
      const double alpha = __ldcg(M + i + (long long)i * m);
      double tau = 0.0, beta = alpha;
      if (xnorm != 0.0) {
        beta = -copysign(hypot(alpha, xnorm), alpha);
        tau = (beta - alpha) / beta;
        const double scal = 1.0 / (alpha - beta);
        for (int r = i + 1 + tid; r < m; r += nthr)
          __stcg(M + r + (long long)i * m, __ldcg(M + r + (long long)i * m) * scal);
      }
      __syncthreads();
      if (tid == 0) {
        __stcg(M + i + (long long)i * m, beta);
        d.rdiag[i] = beta;
        __stcg(gd.tau, tau);
      }
    }
    group_barrier(gd.sync, group, status, &s_ok);
    if (!s_ok) break;
    // ---- every CTA: cache the reflector, update its own columns > i
    const double tau = __ldcg(gd.tau);
    for (int r = i + 1 + tid; r < m; r += nthr) vsh[r - i - 1] = __ldcg(M + r + (long long)i * m);
    __syncthreads();
    const int len = m - i - 1;
    const int jfirst = i + 1 + ((me - (i + 1) % group + group) % group);
    if (tau != 0.0) {
      for (int j = jfirst + warp * group; j < n; j += nw * group) {
        double* cj = M + (long long)j * m;
        double w0 = 0.0, w1 = 0.0, w2 = 0.0, w3 = 0.0;
        int r = lane;
        for (; r + 96 < len; r += 128) {
          w0 = fma(vsh[r], __ldcg(cj + i + 1 + r), w0);
          w1 = fma(vsh[r + 32], __ldcg(cj + i + 1 + r + 32), w1);
          w2 = fma(vsh[r + 64], __ldcg(cj + i + 1 + r + 64), w2);
          w3 = fma(vsh[r + 96], __ldcg(cj + i + 1 + r + 96), w3);
        }
        for (; r < len; r += 32) w0 = fma(vsh[r], __ldcg(cj + i + 1 + r), w0);
        double w = warp_sum((w0 + w1) + (w2 + w3));
        const double ci = __ldcg(cj + i);
        w = (w + ci) * tau;
        if (lane == 0) __stcg(cj + i, ci - w);
        for (r = lane; r < len; r += 32)
          __stcg(cj + i + 1 + r, fma(-w, vsh[r], __ldcg(cj + i + 1 + r)));
      }
    }
    __syncthreads();
    // ---- norm downdate of own columns (thread per column), recompute on cancellation
    for (int j = jfirst + tid * group; j < n; j += nthr * group) {
      const double v1 = __ldcg(vn1 + j);
      if (v1 != 0.0) {
        double temp = fabs(__ldcg(M + i + (long long)j * m)) / v1;
        temp = fmax(1.0 - temp * temp, 0.0);
        const double q = v1 / __ldcg(vn2 + j);
        if (temp * q * q <= tol3z) __stcg(vn2 + j, -1.0);  // flag: recompute
        else __stcg(vn1 + j, v1 * sqrt(temp));
      }
    }
    __syncthreads();
    for (int j = jfirst + warp * group; j < n; j += nw * group) {
      if (__ldcg(vn2 + j) != -1.0) continue;
      double sacc = 0.0;
      for (int r = i + 1 + lane; r < m; r += 32) {
        const double v = __ldcg(M + r + (long long)j * m);
        sacc = fma(v, v, sacc);
      }
      sacc = warp_sum(sacc);
      if (lane == 0) {
        const double nv = (i + 1 < m) ? sqrt(sacc) : 0.0;
        __stcg(vn1 + j, nv);
        __stcg(vn2 + j, nv);
      }
    }
    __syncthreads();
  }
  group_barrier(gd.sync, group, status, &s_ok);
  if (!s_ok) return;

  // ---- rank test (every CTA computes the same list) and W (red columns split over the group)
  int* flag = reinterpret_cast<int*>(vsh);
  int* pos = flag + n;
  __shared__ int s_k;
  const double r00 = fabs(__ldcg(M));
  const double tol = r00 * eps;
  if (tid == 0) {
    int k = 0;
    for (int i = 0; i < n; ++i) {
      const int kp = fabs(__ldcg(M + i + (long long)i * m)) > tol;
      flag[i] = kp;
      if (kp) pos[k++] = i;
    }
    int rr = k;
    for (int i = 0; i < n; ++i)
      if (!flag[i]) pos[rr++] = i;
    s_k = k;
    if (me == 0) {
      *d.rank = k;
      if (r00 == 0.0) atomicOr(status, kStatusIdZero);
    }
  }
  __syncthreads();
  const int k = s_k;
  if (me == 0)
    for (int j = tid; j < n; j += nthr) {
      d.jpvt[j] = __ldcg(jp + j);
      d.keep[j] = flag[j];
    }
  const int nred = n - k;
  for (int b = me * nthr + tid; b < nred; b += nthr * group) {
    const int c = pos[k + b];
    double* x = d.W + (long long)b * k;
    for (int a = 0; a < k; ++a) x[a] = (c >= a) ? __ldcg(M + pos[a] + (long long)c * m) : 0.0;
    for (int a = k - 1; a >= 0; --a) {
      const double xa = x[a] / __ldcg(M + pos[a] + (long long)a * m);
      x[a] = xa;
      for (int t = 0; t < a; ++t) x[t] = fma(-__ldcg(M + pos[t] + (long long)a * m), xa, x[t]);
    }
  }
}

cudaError_t launch_id_group(const IdGroupDesc* d_desc, int nd, int group, double eps,
                            int* d_status, cudaStream_t s, int max_m, int max_n) {
  if (nd <= 0) return cudaSuccess;
  size_t smem = (size_t)std::max(max_m, 2 * max_n) * sizeof(double) + 64;
  if (smem > 48 * 1024) ensure_smem((const void*)k_id_group, smem);
  int grid = nd * group;
  if (group > 1) {
    // co-residency of the whole grid is required by the group barriers; the
    // cooperative launch guarantees it or fails without running
    void* args[] = {(void*)&d_desc, (void*)&group, (void*)&eps, (void*)&d_status};
    return cudaLaunchCooperativeKernel((const void*)k_id_group, dim3(grid), dim3(512), args, smem,
                                       s);
  }
  k_id_group<<<grid, 512, smem, s>>>(d_desc, group, eps, d_status);
  return cudaGetLastError();
}

template <int NW, int RPL>
static void launch_id_small(const IdDesc* d_desc, int nd, int max_n, double eps, int* d_status,
                            cudaStream_t s, int max_mn) {
  const int per = NW == 1 ? 4 : 1;
  const size_t smem = (size_t)per * (max_mn + 8 * max_n) * sizeof(double);
  ensure_smem((const void*)k_id_small<NW, RPL>, smem);
  k_id_small<NW, RPL><<<(nd + per - 1) / per, NW == 1 ? 128 : NW * 32, smem, s>>>(
      d_desc, nd, eps, d_status, max_mn, max_n);
}

void launch_id(const IdDesc* d_desc, int nd, int max_n, double eps, int* d_status,
               cudaStream_t s, long long max_mn, int max_m) {
  if (nd <= 0) return;
  // narrow faces that fit in shared memory, their M not needed afterwards: a warp a face
  // up to 16 columns and 128 rows, else sixteen
  if (max_mn > 0 && max_m > 0 && max_n <= 64 && max_m <= 640 &&
      (size_t)(max_mn + 8 * max_n) * sizeof(double) <= (size_t)220 * 1024) {
    if (max_m <= 128 && max_n <= 16)
      launch_id_small<1, 4>(d_desc, nd, max_n, eps, d_status, s, (int)max_mn);
    else if (max_m <= 128)
      launch_id_small<16, 4>(d_desc, nd, max_n, eps, d_status, s, (int)max_mn);
    else
      launch_id_small<16, 20>(d_desc, nd, max_n, eps, d_status, s, (int)max_mn);
    return;
  }
  size_t smem = (size_t)max_n * 2 * sizeof(double) + 64 * sizeof(double) +
                (size_t)max_n * 3 * sizeof(int) + 32 * sizeof(int);
  // faces that fit run from shared memory (the Householder updates then read
  // and write the face on chip instead of through L2)
  int stage_off = 0;
  const size_t off = (smem + sizeof(double) - 1) / sizeof(double);
  if (max_mn > 0 && (off + (size_t)max_mn) * sizeof(double) <= (size_t)200 * 1024) {
    stage_off = (int)off;
    smem = (off + (size_t)max_mn) * sizeof(double);
  }
  // narrow faces: fewer threads per face, more faces per SM
  const int threads = max_n <= 16 ? 128 : 512;
  if (smem > 48 * 1024) ensure_smem((const void*)k_id, smem);
  k_id<<<nd, threads, smem, s>>>(d_desc, eps, d_status, stage_off);
}

// ===========================================================================
// Batched sub-matrix copy (32 x 32 tiles)
// ===========================================================================
int copy_tiles(int m, int n) {
  if (m <= 0 || n <= 0) return 0;
  return ((m + 31) / 32) * ((n + 31) / 32);
}

__global__ void __launch_bounds__(256) k_copy(const CopyDesc* __restrict__ descs,
                                              const int* __restrict__ tile_off, int nd) {
  const int di = find_desc(tile_off, nd, blockIdx.x);
  const CopyDesc c = descs[di];
  const int local = blockIdx.x - tile_off[di];
  const int tm = (c.m + 31) / 32;
  const int i0 = (local % tm) * 32, j0 = (local / tm) * 32;
  for (int e = threadIdx.x; e < 1024; e += blockDim.x) {
    const int i = i0 + (e & 31), j = j0 + (e >> 5);
    if (i < c.m && j < c.n) c.dst[i + (long long)j * c.ldd] = c.src[i + (long long)j * c.lds];
  }
}

void launch_copy(const CopyDesc* d_desc, const int* d_tile_off, int nd, int total_tiles,
                 cudaStream_t s) {
  if (total_tiles <= 0) return;
  k_copy<<<total_tiles, 256, 0, s>>>(d_desc, d_tile_off, nd);
}

// Transposing copy through a shared-memory tile (coalesced on both sides).
__global__ void __launch_bounds__(256) k_tcopy(const TCopyDesc* __restrict__ descs,
                                               const int* __restrict__ tile_off, int nd) {
  const int di = find_desc(tile_off, nd, blockIdx.x);
  const TCopyDesc c = descs[di];
  const int local = blockIdx.x - tile_off[di];
  const int tm = (c.m + 31) / 32;
  const int i0 = (local % tm) * 32, j0 = (local / tm) * 32;
  __shared__ double t[32][33];
  // read: consecutive threads take consecutive j (contiguous in src)
  for (int e = threadIdx.x; e < 1024; e += blockDim.x) {
    const int jj = e & 31, ii = e >> 5;
    const int i = i0 + ii, j = j0 + jj;
    t[jj][ii] = (i < c.m && j < c.n) ? c.src[j + (long long)i * c.lds] : 0.0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 1024; e += blockDim.x) {
    const int ii = e & 31, jj = e >> 5;
    const int i = i0 + ii, j = j0 + jj;
    if (i < c.m && j < c.n) c.dst[i + (long long)j * c.ldd] = c.alpha * t[jj][ii];
  }
}

void launch_tcopy(const TCopyDesc* d_desc, const int* d_tile_off, int nd, int total_tiles,
                  cudaStream_t s) {
  if (total_tiles <= 0) return;
  k_tcopy<<<total_tiles, 256, 0, s>>>(d_desc, d_tile_off, nd);
}

// ===========================================================================
// Row compression: blocked Householder QR panels (one CTA per face)
// ===========================================================================
__global__ void __launch_bounds__(512) k_qr_panel(const QrDesc* __restrict__ descs,
                                                  const int* __restrict__ active, int k0,
                                                  int vrow0) {
  const QrDesc d = descs[active[blockIdx.x]];
  const int m = d.m, kb = min(kQrNB, d.n - k0);
  double* Vout = d.V + (long long)(k0 - vrow0) * m;  // this sub-panel's columns of V
  double* M = d.M;
  __shared__ double s_tau[kQrNB];
  __shared__ double scratch[64];
  __shared__ double T[kQrNB * kQrNB];
  __shared__ double Wd[kQrNB * kQrNB];
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int nw = nthr >> 5;
  for (int j = 0; j < kb; ++j) {
    const int col = k0 + j;
    double* cc = M + (long long)col * m;
    double xs = 0.0;
    for (int r = col + 1 + tid; r < m; r += nthr) xs = fma(cc[r], cc[r], xs);
    const double xnorm = sqrt(block_sum(xs, scratch));
    const double alpha = cc[col];
    double tau = 0.0, beta = alpha;
    if (xnorm != 0.0) {
      beta = -copysign(hypot(alpha, xnorm), alpha);
      tau = (beta - alpha) / beta;
      const double scal = 1.0 / (alpha - beta);
      for (int r = col + 1 + tid; r < m; r += nthr) cc[r] *= scal;
    }
    __syncthreads();
    if (tid == 0) {
      cc[col] = beta;
      s_tau[j] = tau;
    }
    __syncthreads();
    if (tau != 0.0) {
      for (int c = col + 1 + warp; c < k0 + kb; c += nw) {
        double* cj = M + (long long)c * m;
        double w = (lane == 0) ? cj[col] : 0.0;
        for (int r = col + 1 + lane; r < m; r += 32) w = fma(cc[r], cj[r], w);
        w = warp_sum(w) * tau;
        if (lane == 0) cj[col] -= w;
        for (int r = col + 1 + lane; r < m; r += 32) cj[r] = fma(-w, cc[r], cj[r]);
      }
    }
    __syncthreads();
  }
  // explicit V (unit diagonal, zeros above) for rows vrow0..m-1
  const int mt = m - vrow0;
  for (long long e = tid; e < (long long)mt * kb; e += nthr) {
    const int rr = (int)(e % mt), j = (int)(e / mt);
    const int r = vrow0 + rr;
    double v = 0.0;
    if (r == k0 + j) v = 1.0;
    else if (r > k0 + j) v = M[r + (long long)(k0 + j) * m];
    Vout[r + (long long)j * m] = v;
  }
  for (int j = tid; j < kb; j += nthr) d.tau[k0 - vrow0 + j] = s_tau[j];
  __syncthreads();
  // Wd = V^T V in one pass over the rows: lane c holds V[r, c]; the products
  // with every other column come by shuffle. Warps add their partial sums in
  // warp order (deterministic).
  {
    double acc[kQrNB];
#pragma unroll
    for (int i = 0; i < kQrNB; ++i) acc[i] = 0.0;
    for (int r = k0 + warp; r < m; r += nw) {
      const double v = (lane < kb) ? Vout[r + (long long)lane * m] : 0.0;
#pragma unroll
      for (int i = 0; i < kQrNB; ++i) acc[i] = fma(__shfl_sync(0xffffffffu, v, i), v, acc[i]);
    }
    for (int e = tid; e < kQrNB * kQrNB; e += nthr) Wd[e] = 0.0;
    __syncthreads();
    for (int w = 0; w < nw; ++w) {
      if (warp == w) {
#pragma unroll
        for (int i = 0; i < kQrNB; ++i) Wd[i + lane * kQrNB] += acc[i];
      }
      __syncthreads();
    }
  }
  // T (forward, columnwise): T[j,j] = tau_j, T[0:j, j] = -tau_j T[0:j,0:j] Wd[0:j, j]
  for (int j = 0; j < kb; ++j) {
    if (tid < j) {
      double acc = 0.0;
      for (int l = tid; l < j; ++l) acc = fma(T[tid + l * kQrNB], Wd[l + j * kQrNB], acc);
      T[tid + j * kQrNB] = -s_tau[j] * acc;
    }
    if (tid == 0) T[j + j * kQrNB] = s_tau[j];
    for (int i = j + 1 + tid; i < kQrNB; i += nthr) T[i + j * kQrNB] = 0.0;
    __syncthreads();
  }
  for (int e = tid; e < kQrNB * kQrNB; e += nthr) {
    const int i = e % kQrNB, j = e / kQrNB;
    d.T[e] = (i < kb && j < kb) ? T[e] : 0.0;
  }
}

// ---------------------------------------------------------------------------
// The same sub-panel factorization by a thread-block cluster per face: the
// cluster's CTAs split the panel's rows (at most kQrcRows each) and keep them
// in shared memory for the whole panel. Per column, every CTA sums over its
// rows the squared norm below the diagonal and the products of the column with
// the columns to its right; the owner of the diagonal row adds that row's
// entries. One cluster barrier, then every CTA adds the CTAs' partial vectors
// in rank order (identical sums everywhere, deterministic), forms the
// reflector (beta, tau) exactly as the single-CTA kernel does and updates its
// rows. Partial vectors alternate between two buffers, so one barrier per
// column orders both the reads of step j and the writes of step j + 2.
// ---------------------------------------------------------------------------
namespace cg = cooperative_groups;
constexpr int kQrcRows = 768;
constexpr int kQrcSlots = 2 * kQrNB + 2;  // [norm^2 | x.A_c (32) | alpha | A[col, c] (32)]

__global__ void __launch_bounds__(512) k_qr_panel_cluster(const QrDesc* __restrict__ descs,
                                                          const int* __restrict__ active,
                                                          int k1, int vrow0) {
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const QrDesc d = descs[active[blockIdx.x / C]];
  const int m = d.m, kb = min(kQrNB, d.n - k1), mt = m - k1;
  const int chunk = (mt + C - 1) / C;
  const int r0 = k1 + rank * chunk, r1 = min(m, r0 + chunk), nr = max(0, r1 - r0);
  const int ld = chunk | 1;  // odd: lanes reading one row of 32 columns hit distinct banks
  extern __shared__ double P[];  // nr x kQrNB, ld ld (local rows r0..r1)
  __shared__ double red[2][kQrcSlots];
  __shared__ double wpart[16][kQrcSlots];
  __shared__ double tot[kQrcSlots];
  __shared__ double gram[kQrNB * kQrNB];
  __shared__ double s_tau[kQrNB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x;
  double* M = d.M;
  for (int e = tid; e < nr * kQrNB; e += nthr) {
    const int i = e % nr, c = e / nr;
    P[i + c * ld] = (c < kb) ? M[(r0 + i) + (long long)(k1 + c) * m] : 0.0;
  }
  __syncthreads();
  for (int j = 0; j < kb; ++j) {
    const int col = k1 + j;
    // partial sums over local rows below the diagonal
    double acc[kQrNB + 1];
#pragma unroll
    for (int c = 0; c <= kQrNB; ++c) acc[c] = 0.0;
    for (int i = tid; i < nr; i += nthr) {
      if (r0 + i <= col) continue;
      const double x = P[i + j * ld];
      acc[0] = fma(x, x, acc[0]);
#pragma unroll
      for (int c = 0; c < kQrNB; ++c)
        if (c > j) acc[1 + c] = fma(x, P[i + c * ld], acc[1 + c]);
    }
    // warp reduce-scatter of acc[1..32] (5 halving exchanges, 31 shuffles):
    // afterwards lane c holds the warp's total of acc[1 + c]; acc[0] by warp_sum
    {
      const double n2 = warp_sum(acc[0]);
      if (lane == 0) wpart[warp][0] = n2;
#pragma unroll
      for (int h = 16; h >= 1; h >>= 1) {
        const bool upper = (lane & h) != 0;
#pragma unroll
        for (int c = 0; c < h; ++c) {
          // keep the half selected by this lane's bit, send the other half
          const double send = upper ? acc[1 + c] : acc[1 + c + h];
          const double keep = upper ? acc[1 + c + h] : acc[1 + c];
          acc[1 + c] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
      }
      // the kept halves follow the lane's bits from high to low: acc[1] of lane c
      // is the warp's total for column c
      wpart[warp][1 + lane] = acc[1];
    }
    __syncthreads();
    double* rb = red[j & 1];
    if (tid <= kQrNB) {
      double sacc = 0.0;
      for (int w = 0; w < (nthr >> 5); ++w) sacc += wpart[w][tid];
      rb[tid] = sacc;
    } else if (tid <= 2 * kQrNB + 1) {
      // diagonal-row entries (alpha and A[col, c]) from the CTA that owns the row
      const int c = tid - (kQrNB + 1);  // 0 -> alpha, 1 + c' -> A[col, c']
      double v = 0.0;
      if (col >= r0 && col < r1) {
        const int cc = (c == 0) ? j : c - 1;
        if (c == 0 || (cc > j && cc < kb)) v = P[(col - r0) + cc * ld];
      }
      rb[tid] = v;
    }
    cl.sync();
    if (tid < kQrcSlots) {
      double v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = (q < C) ? cl.map_shared_rank(rb, q)[tid] : 0.0;
      double sacc = 0.0;
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (q < C) sacc += v[q];
      tot[tid] = sacc;
    }
    __syncthreads();
    const double xnorm = sqrt(tot[0]);
    const double alpha = tot[kQrNB + 1];
    double tau = 0.0, beta = alpha, scal = 1.0;
    if (xnorm != 0.0) {
      beta = -copysign(hypot(alpha, xnorm), alpha);
      tau = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    // update the local rows: v = x * scal below the diagonal, w_c = tau (A[col, c] + v . A_c)
    for (int i = tid; i < nr; i += nthr) {
      const int r = r0 + i;
      if (r < col) continue;
      if (r == col) {
        P[i + j * ld] = beta;
        for (int c = j + 1; c < kb; ++c) {
          const double w = tau * (tot[kQrNB + 2 + c] + scal * tot[1 + c]);
          P[i + c * ld] -= w;
        }
      } else {
        const double v = (xnorm != 0.0) ? P[i + j * ld] * scal : P[i + j * ld];
        P[i + j * ld] = v;
        for (int c = j + 1; c < kb; ++c) {
          const double w = tau * (tot[kQrNB + 2 + c] + scal * tot[1 + c]);
          P[i + c * ld] = fma(-w, v, P[i + c * ld]);
        }
      }
    }
    if (tid == 0) s_tau[j] = tau;
    __syncthreads();
  }
  // results: the panel back to M, V (unit diagonal, zeros above) for rows
  // vrow0.., tau
  double* Vout = d.V + (long long)(k1 - vrow0) * m;
  for (int e = tid; e < nr * kb; e += nthr) {
    const int i = e % nr, c = e / nr;
    const int r = r0 + i;
    const double p = P[i + c * ld];
    M[r + (long long)(k1 + c) * m] = p;
    Vout[r + (long long)c * m] = (r == k1 + c) ? 1.0 : (r > k1 + c ? p : 0.0);
  }
  if (rank == 0) {
    for (int e = tid; e < (k1 - vrow0) * kb; e += nthr) {
      const int i = e % (k1 - vrow0), c = e / (k1 - vrow0);
      Vout[vrow0 + i + (long long)c * m] = 0.0;
    }
    for (int j = tid; j < kb; j += nthr) d.tau[k1 - vrow0 + j] = s_tau[j];
  }
  // W = V^T V: local partial Gram (lane c holds column c; products with every
  // other column by shuffle), warps added in warp order, CTAs summed by rank 0
  // in rank order
  {
    double accg[kQrNB];
#pragma unroll
    for (int a = 0; a < kQrNB; ++a) accg[a] = 0.0;
    for (int i = warp; i < nr; i += (nthr >> 5)) {
      const int r = r0 + i;
      const double v = (lane < kb) ? (r == k1 + lane ? 1.0 : (r > k1 + lane ? P[i + lane * ld] : 0.0))
                                   : 0.0;
#pragma unroll
      for (int a = 0; a < kQrNB; ++a) accg[a] = fma(__shfl_sync(0xffffffffu, v, a), v, accg[a]);
    }
    for (int e = tid; e < kQrNB * kQrNB; e += nthr) gram[e] = 0.0;
    __syncthreads();
    for (int w = 0; w < (nthr >> 5); ++w) {
      if (warp == w) {
#pragma unroll
        for (int a = 0; a < kQrNB; ++a) gram[a + lane * kQrNB] += accg[a];
      }
      __syncthreads();
    }
  }
  cl.sync();
  if (rank == 0) {
    // the panel rows are no longer needed: W and T live in their space
    double* Wsum = P;
    double* Tl = P + kQrNB * kQrNB;
    for (int e = tid; e < kQrNB * kQrNB; e += nthr) {
      double g = 0.0;
      for (int q = 0; q < C; ++q) g += cl.map_shared_rank(gram, q)[e];
      Wsum[e] = g;
      Tl[e] = 0.0;
    }
    __syncthreads();
    for (int j = 0; j < kb; ++j) {
      if (tid < j) {
        double a = 0.0;
        for (int l = tid; l < j; ++l) a = fma(Tl[tid + l * kQrNB], Wsum[l + j * kQrNB], a);
        Tl[tid + j * kQrNB] = -s_tau[j] * a;
      }
      if (tid == 0) Tl[j + j * kQrNB] = s_tau[j];
      __syncthreads();
    }
    for (int e = tid; e < kQrNB * kQrNB; e += nthr) d.T[e] = Tl[e];
  }
  cl.sync();  // no CTA leaves while rank 0 reads its shared memory
}

void launch_qr_panel(const QrDesc* d_desc, const int* d_active, int nact, int k1, int k0,
                     cudaStream_t s) {
  if (nact <= 0) return;
  k_qr_panel<<<nact, 512, 0, s>>>(d_desc, d_active, k1, k0);
}

int qr_cluster_max_rows() {
  // per device: the attributes and the cluster occupancy belong to the device
  static std::mutex mu;
  static std::map<int, int> caps;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  int& cap = caps.emplace(dev, -1).first->second;
  if (cap < 0) {
    ensure_smem((const void*)k_qr_panel_cluster, (kQrcRows + 1) * kQrNB * 8);
    cudaFuncSetAttribute(k_qr_panel_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    // the largest cluster the device can place with this kernel's footprint
    int best = 1;
    for (int c : {16, 8}) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(c, 1, 1);
      cfg.blockDim = dim3(512, 1, 1);
      cfg.dynamicSmemBytes = (kQrcRows + 1) * kQrNB * 8;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = c;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, k_qr_panel_cluster, &cfg) == cudaSuccess && n > 0) {
        best = c;
        break;
      }
      cudaGetLastError();
    }
    cap = best * kQrcRows;
  }
  return cap;
}

void launch_qr_panel_cluster(const QrDesc* d_desc, const int* d_active, int nact, int k1,
                             int k0, int max_rows, cudaStream_t s) {
  if (nact <= 0) return;
  const int C = std::max(1, (max_rows + kQrcRows - 1) / kQrcRows);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nact * C, 1, 1);
  cfg.blockDim = dim3(512, 1, 1);
  cfg.dynamicSmemBytes = (kQrcRows + 1) * kQrNB * 8;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_qr_panel_cluster, d_desc, d_active, k1, k0);
}

// One CTA per outer panel: the forward column recurrence for T over kQrNB2
// reflectors (T kept in shared memory, 128 KB).
__global__ void __launch_bounds__(256) k_qr_tfactor(const TFactorDesc* __restrict__ descs) {
  const TFactorDesc d = descs[blockIdx.x];
  extern __shared__ double Ts[];  // kQrNB2 x kQrNB2
  const int nb = d.nb, tid = threadIdx.x;
  for (int e = tid; e < kQrNB2 * kQrNB2; e += blockDim.x) Ts[e] = 0.0;
  __syncthreads();
  for (int j = 0; j < nb; ++j) {
    const double tj = d.tau[j];
    for (int i = tid; i < j; i += blockDim.x) {
      double acc = 0.0;
      for (int l = i; l < j; ++l) acc = fma(Ts[i + l * kQrNB2], d.W[l + j * kQrNB2], acc);
      Ts[i + j * kQrNB2] = -tj * acc;
    }
    if (tid == 0) Ts[j + j * kQrNB2] = tj;
    __syncthreads();
  }
  for (int e = tid; e < kQrNB2 * kQrNB2; e += blockDim.x) d.T[e] = Ts[e];
}

void launch_qr_tfactor(const TFactorDesc* d_desc, int nd, cudaStream_t s) {
  if (nd <= 0) return;
  ensure_smem((const void*)k_qr_tfactor, kQrNB2 * kQrNB2 * 8);
  k_qr_tfactor<<<nd, 256, kQrNB2 * kQrNB2 * 8, s>>>(d_desc);
}

__global__ void k_triu(const TriuDesc* __restrict__ descs) {
  const TriuDesc d = descs[blockIdx.y];
  const long long nn = (long long)d.n * d.n;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nn;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % d.n), j = (int)(e / d.n);
    d.dst[i + j * d.ldd] = (i <= j) ? d.src[i + j * d.lds] : 0.0;
  }
}

void launch_triu(const TriuDesc* d_desc, int nd, cudaStream_t s) {
  if (nd <= 0) return;
  dim3 grid(64, nd);
  k_triu<<<grid, 256, 0, s>>>(d_desc);
}

__global__ void k_trsm_upper(const double* __restrict__ R, long long ldr, int k,
                             double* __restrict__ B, long long ldb, int nb) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nb) return;
  double* x = B + (long long)c * ldb;
  for (int a = k - 1; a >= 0; --a) {
    const double xa = x[a] / R[a + (long long)a * ldr];
    x[a] = xa;
    for (int t = 0; t < a; ++t) x[t] = fma(-R[t + (long long)a * ldr], xa, x[t]);
  }
}

void launch_trsm_upper(const double* R, long long ldr, int k, double* B, long long ldb, int nb,
                       cudaStream_t s) {
  if (nb <= 0 || k <= 0) return;
  k_trsm_upper<<<(nb + 127) / 128, 128, 0, s>>>(R, ldr, k, B, ldb, nb);
}

// ===========================================================================
// Pivoted Cholesky panels: nb steps of a face's G, by one CTA, or a cluster that
// splits the columns of a wide face (the panel's rows of R stay in shared memory).
// Bound by the latency of a step: the pivot search, the pivot's column of G from L2 or
// HBM, the products with the panel's earlier rows. A step is one block barrier (and one
// cluster barrier): every warp reduces the warps' candidates itself, and the earlier
// rows' pivot entries are broadcast reads. With R's rows re-read from L2 and a serial
// search a step took about 15 us (144 faces of 767 columns, 0.5 ms a panel); the
// panels of an n = 128 factorization take 7.0 ms mixed and 9.5 ms FP64, 18 ms mixed then.
// ===========================================================================
constexpr int kPcMaxW = 832;  // columns of one CTA: 32 rows of them in shared memory
__device__ __forceinline__ void argmax_step(double& best, int& bi, double ob, int oi) {
  if (ob > best || (ob == best && oi < bi)) {
    best = ob;
    bi = oi;
  }
}
__global__ void __launch_bounds__(512) k_pchol_panel(const PcholDesc* __restrict__ descs,
                                                     const int* __restrict__ active, int i0,
                                                     int nb, double eps, int* __restrict__ status) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const PcholDesc P = descs[active[blockIdx.x / C]];
  const int n = P.id.n, tid = threadIdx.x, nthr = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nthr >> 5;
  const int w = (n + C - 1) / C, c0 = rank * w, cols = max(0, min(w, n - c0));
  extern __shared__ double pc_sm[];  // [row of the panel][own column], ld w
  __shared__ double s_v[2][16];
  __shared__ int s_i[2][16];
  __shared__ double x_v[2][16];  // candidates of the cluster's CTAs
  __shared__ int x_i[2][16];
  __shared__ double pcol[32];
  const double* G = P.G;
  double* R = P.R;
  if (P.info[1]) return;  // the same in every CTA of the face
  if (C > 1) cl.sync();   // every CTA runs before its shared memory is written from outside
  // own columns tid, tid + nthr: remaining diagonal, -1 once chosen
  constexpr int Q = 2;
  double d[Q];
  double mx = 0.0;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int j = tid + q * nthr;
    d[q] = -1.0;
    if (j < cols && (i0 == 0 || !P.chosen[c0 + j])) {
      d[q] = fmax(G[(c0 + j) + (long long)(c0 + j) * n], 0.0);
      mx = fmax(mx, d[q]);
    }
  }
  double d0;
  int buf = 0;
  // best over the face of each thread's (best, index): the same on every thread
  auto face_argmax = [&](double& best, int& bi) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      argmax_step(best, bi, __shfl_xor_sync(0xffffffffu, best, o),
                  __shfl_xor_sync(0xffffffffu, bi, o));
    if (lane == 0) {
      s_v[buf][warp] = best;
      s_i[buf][warp] = bi;
    }
    __syncthreads();
    best = lane < nw ? s_v[buf][lane & 15] : -2.0;
    bi = lane < nw ? s_i[buf][lane & 15] : INT_MAX;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
      argmax_step(best, bi, __shfl_xor_sync(0xffffffffu, best, o),
                  __shfl_xor_sync(0xffffffffu, bi, o));
    best = __shfl_sync(0xffffffffu, best, 0);
    bi = __shfl_sync(0xffffffffu, bi, 0);
    if (C > 1) {
      if (tid < C) {
        cl.map_shared_rank(&x_v[buf][0], tid)[rank] = best;
        cl.map_shared_rank(&x_i[buf][0], tid)[rank] = bi;
      }
      cl.sync();
      best = x_v[buf][0];
      bi = x_i[buf][0];
      for (int q = 1; q < C; ++q) argmax_step(best, bi, x_v[buf][q], x_i[buf][q]);
    }
    buf ^= 1;
  };
  if (i0 == 0) {
    int dummy = 0;
    face_argmax(mx, dummy);
    d0 = mx;
    if (tid == 0 && rank == 0) {
      *P.d0 = d0;
      if (!(d0 > 0.0)) atomicOr(status, kStatusIdZero);
    }
  } else {
    d0 = *P.d0;
  }
  const double thr = eps * eps * d0;
  const int iend = min(n, i0 + nb);
  int i = i0;
  bool stop = false;
  for (; i < iend; ++i) {
    // pivot: largest remaining diagonal, smallest index on ties
    double best = -2.0;
    int bi = INT_MAX;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int j = tid + q * nthr;
      if (j < cols && d[q] >= 0.0) argmax_step(best, bi, d[q], c0 + j);
    }
    face_argmax(best, bi);
    // R_ii <= eps R_00 (or nothing left): the rank is i
    if (bi == INT_MAX || !(best > thr)) {
      stop = true;
      break;
    }
    const int p = bi, rows = i - i0;
    double g[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int j = c0 + tid + q * nthr;
      // only the lower triangle of G is kept: G[j, p] for j > p, G[p, j] above
      g[q] = (tid + q * nthr < cols && d[q] >= 0.0 && j != p)
                 ? ((j > p) ? G[j + (long long)p * n] : G[p + (long long)j * n]) : 0.0;
    }
    const double rii = sqrt(best), inv = 1.0 / rii;
    const double* pr;  // the earlier rows' entries at the pivot
    int ps;
    if (C == 1) {
      pr = pc_sm + p;
      ps = w;
    } else {
      const int own = p / w;
      if (tid < rows) pcol[tid] = cl.map_shared_rank(pc_sm, own)[tid * w + (p - own * w)];
      __syncthreads();
      pr = pcol;
      ps = 1;
    }
    double* Ri = R + (long long)i * n + c0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int j = tid + q * nthr;
      if (j >= cols) continue;
      double r = 0.0;
      if (d[q] >= 0.0) {
        if (c0 + j == p) {
          r = rii;
          d[q] = -1.0;
        } else {
          double s0 = g[q], s1 = 0.0;
          int l = 0;
#pragma unroll 4
          for (; l + 1 < rows; l += 2) {
            s0 = fma(-pr[l * ps], pc_sm[l * w + j], s0);
            s1 = fma(-pr[(l + 1) * ps], pc_sm[(l + 1) * w + j], s1);
          }
          if (l < rows) s0 = fma(-pr[l * ps], pc_sm[l * w + j], s0);
          r = (s0 + s1) * inv;
          // the remaining diagonal stays a candidate: not below zero
          d[q] = fmax(fma(-r, r, d[q]), 0.0);
        }
      }
      pc_sm[(i - i0) * w + j] = r;
      Ri[j] = r;
    }
    if (tid == 0 && rank == 0) P.piv[i] = p;
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int j = tid + q * nthr;
    if (j < cols) P.chosen[c0 + j] = d[q] < 0.0;
  }
  if (C > 1) cl.sync();  // every CTA has read info[1], and the last remote rows
  if (tid == 0 && rank == 0) {
    P.info[0] = i;
    if (stop || i == n) P.info[1] = 1;
  }
}

void launch_pchol_panel(const PcholDesc* d_desc, const int* d_active, int nact, int i0, int nb,
                        double eps, int max_n, int* d_status, cudaStream_t s) {
  if (nact <= 0) return;
  int C = 1;
  while (C < 16 && max_n > C * kPcMaxW) C *= 2;
  if (C == 16)
    cudaFuncSetAttribute(k_pchol_panel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  const int w = (max_n + C - 1) / C;
  const size_t smem = (size_t)nb * w * sizeof(double);
  ensure_smem((const void*)k_pchol_panel, (size_t)32 * kPcMaxW * sizeof(double));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nact * C, 1, 1);
  cfg.blockDim = dim3(w <= 256 ? 256 : 512, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = C > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_pchol_panel, d_desc, d_active, i0, nb, eps, d_status);
}

__global__ void __launch_bounds__(512) k_pchol_finish(const PcholDesc* __restrict__ descs) {
  const PcholDesc P = descs[blockIdx.x];
  const int n = P.id.n, tid = threadIdx.x, nthr = blockDim.x;
  extern __shared__ int pf_sm[];  // order: n
  __shared__ int s_k;
  if (tid == 0) {
    const int k = P.info[0];
    int q = 0;
    for (int i = 0; i < k; ++i) pf_sm[q++] = P.piv[i];
    for (int j = 0; j < n; ++j)
      if (!P.chosen[j]) pf_sm[q++] = j;
    s_k = k;
    *P.id.rank = k;
  }
  __syncthreads();
  const int k = s_k;
  const double* R = P.R;
  for (int i = tid; i < n; i += nthr) {
    P.id.jpvt[i] = pf_sm[i];
    P.id.keep[i] = i < k;
    P.id.rdiag[i] = (i < k) ? R[(long long)i * n + pf_sm[i]] : 0.0;
  }
  // R11 (k x k, ld k, upper) into G's space; R12 into W (k x (n - k), ld k)
  double* R11 = P.G;
  for (long long e = tid; e < (long long)k * k; e += nthr) {
    const int a = (int)(e % k), b = (int)(e / k);
    R11[e] = (b >= a) ? R[(long long)a * n + pf_sm[b]] : 0.0;
  }
  const int nr = n - k;
  for (long long e = tid; e < (long long)k * nr; e += nthr) {
    const int a = (int)(e % k), c = (int)(e / k);
    P.id.W[e] = R[(long long)a * n + pf_sm[k + c]];
  }
}

void launch_pchol_finish(const PcholDesc* d_desc, int nd, int max_n, cudaStream_t s) {
  if (nd <= 0) return;
  const size_t smem = (size_t)max_n * sizeof(int);
  if (smem > 48 * 1024) ensure_smem((const void*)k_pchol_finish, smem);
  k_pchol_finish<<<nd, 512, smem, s>>>(d_desc);
}

// One CTA per (face, 128 columns): the diagonal block of R11 in shared memory,
// one column of W per thread, back substitution over the block's rows.
__global__ void __launch_bounds__(128) k_trsm_block(const TrsmBlockDesc* __restrict__ descs,
                                                    int chunks) {
  const TrsmBlockDesc t = descs[blockIdx.x / chunks];
  const int c = (blockIdx.x % chunks) * 128 + threadIdx.x;
  const int bs = t.a1 - t.a0;
  extern __shared__ double tb_sm[];
  double* Rb = tb_sm;                    // kTrsmNB x kTrsmNB
  double* X = tb_sm + kTrsmNB * kTrsmNB;  // kTrsmNB x 128
  if (bs <= 0) return;
  for (int e = threadIdx.x; e < bs * bs; e += blockDim.x) {
    const int a = e % bs, b = e / bs;
    Rb[a + b * kTrsmNB] = t.R[(t.a0 + a) + (long long)(t.a0 + b) * t.k];
  }
  const bool live = c < t.ncols;
  if (live)
    for (int a = 0; a < bs; ++a)
      X[a * 128 + threadIdx.x] = t.W[(t.a0 + a) + (long long)c * t.k];
  __syncthreads();
  if (!live) return;
  for (int a = bs - 1; a >= 0; --a) {
    const double xa = X[a * 128 + threadIdx.x] / Rb[a + a * kTrsmNB];
    X[a * 128 + threadIdx.x] = xa;
    for (int r = 0; r < a; ++r)
      X[r * 128 + threadIdx.x] = fma(-Rb[r + a * kTrsmNB], xa, X[r * 128 + threadIdx.x]);
  }
  for (int a = 0; a < bs; ++a) t.W[(t.a0 + a) + (long long)c * t.k] = X[a * 128 + threadIdx.x];
}

void launch_trsm_block(const TrsmBlockDesc* d_desc, int nd, int max_cols, cudaStream_t s) {
  if (nd <= 0 || max_cols <= 0) return;
  const int chunks = (max_cols + 127) / 128;
  const int smem = (kTrsmNB * kTrsmNB + kTrsmNB * 128) * (int)sizeof(double);
  ensure_smem((const void*)k_trsm_block, smem);
  k_trsm_block<<<nd * chunks, 128, smem, s>>>(d_desc, chunks);
}

// ===========================================================================
// Column-pivoted QR of tall faces by phases (see PqrDesc). The flops are in the
// batched products (Gram, Q1, Q1^T T, T -= Q1 D); these kernels move columns and
// do the k x k work around them, bound by their traffic or by launch latency.
// At n = 128 the three wide levels' decompositions took 758 ms as row compression
// plus a column-by-column pivoted QR (each step reading and writing the whole
// trailing face), 218 ms by phases.
// ===========================================================================

// Thread = row of a 256-row chunk, so every column access is coalesced and a row's
// picked entries are saved before the displaced columns overwrite them.
__global__ void __launch_bounds__(256) k_pqr_extract(const PqrDesc* __restrict__ descs) {
  const PqrDesc d = descs[blockIdx.y];
  const int k = d.k, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((int)blockIdx.x * 256 >= d.m) return;
  __shared__ int piv[kPqrCap], sel[kPqrCap], from[kPqrCap], to[kPqrCap], wsum[2][8];
  if (tid < kPqrCap) sel[tid] = 0;
  __syncthreads();
  int p = -1;
  if (tid < k) {
    p = d.piv[tid];
    piv[tid] = p;
    if (p < k) sel[p] = 1;
  }
  __syncthreads();
  // unpicked positions below k (ascending) go to the picked positions beyond k
  const bool isf = tid < k && !sel[tid], ist = tid < k && p >= k;
  const unsigned bf = __ballot_sync(0xffffffffu, isf), bt = __ballot_sync(0xffffffffu, ist);
  if (lane == 0) {
    wsum[0][warp] = __popc(bf);
    wsum[1][warp] = __popc(bt);
  }
  __syncthreads();
  int of = 0, ot = 0, nmove = 0;
  for (int w = 0; w < 8; ++w) {
    if (w < warp) {
      of += wsum[0][w];
      ot += wsum[1][w];
    }
    nmove += wsum[0][w];
  }
  const unsigned below = (1u << lane) - 1u;
  if (isf) from[of + __popc(bf & below)] = tid;
  if (ist) to[ot + __popc(bt & below)] = p;
  __syncthreads();
  // eight columns' loads in flight before their stores
  const int r = blockIdx.x * 256 + tid;
  if (r < d.m) {
    double* T = d.T + (long long)d.o * d.m + r;
    double* S = d.S + r;
    for (int i0 = 0; i0 < k; i0 += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = (i0 + u < k) ? T[(long long)piv[i0 + u] * d.m] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i0 + u < k) S[(long long)(i0 + u) * d.m] = v[u];
    }
    // sources lie below k, destinations beyond: no overlap
    for (int q0 = 0; q0 < nmove; q0 += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = (q0 + u < nmove) ? T[(long long)from[q0 + u] * d.m] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (q0 + u < nmove) T[(long long)to[q0 + u] * d.m] = v[u];
    }
  }
  if (blockIdx.x == 0) {
    int* perm = d.perm + d.o;
    int mine = 0, moved = 0;
    if (tid < k) mine = perm[piv[tid]];
    if (tid < nmove) moved = perm[from[tid]];
    __syncthreads();
    if (tid < k) perm[tid] = mine;
    if (tid < nmove) perm[to[tid]] = moved;
    const int w = d.n - d.o;
    for (int e = tid; e < k * k; e += 256) {
      const int a = e % k, b = e / k;
      d.R1[e] = (b >= a) ? d.Rsel[(long long)a * w + piv[b]] : 0.0;
    }
  }
}

void launch_pqr_extract(const PqrDesc* d_desc, int nd, int max_m, cudaStream_t s) {
  if (nd <= 0) return;
  k_pqr_extract<<<dim3((max_m + 255) / 256, nd), 256, 0, s>>>(d_desc);
}

// R1^{-1} by 32-wide block columns, a CTA each (they are independent): block row i
// of column j is R_ii^{-1} (I_ij - sum_{l > i} R_il X_lj), from the diagonal up.
constexpr int kPqrTi = 32;
__global__ void __launch_bounds__(256) k_pqr_trinv(const PqrDesc* __restrict__ descs) {
  const PqrDesc d = descs[blockIdx.y];
  const int k = d.k, j0 = blockIdx.x * kPqrTi, tid = threadIdx.x;
  if (j0 >= k) return;
  const int nc = min(kPqrTi, k - j0), rows = j0 + nc;
  extern __shared__ double ti_sm[];
  double* X = ti_sm;                                  // [c][row], rows <= kPqrCap
  double* Rt = X + kPqrTi * (kPqrCap + 1);            // 32 x 33
  double* Y = Rt + kPqrTi * (kPqrTi + 1);             // 32 x 33: [c][row]
  const int tx = tid & 31, ty = tid >> 5;             // row, column group of 4
  for (int i0 = j0; i0 >= 0; i0 -= kPqrTi) {
    const int nr = min(kPqrTi, k - i0);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const double* Ri = d.R1 + i0 + tx;
    for (int l = i0 + kPqrTi; l < rows; ++l) {
      const double rv = (tx < nr) ? Ri[(long long)l * k] : 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = fma(rv, X[(ty * 4 + q) * (kPqrCap + 1) + l], acc[q]);
    }
    for (int e = tid; e < kPqrTi * kPqrTi; e += 256) {
      const int a = e % kPqrTi, b = e / kPqrTi;
      const double v = (a < nr && b < nr) ? d.R1[(i0 + a) + (long long)(i0 + b) * k]
                                          : (a == b ? 1.0 : 0.0);
      Rt[b * (kPqrTi + 1) + a] = (a == b) ? 1.0 / v : v;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = ty * 4 + q;
      Y[c * (kPqrTi + 1) + tx] =
          (tx < nr) ? ((i0 == j0 && tx == c) ? 1.0 : 0.0) - acc[q] : 0.0;
    }
    __syncthreads();
    if (tid < nc) {
      double y[kPqrTi];
#pragma unroll
      for (int a = 0; a < kPqrTi; ++a) y[a] = Y[tid * (kPqrTi + 1) + a];
#pragma unroll
      for (int a = kPqrTi - 1; a >= 0; --a) {
        y[a] *= Rt[a * (kPqrTi + 1) + a];
#pragma unroll
        for (int t = 0; t < kPqrTi; ++t)
          if (t < a) y[t] = fma(-Rt[a * (kPqrTi + 1) + t], y[a], y[t]);
      }
#pragma unroll
      for (int a = 0; a < kPqrTi; ++a)
        if (a < nr) X[tid * (kPqrCap + 1) + i0 + a] = y[a];
    }
    __syncthreads();
  }
  for (int e = tid; e < k * nc; e += 256) {
    const int a = e % k, c = e / k;
    d.R1inv[a + (long long)(j0 + c) * k] = (a < rows) ? X[c * (kPqrCap + 1) + a] : 0.0;
  }
}

void launch_pqr_trinv(const PqrDesc* d_desc, int nd, int max_k, cudaStream_t s) {
  if (nd <= 0) return;
  const int smem = (kPqrTi * (kPqrCap + 1) + 2 * kPqrTi * (kPqrTi + 1)) * (int)sizeof(double);
  ensure_smem((const void*)k_pqr_trinv, smem);
  k_pqr_trinv<<<dim3((max_k + kPqrTi - 1) / kPqrTi, nd), 256, smem, s>>>(d_desc);
}

// A CTA per 32 columns of [R1 | Q1^T T], C in shared memory: row a needs the sums of
// E(a, l) C(l) over l < a and l > a. A thread holds 4 rows (32 apart) x 4 columns; E goes
// through shared memory 32 columns at a time, in ascending l, so a row block's running
// sum is the first until its diagonal block and the second after it. (Reading E from L2
// at every l, bound by that latency: 3.0 ms a launch over 1344 faces of 224 columns,
// 2.0 ms now.)
constexpr int kPqrFc = 32;
__global__ void __launch_bounds__(256, 2) k_pqr_fix(const PqrDesc* __restrict__ descs) {
  const PqrDesc d = descs[blockIdx.y];
  const int k = d.k, cols = d.n - d.o, c0 = blockIdx.x * kPqrFc, tid = threadIdx.x;
  if (c0 >= cols) return;
  const int nc = min(kPqrFc, cols - c0);
  extern __shared__ double fx_sm[];  // [row][c], ld kPqrFc
  __shared__ double Es[32][128];
  for (int e = tid; e < k * kPqrFc; e += 256) {
    const int a = e % k, c = e / k, j = c0 + c;
    fx_sm[a * kPqrFc + c] =
        c >= nc ? 0.0 : (j < k) ? d.R1[a + (long long)j * k] : d.Z[a + (long long)j * k];
  }
  const int tx = tid & 31, ty = tid >> 5;  // row within 32, group of 4 columns
  const double* E = d.Z;                   // Q1^T Q1 (symmetric), ld k
  const double r00 = d.o == 0 ? d.R1[0] : d.Rr[(long long)d.perm[0] * d.n];
  const double lim = fmin(kPqrMaxE * sqrt(fabs(r00) / d.R1[0]), kPqrCapE);
  bool bad = false;
  for (int a0 = 0; a0 < k; a0 += 128) {
    double lo[4][4] = {}, acc[4][4] = {}, ed[4] = {};
    const int nu = min(4, (k - a0 + 31) / 32);
    for (int l0 = 0; l0 < k; l0 += 32) {
      const int nl = min(32, k - l0);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int e = tid + 256 * q, r = e & 127, l = e >> 7, a = a0 + r;
        double v = (l < nl && a < k) ? E[a + (long long)(l0 + l) * k] : 0.0;
        if (l < nl && a == l0 + l) v -= 1.0;
        bad |= !(fabs(v) <= lim);
        Es[l][r] = v;
      }
      __syncthreads();
      const int ud = (l0 - a0) / 32;  // row block of this chunk's diagonal, if in [0, 4)
      const bool diag = l0 >= a0 && ud < 4;
      for (int l = 0; l < nl; ++l) {
        const double2* cp = reinterpret_cast<const double2*>(fx_sm + (l0 + l) * kPqrFc + ty * 4);
        const double2 c01 = cp[0], c23 = cp[1];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (u >= nu) break;
          const double e = (diag && u == ud) ? 0.0 : Es[l][tx + 32 * u];
          acc[u][0] = fma(e, c01.x, acc[u][0]);
          acc[u][1] = fma(e, c01.y, acc[u][1]);
          acc[u][2] = fma(e, c23.x, acc[u][2]);
          acc[u][3] = fma(e, c23.y, acc[u][3]);
        }
      }
      if (diag) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (u != ud) continue;
          double dn[4] = {0.0, 0.0, 0.0, 0.0};
          for (int l = 0; l < nl; ++l) {
            const double e = Es[l][tx + 32 * u];
            const double el = l < tx ? e : 0.0, eu = l > tx ? e : 0.0;
            if (l == tx) ed[u] = e;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const double c = fx_sm[(l0 + l) * kPqrFc + ty * 4 + q];
              acc[u][q] = fma(el, c, acc[u][q]);
              dn[q] = fma(eu, c, dn[q]);
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            lo[u][q] = acc[u][q];
            acc[u][q] = dn[q];
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int a = a0 + tx + 32 * u;
      if (a >= k) continue;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = ty * 4 + q, j = c0 + c;
        if (c >= nc) continue;
        const double v = fx_sm[a * kPqrFc + c];
        double* out = d.Rr + (long long)d.perm[d.o + j] * d.n + d.o + a;
        if (j < k) {
          // column j of R11 = (I + U) R1 (zero below the diagonal)
          *out = (j >= a) ? v + 0.5 * ed[u] * v + acc[u][q] : 0.0;
        } else {
          *out = v - (lo[u][q] + 0.5 * ed[u] * v);
          d.Z[a + (long long)j * k] = v - (lo[u][q] + ed[u] * v + acc[u][q]);
        }
      }
    }
  }
  if (bad) atomicOr(d.flag, 1);
}

void launch_pqr_fix(const PqrDesc* d_desc, int nd, int max_k, int max_cols, cudaStream_t s) {
  if (nd <= 0) return;
  const int smem = kPqrFc * max_k * (int)sizeof(double);
  ensure_smem((const void*)k_pqr_fix, kPqrFc * kPqrCap * sizeof(double));
  k_pqr_fix<<<dim3((max_cols + kPqrFc - 1) / kPqrFc, nd), 256, smem, s>>>(d_desc);
}

__global__ void __launch_bounds__(512) k_pqr_finish(const PqrOut* __restrict__ outs, double eps,
                                                    int* __restrict__ status) {
  const PqrOut o = outs[blockIdx.x];
  const int n = o.id.n, tid = threadIdx.x, nthr = blockDim.x;
  extern __shared__ int pn_sm[];  // perm
  __shared__ int s_k, s_last;
  if (tid == 0) s_k = s_last = 0;
  for (int i = tid; i < n; i += nthr) pn_sm[i] = o.perm[i];
  __syncthreads();
  const double r00 = fabs(o.Rr[(long long)pn_sm[0] * n]), tol = r00 * eps;
  for (int i = tid; i < n; i += nthr) {
    const double v = o.Rr[(long long)pn_sm[i] * n + i];
    const int kp = fabs(v) > tol;
    if (blockIdx.y == 0) {
      o.id.jpvt[i] = pn_sm[i];
      o.id.rdiag[i] = v;
      o.id.keep[i] = kp;
    }
    if (kp) {
      atomicAdd(&s_k, 1);
      atomicMax(&s_last, i + 1);
    }
  }
  __syncthreads();
  const int k = s_k;
  if (tid == 0 && blockIdx.y == 0) {
    *o.id.rank = k;
    if (s_last != k) atomicOr(o.flag, 2);
    if (r00 == 0.0) atomicOr(status, kStatusIdZero);
  }
  // R by position: R11 (ld k, upper) and R12, split over the face's CTAs
  for (long long e = tid + (long long)blockIdx.y * nthr; e < (long long)k * n;
       e += (long long)nthr * gridDim.y) {
    const int a = (int)(e % k), i = (int)(e / k);
    const double v = (i >= a) ? o.Rr[(long long)pn_sm[i] * n + a] : 0.0;
    if (i < k) o.R11[a + (long long)i * k] = v;
    else o.id.W[a + (long long)(i - k) * k] = v;
  }
}

void launch_pqr_finish(const PqrOut* d_out, int nd, double eps, int max_n, int* status,
                       cudaStream_t s) {
  if (nd <= 0) return;
  const size_t smem = (size_t)max_n * sizeof(int);
  if (smem > 48 * 1024) ensure_smem((const void*)k_pqr_finish, smem);
  k_pqr_finish<<<dim3(nd, nd < sm_count() ? 16 : 2), 512, smem, s>>>(d_out, eps, status);
}

// ===========================================================================
// Source membership (one CTA per cell / face)
// ===========================================================================
__global__ void k_member_cells(const int* __restrict__ skel, const long long* __restrict__ off,
                               const int* __restrict__ src, int cpd, int w, int NC,
                               int* __restrict__ dof_src) {
  const int b = blockIdx.x;
  const int id = src[b];
  if (id < 0) return;
  const long long n3 = (long long)NC * NC * NC;
  const int c[3] = {b / (cpd * cpd), (b / cpd) % cpd, b % cpd};
  const long long o = off[b], s = off[b + 1] - o;
  for (long long t = threadIdx.x; t < s; t += blockDim.x) {
    const int p = skel[o + t];
    const int x[3] = {p % NC, (p / NC) % NC, p / (NC * NC)};
    int slot = 1;  // high face
    for (int a = 0; a < 3; ++a)
      if (x[a] % w == 0 && x[a] == w * c[a]) slot = 0;  // low face
    dof_src[(2 * slot) * n3 + p] = id;
    dof_src[(2 * slot + 1) * n3 + p] = (int)t;
  }
}

void launch_member_cells(const int* d_skel, const long long* d_off, const int* d_src, int ncell,
                         int cpd, int w, int NC, int* d_dof_src, cudaStream_t s) {
  if (ncell <= 0) return;
  k_member_cells<<<ncell, 128, 0, s>>>(d_skel, d_off, d_src, cpd, w, NC, d_dof_src);
}

__global__ void k_member_faces(const int* __restrict__ skel, const long long* __restrict__ off,
                               const int* __restrict__ cnt, const int* __restrict__ src,
                               long long n3, int* __restrict__ dof_src) {
  const int q = blockIdx.x;
  const long long o = off[q];
  for (int t = threadIdx.x; t < cnt[q]; t += blockDim.x) {
    const int p = skel[o + t];
    dof_src[4 * n3 + p] = src[q];
    dof_src[5 * n3 + p] = t;
  }
}

void launch_member_faces(const int* d_skel, const long long* d_off, const int* d_cnt,
                         const int* d_src, int nq, long long n3, int* d_dof_src, cudaStream_t s) {
  if (nq <= 0) return;
  k_member_faces<<<nq, 128, 0, s>>>(d_skel, d_off, d_cnt, d_src, n3, d_dof_src);
}

// ===========================================================================
// Apply sweeps: y = op(M) x[in] for every block of a phase, x and y through DOF lists.
// The work vectors hold the right-hand sides of a DOF side by side (element (p, c) at
// u[p * nrhs + c]; contribution slots likewise), so that a gather or scatter moves
// whole rows of right-hand sides. One vector: streaming GEMVs, bound by reading the
// factor once. Several: DMMA tiles over all of them, each factor entry read once per
// 64. Every sum has a fixed order.
// ===========================================================================
struct GemvCtx {
  const double* uin;
  double* uout;
  double* contrib;
  int nrhs;
};
__device__ __forceinline__ GemvCtx gemv_ctx(const GemvDesc& g, const GemvCtx& k) {
  return g.uin ? GemvCtx{g.uin, g.uout, g.contrib, g.nrhs} : k;
}

__device__ __forceinline__ void gemv_emit(const GemvDesc& g, const GemvCtx& x, int i, int c,
                                          double y) {
  if (g.mode == 1) {
    x.contrib[(g.cslot + i) * x.nrhs + c] = y;
  } else {
    double* u = x.uout + (long long)g.out_idx[i] * x.nrhs + c;
    *u = g.mode == 0 ? *u + g.alpha * y : g.alpha * y;
  }
}

// One vector, blocks of at most kGemvSmallElems entries, a warp each: the whole block
// and its x go to shared memory first, every load independent of the others (a warp
// that loads an index, then x, then a column at a time waits for each: 0.9 TB/s on
// level 0's 27 x 54 blocks), then lane = output.
__global__ void __launch_bounds__(256) k_gemv_small(const GemvFastSeg* __restrict__ segs,
                                                    const int* __restrict__ seg_off, int nseg,
                                                    GemvCtx k, int elems) {
  extern __shared__ double gs_sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = blockIdx.x * 8 + warp;
  if (unit >= seg_off[nseg]) return;
  const int si = nseg == 1 ? 0 : find_desc(seg_off, nseg, unit);
  const GemvDesc g = segs[si].desc[unit - seg_off[si]];
  const GemvCtx x = gemv_ctx(g, k);
  double* S = gs_sm + warp * (elems + kGemvSmallMax);
  double* xs = S + elems;
  const int len = g.trans ? g.m : g.n, out = g.trans ? g.n : g.m, mn = g.m * g.n;
  // ld == m: the block is contiguous
  for (int e0 = 0; e0 < mn; e0 += 32 * 16) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int e = e0 + u * 32 + lane;
      v[u] = e < mn ? __ldg(g.M + e) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int e = e0 + u * 32 + lane;
      if (e < mn) S[e] = v[u];
    }
  }
#pragma unroll
  for (int h = 0; h < kGemvSmallMax / 32; ++h) {
    const int j = lane + 32 * h;
    if (j < len) xs[j] = x.uin[g.in_idx[j]];
  }
  __syncwarp();
  for (int i = lane; i < out; i += 32) {
    double acc = 0.0;
    if (g.trans == 0) {
      const int jend = g.tri ? min(g.n, i + 1) : g.n;
#pragma unroll 8
      for (int j = 0; j < jend; ++j) acc = fma(S[i + j * g.m], xs[j], acc);
    } else {
      const int r0 = g.tri ? i : 0;
#pragma unroll 8
      for (int r = r0; r < g.m; ++r) acc = fma(S[r + i * g.m], xs[r], acc);
    }
    gemv_emit(g, x, i, 0, acc);
  }
}

// One vector, larger blocks: a unit is a run of 32-wide tiles of outputs of one block.
// y = M x: lane = row, the columns of a chunk split over the 8 warps; y = M^T x: a
// warp's four columns at each row. x goes to shared memory in chunks (kept from tile
// to tile where one chunk is all of it) after the first 16 entries of M a thread needs
// have been requested, so the two gathers and the stream of M overlap. Where a launch
// has few units, a cluster of CTAs shares each and adds its parts in rank order
// through distributed shared memory: the top levels' blocks, 82 tiles of 2612 columns
// at n = 96, else leave half the SMs idle and the others latency-bound (1.8 TB/s).
constexpr int kG1Chunk = 1024;
__global__ void __launch_bounds__(256, 3) k_gemv1(const GemvFastSeg* __restrict__ segs,
                                                  const int* __restrict__ seg_off, int nseg,
                                                  GemvCtx k) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  __shared__ double xs[kG1Chunk];
  __shared__ double red[8][33];
  __shared__ double part[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int unit = blockIdx.x / C;
  const int si = nseg == 1 ? 0 : find_desc(seg_off, nseg, unit);
  const int4 t = segs[si].tab[unit - seg_off[si]];
  const GemvDesc g = segs[si].desc[t.x];
  const GemvCtx x = gemv_ctx(g, k);
  const int len = g.trans ? g.m : g.n, out = g.trans ? g.n : g.m;
  int held0 = -1, held1 = -1;  // range of x in xs
  for (int tile = t.y; tile < t.y + t.z; ++tile) {
    const int o0 = tile * 32;
    // lower triangular: a strip of rows needs no column past its last row, a tile of
    // columns no row before its first
    const int lo = (g.tri && g.trans) ? o0 : 0, hi = (g.tri && !g.trans) ? min(len, o0 + 32) : len;
    const int per = (((hi - lo + C - 1) / C) + 31) & ~31;
    const int a = lo + rank * per, b = min(hi, a + per);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int c0 = a; c0 < b; c0 += kG1Chunk) {
      const int nj = min(kG1Chunk, b - c0);
      const bool stage = c0 != held0 || c0 + nj != held1;
      // first loads of M, then x
      double v[16];
      const double* Mp;
      int j0, j1;  // columns of this warp in the chunk (y = M x)
      if (g.trans == 0) {
        const int cnt = (nj + 7) / 8;
        j0 = warp * cnt;
        j1 = min(nj, j0 + cnt);
        Mp = g.M + min(o0 + lane, g.m - 1) + (long long)c0 * g.ld;
#pragma unroll
        for (int u = 0; u < 16; ++u)
          v[u] = j0 + u < j1 ? __ldg(Mp + (long long)(j0 + u) * g.ld) : 0.0;
      } else {
        j0 = j1 = 0;
        Mp = g.M + c0 + lane;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double* col = Mp + (long long)min(o0 + warp * 4 + q, g.n - 1) * g.ld;
#pragma unroll
          for (int u = 0; u < 4; ++u)
            v[q * 4 + u] = u * 32 + lane < nj ? __ldg(col + u * 32) : 0.0;
        }
      }
      if (stage) {
        __syncthreads();  // readers of the previous chunk are done
        int id[kG1Chunk / 256];
#pragma unroll
        for (int u = 0; u < kG1Chunk / 256; ++u) {
          const int e = u * 256 + tid;
          id[u] = e < nj ? g.in_idx[c0 + e] : -1;
        }
#pragma unroll
        for (int u = 0; u < kG1Chunk / 256; ++u)
          xs[u * 256 + tid] = id[u] >= 0 ? x.uin[id[u]] : 0.0;
        __syncthreads();
        held0 = c0;
        held1 = c0 + nj;
      }
      if (g.trans == 0) {
        double s0 = acc[0];
        for (int j = j0; j < j1; j += 16) {
          if (j > j0) {
#pragma unroll
            for (int u = 0; u < 16; ++u)
              v[u] = j + u < j1 ? __ldg(Mp + (long long)(j + u) * g.ld) : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 16; ++u)
            if (j + u < j1) s0 = fma(v[u], xs[j + u], s0);
        }
        acc[0] = s0;
      } else {
        for (int r0 = 0; r0 < nj; r0 += 128) {
          if (r0 > 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const double* col = Mp + r0 + (long long)min(o0 + warp * 4 + q, g.n - 1) * g.ld;
#pragma unroll
              for (int u = 0; u < 4; ++u)
                v[q * 4 + u] = r0 + u * 32 + lane < nj ? __ldg(col + u * 32) : 0.0;
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const double xv = r0 + u * 32 + lane < nj ? xs[r0 + u * 32 + lane] : 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] = fma(v[q * 4 + u], xv, acc[q]);
          }
        }
      }
    }
    if (g.trans == 0) {
      red[warp][lane] = acc[0];
      __syncthreads();
      if (warp == 0) {
        double y = red[0][lane];
#pragma unroll
        for (int w = 1; w < 8; ++w) y += red[w][lane];
        part[lane] = y;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double y = warp_sum(acc[q]);
        if (lane == 0) part[warp * 4 + q] = y;
      }
    }
    if (C > 1) {
      cl.sync();
      if (rank == 0 && tid < 32 && o0 + tid < out) {
        double y = part[tid];
        for (int q = 1; q < C; ++q) y += cl.map_shared_rank(part, q)[tid];
        gemv_emit(g, x, o0 + tid, 0, y);
      }
      cl.sync();
    } else {
      __syncthreads();
      if (tid < 32 && o0 + tid < out) gemv_emit(g, x, o0 + tid, 0, part[tid]);
      __syncthreads();
    }
  }
}

// Several vectors: 64 outputs x BN right-hand sides per CTA on DMMA, the reduction
// through the cp.async pipeline of k_dgemm with the B rows gathered from u. Four warps
// of 16 outputs; a cluster shares the reduction where tiles are few (as in k_gemv1),
// each rank adding up its share of the outputs. Bound by the factor's stream up to
// about 20 right-hand sides, by the DMMA pipe beyond. It replaced gather, product and
// emit launches for 16 and more vectors, padded to 64 (F u of 24 vectors at n = 48:
// 1.21 ms), and GEMVs over groups of 4 below that.
constexpr int kMmaIdx = 2048;
template <int BN>
constexpr int apply_mma_smem() {
  return (BN >= 32 ? 3 : 4) * kGBK * (64 + 4 + BN + 4) * (int)sizeof(double);
}
template <int BN>
__global__ void __launch_bounds__(128, BN == 64 ? 3 : 4)
    k_apply_mma(const GemvFastSeg* __restrict__ segs, const int* __restrict__ seg_off, int nseg,
                GemvCtx kx) {
  namespace cg = cooperative_groups;
  constexpr int T = 128, BM = 64, ST = BN >= 32 ? 3 : 4;
  constexpr int SA = BM + 4, SB = BN + 4, QA = BM * kGBK / T, QB = BN * kGBK / T;
  constexpr int NB = BN / 8;
  extern __shared__ double lsm[];
  double* As = lsm;
  double* Bs = lsm + ST * kGBK * SA;
  __shared__ int idx[kMmaIdx];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int unit = blockIdx.x / C;
  const int si = nseg == 1 ? 0 : find_desc(seg_off, nseg, unit);
  const int4 tb = segs[si].tab[unit - seg_off[si]];
  const GemvDesc g = segs[si].desc[tb.x];
  const GemvCtx x = gemv_ctx(g, kx);
  const int r0 = blockIdx.y * BN;  // first right-hand side
  if (r0 >= x.nrhs) return;        // the same in every CTA of the cluster
  const int nr = min(BN, x.nrhs - r0);
  const int len = g.trans ? g.m : g.n, out = g.trans ? g.n : g.m;
  const int m0 = tb.y * BM;
  const int lo = (g.tri && g.trans) ? m0 : 0, hi = (g.tri && !g.trans) ? min(len, m0 + BM) : len;
  const int per = (((hi - lo + C - 1) / C) + kGBK - 1) / kGBK * kGBK;
  const int ka = lo + rank * per, kb = min(hi, ka + per);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  // A(row, k): M[row + k ld], or M[k + row ld] transposed; copies as in k_dgemm
  const bool ta = g.trans != 0;
  const int amm = ta ? tid / kGBK : tid % BM, akk = ta ? tid % kGBK : tid / BM;
  const long long astep = (long long)(ta ? T / kGBK : T / BM) * g.ld;
  const long long aadv = ta ? kGBK : (long long)kGBK * g.ld;
  const int as0 = akk * SA + amm, asq = ta ? T / kGBK : (T / BM) * SA;
  const int bc = tid % BN, bkk = tid / BN;
  const bool bok = bc < nr;
  unsigned amask = 0;
#pragma unroll
  for (int q = 0; q < QA; ++q)
    if (m0 + amm + (ta ? (T / kGBK) * q : 0) < out) amask |= 1u << q;
  double acc[2][NB][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  for (int s0 = ka; s0 < kb; s0 += kMmaIdx) {
    const int s1 = min(kb, s0 + kMmaIdx), nk = (s1 - s0 + kGBK - 1) / kGBK;
    __syncthreads();
    for (int e = tid; e < s1 - s0; e += T) idx[e] = g.in_idx[s0 + e];
    __syncthreads();
    const double* ap = ta ? g.M + s0 + akk + (long long)(m0 + amm) * g.ld
                          : g.M + (m0 + amm) + (long long)(s0 + akk) * g.ld;
    auto issue_a = [&](int stage, int k0, int part, int parts) {
      double* as = As + stage * kGBK * SA + as0;
#pragma unroll
      for (int q = 0; q < QA; ++q)
        if (q >= QA / parts * part && q < QA / parts * (part + 1)) {
          const bool ok = (amask >> q & 1) && k0 + akk + (ta ? 0 : (T / BM) * q) < s1;
          cp_async8(as + q * asq, ok ? ap + q * astep : g.M, ok);
        }
    };
    auto issue_b = [&](int stage, int k0) {
      double* bs = Bs + stage * kGBK * SB;
#pragma unroll
      for (int q = 0; q < QB; ++q) {
        const int kk = bkk + (T / BN) * q;
        const bool ok = bok && k0 + kk < s1;
        cp_async8(bs + kk * SB + bc,
                  ok ? x.uin + (long long)idx[k0 + kk - s0] * x.nrhs + r0 + bc : x.uin, ok);
      }
    };
#pragma unroll
    for (int st = 0; st < ST - 1; ++st) {
      if (st < nk) {
        issue_a(st, s0 + st * kGBK, 0, 1);
        issue_b(st, s0 + st * kGBK);
        ap += aadv;
      }
      cp_async_commit();
    }
    for (int t = 0; t < nk; ++t) {
      cp_async_wait<ST - 2>();
      __syncthreads();
      const int nt = t + ST - 1, k0n = s0 + nt * kGBK;
      const double* as = As + (t % ST) * kGBK * SA + tq * SA + warp * 16 + gq;
      const double* bs = Bs + (t % ST) * kGBK * SB + tq * SB + gq;
      if (nt < nk) issue_b(nt % ST, k0n);
#pragma unroll
      for (int k4 = 0; k4 < kGBK / 4; ++k4) {
        double af[2], bf[NB];
#pragma unroll
        for (int a = 0; a < 2; ++a) af[a] = as[k4 * 4 * SA + a * 8];
#pragma unroll
        for (int b = 0; b < NB; ++b) bf[b] = bs[k4 * 4 * SB + b * 8];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < NB; ++b) dmma(acc[a][b], af[a], bf[b]);
        if (nt < nk) issue_a(nt % ST, k0n, k4, kGBK / 4);
      }
      cp_async_commit();
      ap += aadv;
    }
    cp_async_wait<0>();
  }
  if (C > 1) {
    // parts to shared memory, [output][right-hand side]
    constexpr int LP = BN + 2;
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          lsm[(warp * 16 + a * 8 + gq) * LP + b * 8 + tq * 2 + c] = acc[a][b][c];
    cl.sync();
    const int rows = BM / C;
    for (int e = tid; e < rows * BN; e += T) {
      const int i = rank * rows + e / BN, c = e % BN;
      if (m0 + i >= out || c >= nr) continue;
      double y = 0.0;
      for (int q = 0; q < C; ++q) y += cl.map_shared_rank(lsm, q)[i * LP + c];
      gemv_emit(g, x, m0 + i, r0 + c, y);
    }
    cl.sync();
  } else {
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int i = m0 + warp * 16 + a * 8 + gq;
      if (i >= out) continue;
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int rc = b * 8 + tq * 2 + c;
          if (rc < nr) gemv_emit(g, x, i, r0 + rc, acc[a][b][c]);
        }
    }
  }
}

template <class K>
void launch_clustered(K kernel, dim3 grid, int threads, int smem, int cluster, cudaStream_t s,
                      const GemvFastSeg* segs, const int* off, int nseg, GemvCtx k) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, segs, off, nseg, k);
}

int apply_rhs_class(int nrhs) {
  return nrhs == 1 ? 1 : nrhs <= 8 ? 8 : nrhs <= 16 ? 16 : nrhs <= 32 ? 32 : 64;
}

void launch_gemv(const GemvFastSeg* d_segs, const int* d_seg_off, int nseg, int units,
                 const GemvLayout& lay, const double* u_in, double* u_out, double* contrib,
                 int nrhs, cudaStream_t s) {
  if (units <= 0) return;
  const GemvCtx k{u_in, u_out, contrib, nrhs};
  const dim3 grid(units * lay.cluster, (nrhs + 63) / 64);
  switch (lay.kind == kGemvMulti ? apply_rhs_class(std::max(2, nrhs)) : lay.kind) {
    case kGemvSmall: {
      const int smem = 8 * (lay.elems + kGemvSmallMax) * (int)sizeof(double);
      ensure_smem((const void*)k_gemv_small, smem);
      k_gemv_small<<<(units + 7) / 8, 256, smem, s>>>(d_segs, d_seg_off, nseg, k, lay.elems);
      break;
    }
    case kGemvTiles:
      launch_clustered(k_gemv1, dim3(units * lay.cluster), 256, 0, lay.cluster, s, d_segs,
                       d_seg_off, nseg, k);
      break;
    case 8:
      ensure_smem((const void*)k_apply_mma<8>, apply_mma_smem<8>());
      launch_clustered(k_apply_mma<8>, grid, 128, apply_mma_smem<8>(), lay.cluster, s, d_segs,
                       d_seg_off, nseg, k);
      break;
    case 16:
      ensure_smem((const void*)k_apply_mma<16>, apply_mma_smem<16>());
      launch_clustered(k_apply_mma<16>, grid, 128, apply_mma_smem<16>(), lay.cluster, s, d_segs,
                       d_seg_off, nseg, k);
      break;
    case 32:
      ensure_smem((const void*)k_apply_mma<32>, apply_mma_smem<32>());
      launch_clustered(k_apply_mma<32>, grid, 128, apply_mma_smem<32>(), lay.cluster, s, d_segs,
                       d_seg_off, nseg, k);
      break;
    default:
      ensure_smem((const void*)k_apply_mma<64>, apply_mma_smem<64>());
      launch_clustered(k_apply_mma<64>, grid, 128, apply_mma_smem<64>(), lay.cluster, s, d_segs,
                       d_seg_off, nseg, k);
  }
}

// ua(p, c) = src[p + c lds], zero on the index-0 planes; ub = 0. Tiles of 32 DOFs x 32
// right-hand sides, transposed through shared memory.
__global__ void __launch_bounds__(256) k_apply_in(const double* __restrict__ src, long long lds,
                                                  double* __restrict__ ua,
                                                  double* __restrict__ ub, int NC, int nrhs) {
  const long long n3 = (long long)NC * NC * NC;
  if (nrhs == 1) {
    const long long p = (long long)blockIdx.x * 256 + threadIdx.x;
    if (p >= n3) return;
    const int i = (int)(p % NC), j = (int)((p / NC) % NC), k = (int)(p / ((long long)NC * NC));
    ua[p] = (i == 0 || j == 0 || k == 0) ? 0.0 : src[p];
    ub[p] = 0.0;
    return;
  }
  __shared__ double tl[32][33];
  const long long p0 = (long long)blockIdx.x * 32;
  const int c0 = blockIdx.y * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long p = p0 + lane;
  const int i = (int)(p % NC), j = (int)((p / NC) % NC), k = (int)(p / ((long long)NC * NC));
  const bool in = p < n3 && i && j && k;
  for (int c = w; c < 32; c += 8)
    tl[c][lane] = (in && c0 + c < nrhs) ? src[p + (c0 + c) * lds] : 0.0;
  __syncthreads();
  for (int q = w; q < 32; q += 8)
    if (p0 + q < n3 && c0 + lane < nrhs) {
      ua[(p0 + q) * nrhs + c0 + lane] = tl[lane][q];
      ub[(p0 + q) * nrhs + c0 + lane] = 0.0;
    }
}

void launch_apply_in(const double* src, long long lds, double* ua, double* ub, int NC, int nrhs,
                     cudaStream_t s) {
  const long long n3 = (long long)NC * NC * NC;
  if (nrhs == 1) k_apply_in<<<(int)((n3 + 255) / 256), 256, 0, s>>>(src, lds, ua, ub, NC, 1);
  else
    k_apply_in<<<dim3((int)((n3 + 31) / 32), (nrhs + 31) / 32), 256, 0, s>>>(src, lds, ua, ub, NC,
                                                                            nrhs);
}

// dst[p + c ldd] = u(p, c)
__global__ void __launch_bounds__(256) k_apply_out(const double* __restrict__ u,
                                                   double* __restrict__ dst, long long ldd,
                                                   long long n3, int nrhs) {
  __shared__ double tl[32][33];
  const long long p0 = (long long)blockIdx.x * 32;
  const int c0 = blockIdx.y * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int q = w; q < 32; q += 8)
    tl[q][lane] = (p0 + q < n3 && c0 + lane < nrhs) ? u[(p0 + q) * nrhs + c0 + lane] : 0.0;
  __syncthreads();
  for (int c = w; c < 32; c += 8)
    if (p0 + lane < n3 && c0 + c < nrhs) dst[p0 + lane + (c0 + c) * ldd] = tl[lane][c];
}

void launch_apply_out(const double* u, double* dst, long long ldd, long long n3, int nrhs,
                      cudaStream_t s) {
  if (nrhs == 1) {
    cudaMemcpyAsync(dst, u, n3 * sizeof(double), cudaMemcpyDeviceToDevice, s);
    return;
  }
  k_apply_out<<<dim3((int)((n3 + 31) / 32), (nrhs + 31) / 32), 256, 0, s>>>(u, dst, ldd, n3, nrhs);
}

// u(dof[d], c) += alpha * sum over the DOF's slots in order; one segment per operator.
__global__ void __launch_bounds__(256) k_reduce_seg(const ReduceSeg* __restrict__ segs,
                                                    const int* __restrict__ seg_off, int nseg) {
  const int total = seg_off[nseg];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const int si = nseg == 1 ? 0 : find_desc(seg_off, nseg, t);
    const ReduceSeg sg = segs[si];
    const int e = t - seg_off[si], d = e / sg.nrhs, c = e - d * sg.nrhs;
    double sum = 0.0;
    const int q1 = sg.off[d + 1];
    for (int q = sg.off[d]; q < q1; ++q) sum += sg.contrib[(long long)sg.slot[q] * sg.nrhs + c];
    sg.u[(long long)sg.dof[d] * sg.nrhs + c] += sg.alpha * sum;
  }
}

void launch_reduce_seg(const ReduceSeg* d_segs, const int* d_seg_off, int nseg, int total,
                       cudaStream_t s) {
  if (total <= 0) return;
  const int blocks = std::min((total + 255) / 256, 4096);
  k_reduce_seg<<<blocks, 256, 0, s>>>(d_segs, d_seg_off, nseg);
}

__global__ void k_reduce_scatter(const int* __restrict__ dof, const int* __restrict__ off,
                                 const int* __restrict__ slot,
                                 const double* __restrict__ contrib, int ndof, double alpha,
                                 double* __restrict__ u, int nrhs) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)ndof * nrhs) return;
  const int d = (int)(t / nrhs), c = (int)(t - (long long)d * nrhs);
  double s = 0.0;
  const int q1 = off[d + 1];
  for (int q = off[d]; q < q1; ++q) s += contrib[(long long)slot[q] * nrhs + c];
  u[(long long)dof[d] * nrhs + c] += alpha * s;
}

void launch_reduce_scatter(const int* d_dof, const int* d_off, const int* d_slot,
                           const double* d_contrib, int ndof, double alpha, double* u, int nrhs,
                           cudaStream_t s) {
  const long long total = (long long)ndof * nrhs;
  if (total <= 0) return;
  k_reduce_scatter<<<(int)((total + 255) / 256), 256, 0, s>>>(d_dof, d_off, d_slot, d_contrib,
                                                             ndof, alpha, u, nrhs);
}

// ===========================================================================
// Operators: 7 bands over the NC^3 DOF grid, band b at band[b * NC^3 + p]:
// 0 diagonal, 1 (-i), 2 (+i), 3 (-j), 4 (+j), 5 (-k), 6 (+k). A band entry is
// zero where the neighbour is not a DOF (an index-0 plane or beyond N).
// ===========================================================================
__global__ void k_setup_node(const double* __restrict__ A, const double* __restrict__ V, int N,
                             double hh, double* __restrict__ band) {
  // SetupStencil, include/setup_stencil.hpp:34-69: entry (p, q) = -A(q)/h^2,
  // diagonal = sum of the six neighbours' A / h^2 + V(p). A, V are (NC+1)^3, i fastest.
  const int NC = N + 1, T = NC + 1;
  const long long n3 = (long long)NC * NC * NC;
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n3) return;
  const int i = (int)(p % NC), j = (int)((p / NC) % NC), k = (int)(p / ((long long)NC * NC));
  if (i == 0 || j == 0 || k == 0) {
    for (int b = 0; b < 7; ++b) band[b * n3 + p] = 0.0;
    return;
  }
  auto a = [&](int x, int y, int z) { return A[x + (long long)T * y + (long long)T * T * z]; };
  double dg = 0.0;
  dg += (a(i - 1, j, k) + a(i + 1, j, k)) / hh;
  dg += (a(i, j - 1, k) + a(i, j + 1, k)) / hh;
  dg += (a(i, j, k - 1) + a(i, j, k + 1)) / hh;
  dg += V[i + (long long)T * j + (long long)T * T * k];
  band[p] = dg;
  band[1 * n3 + p] = (i - 1 >= 1) ? -a(i - 1, j, k) / hh : 0.0;
  band[2 * n3 + p] = (i + 1 <= N) ? -a(i + 1, j, k) / hh : 0.0;
  band[3 * n3 + p] = (j - 1 >= 1) ? -a(i, j - 1, k) / hh : 0.0;
  band[4 * n3 + p] = (j + 1 <= N) ? -a(i, j + 1, k) / hh : 0.0;
  band[5 * n3 + p] = (k - 1 >= 1) ? -a(i, j, k - 1) / hh : 0.0;
  band[6 * n3 + p] = (k + 1 <= N) ? -a(i, j, k + 1) / hh : 0.0;
}

void launch_setup_node(const double* d_A, const double* d_V, int N, double h, double* d_band,
                       cudaStream_t s) {
  const long long n3 = (long long)(N + 1) * (N + 1) * (N + 1);
  k_setup_node<<<(int)((n3 + 255) / 256), 256, 0, s>>>(d_A, d_V, N, h * h, d_band);
}

__global__ void k_setup_faces(const double* __restrict__ ax, const double* __restrict__ ay,
                              const double* __restrict__ az, const double* __restrict__ V,
                              int N, double hh, double* __restrict__ band) {
  // Flux form: face coefficients ax(i,j,k) between (i,j,k) and (i+1,j,k), etc.,
  // on (NC+1)^3 arrays, i fastest. Symmetric by construction.
  const int NC = N + 1, T = NC + 1;
  const long long n3 = (long long)NC * NC * NC;
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n3) return;
  const int i = (int)(p % NC), j = (int)((p / NC) % NC), k = (int)(p / ((long long)NC * NC));
  if (i == 0 || j == 0 || k == 0) {
    for (int b = 0; b < 7; ++b) band[b * n3 + p] = 0.0;
    return;
  }
  auto at = [&](const double* F, int x, int y, int z) {
    return F[x + (long long)T * y + (long long)T * T * z];
  };
  const double xm = at(ax, i - 1, j, k), xp = at(ax, i, j, k);
  const double ym = at(ay, i, j - 1, k), yp = at(ay, i, j, k);
  const double zm = at(az, i, j, k - 1), zp = at(az, i, j, k);
  band[p] = (xm + xp + ym + yp + zm + zp) / hh + V[i + (long long)T * j + (long long)T * T * k];
  band[1 * n3 + p] = (i - 1 >= 1) ? -xm / hh : 0.0;
  band[2 * n3 + p] = (i + 1 <= N) ? -xp / hh : 0.0;
  band[3 * n3 + p] = (j - 1 >= 1) ? -ym / hh : 0.0;
  band[4 * n3 + p] = (j + 1 <= N) ? -yp / hh : 0.0;
  band[5 * n3 + p] = (k - 1 >= 1) ? -zm / hh : 0.0;
  band[6 * n3 + p] = (k + 1 <= N) ? -zp / hh : 0.0;
}

void launch_setup_faces(const double* d_ax, const double* d_ay, const double* d_az,
                        const double* d_V, int N, double h, double* d_band, cudaStream_t s) {
  const long long n3 = (long long)(N + 1) * (N + 1) * (N + 1);
  k_setup_faces<<<(int)((n3 + 255) / 256), 256, 0, s>>>(d_ax, d_ay, d_az, d_V, N, h * h,
                                                        d_band);
}

// y = A x (transpose = 0) or y = A^T x (transpose = 1, the reference's SpMV).
__global__ void k_stencil(const double* __restrict__ band, int NC, const double* __restrict__ x,
                          double* __restrict__ y, int nrhs, long long ldx, int transpose) {
  const long long n3 = (long long)NC * NC * NC;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n3 * nrhs) return;
  const long long p = t % n3;
  const int c = (int)(t / n3);
  const double* xc = x + c * ldx;
  const long long off[7] = {0, -1, 1, -(long long)NC, (long long)NC, -(long long)NC * NC,
                            (long long)NC * NC};
  const int rev[7] = {0, 2, 1, 4, 3, 6, 5};
  double s = 0.0;
  if (transpose == 0) {
    s = band[p] * xc[p];
#pragma unroll
    for (int b = 1; b < 7; ++b) {
      const double a = band[b * n3 + p];
      if (a != 0.0) s = fma(a, xc[p + off[b]], s);
    }
  } else {
    s = band[p] * xc[p];
#pragma unroll
    for (int b = 1; b < 7; ++b) {
      // (A^T)(p, q) = A(q, p) with q = p + off[b]: the band of q pointing back to p
      const long long q = p + off[b];
      if (q < 0 || q >= n3) continue;
      const double a = band[rev[b] * n3 + q];
      if (a != 0.0) s = fma(a, xc[q], s);
    }
  }
  y[p + c * ldx] = s;
}

void launch_stencil_apply(const double* d_band, int NC, const double* x, double* y, int nrhs,
                          long long ldx, int transpose, cudaStream_t s) {
  const long long total = (long long)NC * NC * NC * nrhs;
  k_stencil<<<(int)((total + 255) / 256), 256, 0, s>>>(d_band, NC, x, y, nrhs, ldx, transpose);
}

__global__ void k_zero_boundary(double* __restrict__ u, int NC, int nrhs, long long ldu) {
  const long long n3 = (long long)NC * NC * NC;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n3 * nrhs) return;
  const long long p = t % n3;
  const int c = (int)(t / n3);
  const int i = (int)(p % NC), j = (int)((p / NC) % NC), k = (int)(p / ((long long)NC * NC));
  if (i == 0 || j == 0 || k == 0) u[p + c * ldu] = 0.0;
}

void launch_zero_boundary(double* u, int NC, int nrhs, long long ldu, cudaStream_t s) {
  const long long total = (long long)NC * NC * NC * nrhs;
  k_zero_boundary<<<(int)((total + 255) / 256), 256, 0, s>>>(u, NC, nrhs, ldu);
}


// ---- deterministic dot products: fixed grid, fixed-order final sum --------
__global__ void __launch_bounds__(256) k_dot_partial(const double* __restrict__ x,
                                                     const double* __restrict__ y, long long n,
                                                     long long ld, double* __restrict__ part) {
  const int c = blockIdx.y;
  const double* xc = x + c * ld;
  const double* yc = y + c * ld;
  double s = 0.0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    s = fma(xc[t], yc[t], s);
  __shared__ double sc[40];
  s = block_sum(s, sc);
  if (threadIdx.x == 0) part[c * gridDim.x + blockIdx.x] = s;
}

__global__ void k_dot_final(const double* __restrict__ part, int nparts,
                            double* __restrict__ out) {
  const int c = blockIdx.x;
  __shared__ double sc[40];
  double s = 0.0;
  for (int t = threadIdx.x; t < nparts; t += blockDim.x) s += part[c * nparts + t];
  s = block_sum(s, sc);
  if (threadIdx.x == 0) out[c] = s;
}

void launch_dot(const double* x, const double* y, long long n, int nrhs, long long ld,
                double* d_partial, double* d_out, cudaStream_t s) {
  dim3 grid(kDotBlocks, nrhs);
  k_dot_partial<<<grid, 256, 0, s>>>(x, y, n, ld, d_partial);
  k_dot_final<<<nrhs, 256, 0, s>>>(d_partial, kDotBlocks, d_out);
}

__global__ void k_pcg_xr(double* __restrict__ x, double* __restrict__ r,
                         const double* __restrict__ p, const double* __restrict__ q,
                         const double* __restrict__ rz, const double* __restrict__ pq,
                         long long n, int nrhs, long long ld) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * nrhs) return;
  const long long i = t % n;
  const int c = (int)(t / n);
  const double den = pq[c];
  const double a = (den != 0.0) ? rz[c] / den : 0.0;
  x[i + c * ld] = fma(a, p[i + c * ld], x[i + c * ld]);
  r[i + c * ld] = fma(-a, q[i + c * ld], r[i + c * ld]);
}

void launch_pcg_update_xr(double* x, double* r, const double* p, const double* q,
                          const double* rz, const double* pq, long long n, int nrhs,
                          long long ld, cudaStream_t s) {
  const long long total = n * nrhs;
  k_pcg_xr<<<(int)((total + 255) / 256), 256, 0, s>>>(x, r, p, q, rz, pq, n, nrhs, ld);
}

__global__ void k_pcg_p(double* __restrict__ p, const double* __restrict__ z,
                        const double* __restrict__ rz_new, const double* __restrict__ rz_old,
                        long long n, int nrhs, long long ld) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * nrhs) return;
  const long long i = t % n;
  const int c = (int)(t / n);
  const double den = rz_old[c];
  const double b = (den != 0.0) ? rz_new[c] / den : 0.0;
  p[i + c * ld] = fma(b, p[i + c * ld], z[i + c * ld]);
}

void launch_pcg_update_p(double* p, const double* z, const double* rz_new,
                         const double* rz_old, long long n, int nrhs, long long ld,
                         cudaStream_t s) {
  const long long total = n * nrhs;
  k_pcg_p<<<(int)((total + 255) / 256), 256, 0, s>>>(p, z, rz_new, rz_old, n, nrhs, ld);
}

// ---------------------------------------------------------------------------
// GMRES vector kernels. A Krylov basis of nb vectors per right-hand side is
// stored as V[(i * nrhs + c) * n + t] (vector i of column c); coefficient
// arrays as coef[i * nrhs + c]. Reductions run in a fixed order (per block,
// then over the kDotBlocks partials), so results are bit-reproducible.
// ---------------------------------------------------------------------------

// partial dots of w against basis vectors i0 .. i0 + nb - 1 (nb <= kGmresGroup):
// part[(q * nrhs + c) * gridDim.x + block]
__global__ void __launch_bounds__(256) k_gmres_dots(const double* __restrict__ V, int i0, int nb,
                                                    const double* __restrict__ w, long long n,
                                                    int nrhs, double* __restrict__ part) {
  const int c = blockIdx.y;
  const double* wc = w + (long long)c * n;
  double acc[kGmresGroup];
#pragma unroll
  for (int q = 0; q < kGmresGroup; ++q) acc[q] = 0.0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const double wv = wc[t];
#pragma unroll
    for (int q = 0; q < kGmresGroup; ++q)
      if (q < nb) acc[q] = fma(V[((long long)(i0 + q) * nrhs + c) * n + t], wv, acc[q]);
  }
  __shared__ double sc[40];
#pragma unroll
  for (int q = 0; q < kGmresGroup; ++q) {
    if (q < nb) {  // nb is the same for the whole block: the barriers inside match
      const double tot = block_sum(acc[q], sc);
      if (threadIdx.x == 0) part[((long long)q * nrhs + c) * gridDim.x + blockIdx.x] = tot;
    }
  }
}

void launch_gmres_dots(const double* V, int nb, const double* w, long long n, int nrhs,
                       double* d_partial, double* d_out, cudaStream_t s) {
  for (int i0 = 0; i0 < nb; i0 += kGmresGroup) {
    const int g = nb - i0 < kGmresGroup ? nb - i0 : kGmresGroup;
    k_gmres_dots<<<dim3(kDotBlocks, nrhs), 256, 0, s>>>(V, i0, g, w, n, nrhs, d_partial);
    k_dot_final<<<g * nrhs, 256, 0, s>>>(d_partial, kDotBlocks, d_out + (long long)i0 * nrhs);
  }
}

// w[:, c] += sign * sum_{i < nb} coef[i * nrhs + c] V_i[:, c]
__global__ void __launch_bounds__(256) k_gmres_axpy(double* __restrict__ w,
                                                    const double* __restrict__ V, int nb,
                                                    const double* __restrict__ coef, double sign,
                                                    long long n, int nrhs) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  if (t >= n) return;
  double acc = 0.0;
  for (int i = 0; i < nb; ++i)
    acc = fma(coef[(long long)i * nrhs + c], V[((long long)i * nrhs + c) * n + t], acc);
  w[(long long)c * n + t] = fma(sign, acc, w[(long long)c * n + t]);
}

void launch_gmres_axpy(double* w, const double* V, int nb, const double* coef, double sign,
                       long long n, int nrhs, cudaStream_t s) {
  if (nb <= 0) return;
  k_gmres_axpy<<<dim3((unsigned)((n + 255) / 256), nrhs), 256, 0, s>>>(w, V, nb, coef, sign, n,
                                                                       nrhs);
}

// dst[:, c] = scale[c] * src[:, c]
__global__ void __launch_bounds__(256) k_gmres_scale(double* __restrict__ dst,
                                                     const double* __restrict__ src,
                                                     const double* __restrict__ scale,
                                                     long long n) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  if (t >= n) return;
  dst[(long long)c * n + t] = scale[c] * src[(long long)c * n + t];
}

void launch_gmres_scale(double* dst, const double* src, const double* scale, long long n, int nrhs,
                        cudaStream_t s) {
  k_gmres_scale<<<dim3((unsigned)((n + 255) / 256), nrhs), 256, 0, s>>>(dst, src, scale, n);
}

}  // namespace hif
