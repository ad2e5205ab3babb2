// gemm_f64.cu -- FP64 contraction on the DMMA tensor-core path
// (mma.sync .f64): the plain-FP64 path of the engine and the arithmetic of the
// reference's XGEMM -> DGEMM (tools/xgemm.F:10-49).
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "gemm.cuh"

namespace acesb200 {

namespace {
// ---------------------------------------------------------------------------
// k_gemm_f64: C = alpha * sum_s A_s B_s^T + beta * C over up to 4 K segments.
//
// A block computes one BM x BN tile (or one split-K slice of it) of one task;
// a launch is a single task passed by value, or a device table of tasks.  The
// k tiles (16 doubles, one 128-byte row per operand row) of all segments form
// one sequence through a 4-stage cp.async pipeline.  Rows lie unpadded in
// shared memory with the 16-byte chunk index XORed by twice the row's index
// modulo 4: the 16 lanes of a 64-bit load phase (four neighbouring rows x four
// k) then cover all 32 banks, and so do the copies (one row per 8 lanes).
//
// Every output of an unsplit product, and every slice of a split one, sums its k
// in ascending order.  (Split K regroups the sums by slice, k_gemm_tiny_f64 by
// lane.)  One 128-bit load per row and k step, with the k taken as 0, 2, 4, 6, 1,
// 3, 5, 7, is 1-2 % faster (the call of 2401 x 1519 x 2049, N/N: 601 us against
// 612), but its other last bits move values across the rounding boundaries of
// the BF16 split: a CCSD with o = 24, v = 220 in split precision, whose lists
// are unsplit products, then differed by up to 1e-9, and by 1e-17 with their
// sums in order.
// ---------------------------------------------------------------------------
constexpr int BK = 16, kStages = 4;

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

template <int VEC>
__device__ __forceinline__ void cp_async(unsigned dst, const double *src, bool valid) {
  int sz = valid ? VEC * 8 : 0;
  if (VEC == 2)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(sz));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(sz));
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// c (16 x 8) += a (16 x 8) b (8 x 8)^T: a = rows g and g+8 x k (t, t+4)
__device__ __forceinline__ void dmma(double (&c)[4], const double2 &a0, const double2 &a1,
                                     const double2 &b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0.x), "d"(a1.x), "d"(a0.y), "d"(a1.y), "d"(b.x), "d"(b.y));
}

// Tile shape: BM x BN, WR x WC warps, OCC blocks per SM the registers allow for
template <int BM_, int BN_, int WR_, int WC_, int OCC_>
struct TileF64 {
  static constexpr int BM = BM_, BN = BN_, WR = WR_, WC = WC_, OCC = OCC_;
  static constexpr int kThreads = 32 * WR * WC;
  static constexpr int TM = BM / WR, TN = BN / WC, MI = TM / 16, NI = TN / 8;
  static constexpr int kStageBytes = (BM + BN) * BK * 8;
  static constexpr int kSmem = kStages * kStageBytes;
  static_assert(TM % 16 == 0 && TN % 8 == 0, "warp tile of 16 x 8 products");
  static_assert(kSmem * OCC <= 225 * 1024, "shared memory");
};

// The copies of one operand tile (ROWS x BK doubles) in VEC-double chunks:
// thread t always takes the chunks of k offset kc in rows r0 + i * RS.
template <int ROWS, int kThreads, int VEC>
struct CopyPlan {
  static constexpr int CPR = BK / VEC;
  static constexpr int RS = kThreads / CPR;
  static constexpr int kPer = (ROWS + RS - 1) / RS;
  static_assert(RS % 4 == 0, "a thread's rows share their swizzle");
  const double *base;   // &X[row0 + r0][kc] of the current segment
  const double *safe;   // any valid address (the source of zero-size copies)
  long long step;       // RS rows
  unsigned live;        // bit i: row r0 + i RS inside the operand and the tile
  int kc, soff;         // k offset; byte offset of chunk 0 inside the stage's tile
  __device__ __forceinline__ void init(int rows, int row0) {
    const int t = threadIdx.x, r0 = t / CPR;
    kc = (t % CPR) * VEC;
    const int ch = (kc >> 1) ^ ((r0 & 3) << 1);
    soff = (r0 * BK + ch * 2 + (kc & 1)) * 8;
    live = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      live |= (r0 + i * RS < ROWS && row0 + r0 + i * RS < rows) ? 1u << i : 0u;
  }
  __device__ __forceinline__ void segment(const double *X, long long ld, int row0) {
    safe = X;
    base = X + (long long)(row0 + (int)threadIdx.x / CPR) * ld + kc;
    step = (long long)RS * ld;
  }
  __device__ __forceinline__ void issue(unsigned tile, int k0, int K) const {
    const bool kok = k0 + kc < K;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      if (ROWS % RS != 0 && i == kPer - 1 && (int)threadIdx.x / CPR + i * RS >= ROWS) break;
      const bool v = kok && ((live >> i) & 1u);
      cp_async<VEC>(tile + soff + i * RS * BK * 8, v ? base + i * step + k0 : safe, v);
    }
  }
};

__host__ __device__ __forceinline__ int f64_ktiles(const F64Task &T) {
  int n = 0;
  for (int s = 0; s < T.nseg; ++s) n += (T.seg[s].K + BK - 1) / BK;
  return n;
}
// output tiles of a task
__host__ __device__ __forceinline__ int f64_tiles(int M, int N, int tri, int BM, int BN) {
  const int tm = (M + BM - 1) / BM, tn = (N + BN - 1) / BN;
  return tri ? tm * (tm + 1) / 2 : tm * tn;
}

struct F64Launch {
  F64Task one;            // the task when table is null
  const F64Task *table;   // device table of ntask tasks
  int ntask;
  int per_task;           // tiles per task when all have the same shape, else 0
  int kchunk;             // k tiles per split-K slice (blockIdx.y), 0: no split
  double alpha, beta;
  double *part;           // split-K partials [z][M][N]
};

template <class T, int VEC>
__global__ void __launch_bounds__(T::kThreads, T::OCC)
    k_gemm_f64(const __grid_constant__ F64Launch L) {
  after_previous();
  constexpr int BM = T::BM, BN = T::BN, MI = T::MI, NI = T::NI;
  extern __shared__ __align__(128) unsigned char f64_smem[];
  int t = blockIdx.x;
  const F64Task *tk = &L.one;
  if (L.table) {
    int i = 0;
    if (L.per_task) {
      i = t / L.per_task;
      t -= i * L.per_task;
    } else {
      while (i + 1 < L.ntask && t >= L.table[i + 1].tile0) ++i;
      t -= L.table[i].tile0;
    }
    tk = L.table + i;
  }
  const int M = tk->M, N = tk->N, tri = tk->tri;
  int tm, tn;
  if (tri) {  // lower triangle of square tiles, row by row
    tm = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while (tm * (tm + 1) / 2 > t) --tm;
    while ((tm + 1) * (tm + 2) / 2 <= t) ++tm;
    tn = t - tm * (tm + 1) / 2;
  } else {
    // bands of 8 m tiles, m fastest inside a band: the tiles running together
    // share few rows of both operands
    const int tilesM = (M + BM - 1) / BM, tilesN = (N + BN - 1) / BN;
    const int g = t / (8 * tilesN), r = t - g * 8 * tilesN, gm = min(8, tilesM - g * 8);
    tm = g * 8 + r % gm;
    tn = r / gm;
  }
  const int m0 = tm * BM, n0 = tn * BN;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp / T::WC, wn = warp % T::WC;
  const int g = lane >> 2, q = lane & 3;

  const int nkt = f64_ktiles(*tk);
  const int kb = L.kchunk ? (int)blockIdx.y * L.kchunk : 0;
  const int ke = L.kchunk ? min(nkt, kb + L.kchunk) : nkt;
  const int nk = max(0, ke - kb);

  CopyPlan<BM, T::kThreads, VEC> pa;
  CopyPlan<BN, T::kThreads, VEC> pb;
  pa.init(M, m0);
  pb.init(N, n0);
  // segment of the next k tile to issue, its K and the k offset inside it
  int sg = 0, segK = 0, kin = kb * BK;
  auto enter = [&]() {
    segK = tk->seg[sg].K;
    pa.segment(tk->seg[sg].A, tk->seg[sg].lda, m0);
    pb.segment(tk->seg[sg].B, tk->seg[sg].ldb, n0);
  };
  if (nk > 0) {
    while (sg + 1 < tk->nseg && kin >= (tk->seg[sg].K + BK - 1) / BK * BK) {
      kin -= (tk->seg[sg].K + BK - 1) / BK * BK;
      ++sg;
    }
    enter();
  }
  const unsigned sbase = smem_u32(f64_smem);
  int issued = 0, slot_w = 0;
  auto issue_next = [&]() {
    if (issued < nk) {
      if (kin >= segK) {  // the previous segment is done
        ++sg;
        kin = 0;
        enter();
      }
      const unsigned st = sbase + slot_w * T::kStageBytes;
      pa.issue(st, kin, segK);
      pb.issue(st + BM * BK * 8, kin, segK);
      kin += BK;
      ++issued;
      slot_w = slot_w + 1 == kStages ? 0 : slot_w + 1;
    }
    cp_commit();
  };

  double acc[MI][NI][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int h = 0; h < 4; ++h) acc[i][j][h] = 0.0;

#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) issue_next();
  // offsets of a row's k = q and k = q + 4 within a k step of 8
  const int sw = (g & 3) << 1;
  int slot = 0;
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<kStages - 2>();   // k tile kt has landed
    __syncthreads();
    issue_next();             // into the slot every thread left before the barrier
    const unsigned char *st = f64_smem + slot * T::kStageBytes;
    slot = slot + 1 == kStages ? 0 : slot + 1;
    const double *a_s = reinterpret_cast<const double *>(st) + (wm * T::TM + g) * BK;
    const double *b_s = reinterpret_cast<const double *>(st) + (BM + wn * T::TN + g) * BK;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int k0 = ((s * 4 + (q >> 1)) ^ sw) * 2 + (q & 1);
      const int k4 = ((s * 4 + 2 + (q >> 1)) ^ sw) * 2 + (q & 1);
      double2 af[MI][2], bf[NI];
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double *r = a_s + (i * 16 + h * 8) * BK;
          af[i][h] = make_double2(r[k0], r[k4]);
        }
#pragma unroll
      for (int j = 0; j < NI; ++j)
        bf[j] = make_double2(b_s[j * 8 * BK + k0], b_s[j * 8 * BK + k4]);
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) dmma(acc[i][j], af[i][0], af[i][1], bf[j]);
    }
  }
  cp_wait<0>();

  if (L.part) {  // split-K partial: dense [z][M][N]
    double *pz = L.part + (size_t)blockIdx.y * M * N;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = m0 + wm * T::TM + i * 16 + h * 8 + g;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int n = n0 + wn * T::TN + j * 8 + q * 2 + e;
            if (n < N) pz[(size_t)m * N + n] = acc[i][j][2 * h + e];
          }
      }
    return;
  }
  // epilogue through the two-level output view; the beta*C loads of a row
  // are issued together before its stores
  const CView C = tk->C;
  const double alpha = L.alpha, beta = L.beta;
  const bool mirror = tri && tm != tn;
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = m0 + wm * T::TM + i * 16 + h * 8 + g;
      if (m >= M) continue;
      const long long mo = cview_dim(C.mdiv, C.sm1, C.sm0, m);
      double old[NI][2];
      if (beta != 0.0) {
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int n = n0 + wn * T::TN + j * 8 + q * 2 + e;
            old[j][e] = n < N ? __ldg(C.p + mo + cview_dim(C.ndiv, C.sn1, C.sn0, n)) : 0.0;
          }
      }
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int n = n0 + wn * T::TN + j * 8 + q * 2 + e;
          if (n >= N) continue;
          double r = alpha * acc[i][j][2 * h + e];
          if (beta != 0.0) r += beta * old[j][e];
          C.p[mo + cview_dim(C.ndiv, C.sn1, C.sn0, n)] = r;
          if (mirror)
            C.p[cview_dim(C.mdiv, C.sm1, C.sm0, n) + cview_dim(C.ndiv, C.sn1, C.sn0, m)] = r;
        }
    }
}

// launch of one tile shape; the shared-memory opt-in is per device
template <class T, int VEC>
int launch_tile(const F64Launch &L, unsigned tiles, unsigned z, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  ACES_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("gemm_nt_f64: device %d outside 0..63", dev);
    return ACES_ERR_ARG;
  }
  if (!attr_set[dev]) {
    ACES_CUDA(cudaFuncSetAttribute(k_gemm_f64<T, VEC>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmem));
    attr_set[dev] = true;
  }
  launch_after(k_gemm_f64<T, VEC>, dim3(tiles, z), T::kThreads, T::kSmem, st, L);
  count_launch();
  ACES_CUDA(cudaGetLastError());
  return ACES_OK;
}
}  // namespace

// C = alpha * sum_z part[z] + beta * C
// part[z][m][n] (mfast false) or part[z][n][m] (mfast true); the slices are
// summed in order z = 0, 1, ... with four of them loaded at a time.  Wide =
// false: M * N below 2^31, the index split with FastDiv (fd: M if mfast, else N).
template <bool Wide>
__global__ void k_splitk_reduce(CView C, const double *__restrict__ part, int M, int N, int Z,
                                double alpha, double beta, bool mfast, FastDiv fd) {
  after_previous();
  const long long total = (long long)M * N;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    int m, n;
    if (Wide) {
      m = mfast ? (int)(idx % M) : (int)(idx / N);
      n = mfast ? (int)(idx / M) : (int)(idx % N);
    } else {
      const unsigned q = fd.div((unsigned)idx), r = (unsigned)idx - q * fd.d;
      m = mfast ? (int)r : (int)q;
      n = mfast ? (int)q : (int)r;
    }
    const double *pz = part + idx;
    double s = 0.0;
    int z = 0;
    for (; z + 4 <= Z; z += 4) {
      const double a0 = __ldg(pz), a1 = __ldg(pz + total), a2 = __ldg(pz + 2 * total),
                   a3 = __ldg(pz + 3 * total);
      s += a0;
      s += a1;
      s += a2;
      s += a3;
      pz += 4 * total;
    }
    for (; z < Z; ++z, pz += total) s += __ldg(pz);
    double *cp = C.p + cview_off(C, m, n);
    double r = alpha * s;
    if (beta != 0.0) r += beta * *cp;
    *cp = r;
  }
}

// y[m] = alpha * sum_k A[m*lda + k] x[k] + beta * y[m]; one warp per row
__global__ void k_gemv_f64(int M, int K, double alpha, const double *__restrict__ A,
                           long long lda, const double *__restrict__ x, double beta, CView C,
                           bool transpose_out) {
  after_previous();
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int m = warp; m < M; m += nwarps) {
    const double *a = A + (long long)m * lda;
    // four independent partial sums keep four row loads in flight per lane
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int k = lane;
    for (; k + 96 < K; k += 128) {
      s0 += a[k] * __ldg(x + k);
      s1 += a[k + 32] * __ldg(x + k + 32);
      s2 += a[k + 64] * __ldg(x + k + 64);
      s3 += a[k + 96] * __ldg(x + k + 96);
    }
    for (; k < K; k += 32) s0 += a[k] * __ldg(x + k);
    double s = (s0 + s1) + (s2 + s3);
    for (int off = 16; off; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) {
      int mm = transpose_out ? 0 : m, nn = transpose_out ? m : 0;
      double *cp = C.p + cview_off(C, mm, nn);
      double r = alpha * s;
      if (beta != 0.0) r += beta * *cp;
      *cp = r;
    }
  }
}

// Partial row sums for products with few rows: warp w takes row w / W and
// the w % W-th K chunk of it (kc elements, a multiple of 128); the partials
// go to part[row * W + chunk].
__global__ void k_gemv_part(int M, int K, int W, int kc, const double *__restrict__ A,
                            long long lda, const double *__restrict__ x,
                            double *__restrict__ part) {
  after_previous();
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= (long long)M * W) return;  // warp-uniform
  const int m = (int)(warp / W), c = (int)(warp - (long long)m * W);
  const int k0 = c * kc, k1 = min(K, k0 + kc);
  const double *a = A + (long long)m * lda;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  int k = k0 + lane;
  for (; k + 96 < k1; k += 128) {
    s0 += a[k] * __ldg(x + k);
    s1 += a[k + 32] * __ldg(x + k + 32);
    s2 += a[k + 64] * __ldg(x + k + 64);
    s3 += a[k + 96] * __ldg(x + k + 96);
  }
  for (; k < k1; k += 32) s0 += a[k] * __ldg(x + k);
  double t = (s0 + s1) + (s2 + s3);
  for (int off = 16; off; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
  if (lane == 0) part[warp] = t;
}

// y[m] = alpha * sum_c part[m * W + c] + beta * y[m], the chunks summed in order
__global__ void k_gemv_final(int M, int W, double alpha, const double *__restrict__ part,
                             double beta, CView C, bool transpose_out) {
  after_previous();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  double t = 0.0;
  for (int c = 0; c < W; ++c) t += part[(long long)m * W + c];
  const int mm = transpose_out ? 0 : m, nn = transpose_out ? m : 0;
  double *cp = C.p + cview_off(C, mm, nn);
  double r = alpha * t;
  if (beta != 0.0) r += beta * *cp;
  *cp = r;
}

// Tiny products (at most kTinyOut outputs): one warp per output, its lanes
// striding K (coalesced row reads) with the sixteen loads of a 256-wide step in
// flight, the ragged last step included (latency bound: with eight and a serial
// remainder 50 x 50 x 1800 took 7.6 us; the 280 launches of an EOM with o = 6,
// v = 50 now take 3.8 us each).  Four partial sums per lane take the k of each
// full 128 in turn, the first one what is left over; shuffles add them in a
// fixed order.
constexpr long long kTinyOut = 8192;
__global__ void k_gemm_tiny_f64(int M, int N, int K, double alpha, const double *__restrict__ A,
                                long long lda, const double *__restrict__ B, long long ldb,
                                double beta, CView C) {
  after_previous();
  const int w = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= M * N) return;  // warp-uniform
  const int m = w % M, n = w / M;
  const double *a = A + (long long)m * lda, *b = B + (long long)n * ldb;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  for (int k0 = lane; k0 < K; k0 += 256) {
    double x[8], y[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + 32 * u;
      x[u] = k < K ? __ldg(a + k) : 0.0;
      y[u] = k < K ? __ldg(b + k) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; u += 4) {
      const bool full = k0 + 32 * u + 96 < K;
      s0 = fma(x[u], y[u], s0);
      if (full) {
        s1 = fma(x[u + 1], y[u + 1], s1);
        s2 = fma(x[u + 2], y[u + 2], s2);
        s3 = fma(x[u + 3], y[u + 3], s3);
      } else {
        s0 = fma(x[u + 1], y[u + 1], s0);
        s0 = fma(x[u + 2], y[u + 2], s0);
      }
    }
  }
  double t = (s0 + s1) + (s2 + s3);
  for (int off = 16; off; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
  if (lane == 0) {
    double *cp = C.p + cview_off(C, m, n);
    double r = alpha * t;
    if (beta != 0.0) r += beta * *cp;
    *cp = r;
  }
}

// Split-K reduction with many slices and few outputs: one warp per output,
// lane k adds slices k, k+32, ..., then a fixed shuffle tree (deterministic).
// part[z][m][n], or part[z][n][m] with mfast.
__global__ void k_reduce_warp(CView C, const double *__restrict__ part, int M, int N, int Z,
                              double alpha, double beta, bool mfast) {
  after_previous();
  const long long total = (long long)M * N;
  const int lane = threadIdx.x & 31;
  for (long long idx = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; idx < total;
       idx += ((long long)gridDim.x * blockDim.x) >> 5) {
    double sum = 0.0;
    for (int z = lane; z < Z; z += 32) sum += part[(size_t)z * total + idx];
    for (int off = 16; off; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
    if (lane == 0) {
      const int m = mfast ? (int)(idx % M) : (int)(idx / N);
      const int n = mfast ? (int)(idx / M) : (int)(idx % N);
      double *cp = C.p + cview_off(C, m, n);
      double v = alpha * sum;
      if (beta != 0.0) v += beta * *cp;
      *cp = v;
    }
  }
}

static void launch_reduce_warp(const CView &C, const double *part, int M, int N, int Z,
                               double alpha, double beta, bool mfast, cudaStream_t st) {
  const long long total = (long long)M * N;
  long long nb = (total + 7) / 8;  // 8 warps per block
  if (nb > 148 * 32) nb = 148 * 32;
  launch_after(k_reduce_warp, (unsigned)nb, 256, 0, st, C, part, M, N, Z, alpha, beta, mfast);
  count_launch();
}

// ---------------------------------------------------------------------------
// Low-rank updates (K <= 32): C(m,n) = alpha sum_k A[m,k] B[n,k] + beta C(m,n).
// Output bound.  A block owns 128 outputs along the "fast" index (the one with
// unit stride in the view, so the update of C coalesces) x 32 along the other.
// Both short operands are staged in shared memory with an odd row stride; each
// thread runs 8 independent FMA chains (one per slow index) over k, then
// updates its 8 outputs: one RED per element for beta = 1 on a coalesced view
// (a single owner per element, so the sum equals load + add + store), else a
// batched read-modify-write.
// ---------------------------------------------------------------------------
constexpr int LR_F = 128, LR_S = 32, LR_K = 32;

__global__ void __launch_bounds__(LR_F)
    k_gemm_lowrank_f64(int M, int N, int K, double alpha, const double *__restrict__ A,
                       long long lda, const double *__restrict__ B, long long ldb, double beta,
                       CView C, bool fast_is_m, int tiles_f) {
  after_previous();
  extern __shared__ double lr_smem[];
  const int ks = K | 1;  // odd row stride: column reads across threads are conflict free
  double *Fs = lr_smem;              // [LR_F][ks]
  double *Ss = lr_smem + LR_F * ks;  // [LR_S][ks]
  const int nf = fast_is_m ? M : N, ns = fast_is_m ? N : M;
  const double *Fp = fast_is_m ? A : B;
  const double *Sp = fast_is_m ? B : A;
  const long long ldf = fast_is_m ? lda : ldb, lds = fast_is_m ? ldb : lda;
  const int f0 = (blockIdx.x % tiles_f) * LR_F;
  const int s0 = (blockIdx.x / tiles_f) * LR_S;
  for (int e = threadIdx.x; e < LR_F * K; e += LR_F) {
    const int rr = e / K, kk = e - rr * K;
    Fs[rr * ks + kk] = f0 + rr < nf ? Fp[(long long)(f0 + rr) * ldf + kk] : 0.0;
  }
  for (int e = threadIdx.x; e < LR_S * K; e += LR_F) {
    const int rr = e / K, kk = e - rr * K;
    Ss[rr * ks + kk] = s0 + rr < ns ? Sp[(long long)(s0 + rr) * lds + kk] : 0.0;
  }
  __syncthreads();
  const int f = f0 + threadIdx.x;
  if (f >= nf) return;
  const int nsl = min(LR_S, ns - s0);
  // fast and slow view dimensions
  const long long fdiv = fast_is_m ? C.mdiv : C.ndiv, fs1 = fast_is_m ? C.sm1 : C.sn1,
                  fs0 = fast_is_m ? C.sm0 : C.sn0;
  const long long sdiv = fast_is_m ? C.ndiv : C.mdiv, ss1 = fast_is_m ? C.sn1 : C.sm1,
                  ss0 = fast_is_m ? C.sn0 : C.sm0;
  double *const cf = C.p + cview_dim(fdiv, fs1, fs0, f);
  ViewWalk w(sdiv, ss1, ss0, s0);
#ifndef ACES_LR_RED
#define ACES_LR_RED 1
#endif
  const bool red = ACES_LR_RED && beta == 1.0 && fs0 == 1;
  const double *fr = Fs + threadIdx.x * ks;
#pragma unroll 1
  for (int sb = 0; sb < nsl; sb += 8) {
    double acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.0;
    const double *sr = Ss + sb * ks;  // rows sb..sb+7 < LR_S (zero past ns)
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
      const double fv = fr[k];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = fma(fv, sr[j * ks + k], acc[j]);
    }
    long long off[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      acc[j] *= alpha;
      off[j] = w.off;
      w.next();
    }
    if (beta == 0.0) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (sb + j < nsl) cf[off[j]] = acc[j];
    } else if (red) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (sb + j < nsl) atomicAdd(cf + off[j], acc[j]);
    } else {
      double old[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) old[j] = sb + j < nsl ? __ldg(cf + off[j]) : 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (sb + j < nsl) cf[off[j]] = acc[j] + beta * old[j];
    }
  }
}

static int launch_lowrank(int M, int N, int K, double alpha, const double *A, long long lda,
                          const double *B, long long ldb, double beta, const CView &C,
                          cudaStream_t st) {
  // run threads along the unit-stride output index
  const bool fast_is_m = C.sm0 == 1 || C.sn0 != 1;
  const int nf = fast_is_m ? M : N, ns = fast_is_m ? N : M;
  const int tiles_f = (nf + LR_F - 1) / LR_F;
  const long long nb = (long long)tiles_f * ((ns + LR_S - 1) / LR_S);
  if (nb > 0x7fffffffLL) {
    set_error("low-rank contraction grid too large (%lld blocks)", nb);
    return ACES_ERR_ARG;
  }
  const size_t smem = (size_t)(LR_F + LR_S) * (K | 1) * sizeof(double);
  launch_after(k_gemm_lowrank_f64, (unsigned)nb, LR_F, smem, st, M, N, K, alpha, A, lda, B, ldb,
               beta, C, fast_is_m, tiles_f);
  count_launch();
  ACES_CUDA(cudaGetLastError());
  return ACES_OK;
}

// split-K partials: the running call's workspace, which its products use in
// turn on one stream
double *splitk_workspace(size_t doubles) {
  return static_cast<double *>(call_workspace(doubles * sizeof(double)));
}

int splitk_reduce(const CView &C, const double *part, int M, int N, int Z, double alpha,
                  double beta, cudaStream_t st, bool mfast) {
  long long total = (long long)M * N;
  if (Z >= 24 && total <= 16384) {
    // few outputs, many slices: a warp per output instead of a serial loop
    launch_reduce_warp(C, part, M, N, Z, alpha, beta, mfast, st);
    ACES_CUDA(cudaGetLastError());
    return ACES_OK;
  }
  long long nb = (total + 255) / 256;
  if (nb > 148 * 16) nb = 148 * 16;
  const FastDiv fd((unsigned)std::max(1, mfast ? M : N));
  if (total < (1LL << 31))
    launch_after(k_splitk_reduce<false>, (unsigned)nb, 256, 0, st, C, part, M, N, Z, alpha, beta,
                 mfast, fd);
  else
    launch_after(k_splitk_reduce<true>, (unsigned)nb, 256, 0, st, C, part, M, N, Z, alpha, beta,
                 mfast, fd);
  count_launch();
  ACES_CUDA(cudaGetLastError());
  return ACES_OK;
}

int gemv_f64(int M, int K, double alpha, const double *A, long long lda, const double *x,
             double beta, const CView &C, bool transpose_out, cudaStream_t st) {
  if (M <= 0) return ACES_OK;
  // few rows: each row split over W warps (about 4736 warps in all, K chunks
  // of at least 128), so the matrix streams with enough loads in flight
  const long long kTargetWarps = 148 * 32;
  if (M <= kTargetWarps && K >= 256) {
    int W = (int)std::min<long long>(32, (kTargetWarps + M - 1) / M);
    int kc = ((K + W - 1) / W + 127) / 128 * 128;
    W = (K + kc - 1) / kc;
    if (W > 1) {
      double *part = splitk_workspace((size_t)M * W);
      if (!part) {
        set_error("gemv: partial-sum workspace allocation failed");
        return ACES_ERR_NOMEM;
      }
      const long long nw = (long long)M * W;
      launch_after(k_gemv_part, (unsigned)((nw * 32 + 255) / 256), 256, 0, st, M, K, W, kc, A, lda,
                   x, part);
      count_launch();
      launch_after(k_gemv_final, (unsigned)((M + 255) / 256), 256, 0, st, M, W, alpha, part, beta,
                   C, transpose_out);
      count_launch();
      ACES_CUDA(cudaGetLastError());
      return ACES_OK;
    }
  }
  long long warps = M;
  long long nb = (warps * 32 + 255) / 256;
  if (nb > 148 * 32) nb = 148 * 32;
  launch_after(k_gemv_f64, (unsigned)nb, 256, 0, st, M, K, alpha, A, lda, x, beta, C,
               transpose_out);
  count_launch();
  ACES_CUDA(cudaGetLastError());
  return ACES_OK;
}

namespace {
// Tile shapes.  The DMMA pipe of an SM is filled by several small blocks rather
// than one large one: while one block waits at its k tile's barrier the others
// issue.  8192 x 4096 x 4096: 34.6 TFLOP/s with 64 x 64 tiles and three blocks
// per SM, 33.9 with 128 x 64 and two, 29.7 with 128 x 128 and one (the
// m8n8k4 and the m16n8k8 form of the instruction measure the same); and the
// last wave and the ragged edges of a 64-wide grid cost less: 2401 x 1519 x
// 2050 takes 513 us against 734 (2049, with the 8-byte copies of odd rows: 578).
// 32 x 32 tiles serve outputs too small for that: 120 x 96 x 150 in 6.5 us
// against 41.9 on one 128 x 128 tile.  The
// 16- and 32-wide tiles are for products with a short side, which stream
// their long operand: 404600 x 14 x 170 in 111 us (550 MB, 4.9 TB/s) against
// 690 us for an FMA kernel with synchronous 64 x 32 tiles.
using T64 = TileF64<64, 64, 2, 2, 3>;
using T32 = TileF64<32, 32, 2, 2, 6>;
using T6432 = TileF64<64, 32, 4, 1, 4>;
using T6416 = TileF64<64, 16, 4, 1, 5>;
enum TileId { kT64, kT32, kT6432, kT6416, kTiles };
struct TileInfo {
  int BM, BN, occ;
  double eff[2];  // share of the DMMA rate with one block per SM, and with occ
};
// (480 x 480 x 1000 on one 64 x 64 or two 32 x 32 blocks per SM, and the large
// shapes above)
constexpr TileInfo kTile[kTiles] = {{64, 64, T64::OCC, {0.60, 0.94}},
                                    {32, 32, T32::OCC, {0.35, 0.88}},
                                    {64, 32, T6432::OCC, {0.40, 0.78}},
                                    {64, 16, T6416::OCC, {0.25, 0.72}}};
constexpr int kSms = 148;

// Estimated time (us) of `tiles` tiles of nkt k tiles each: the blocks of the
// fullest SM at the rate of the blocks running there together, plus the
// pipeline's fill and drain per round of resident blocks.
double est_us(const TileInfo &t, double tiles, double nkt) {
  const double per_sm = std::ceil(tiles / kSms), r = std::min(per_sm, (double)t.occ);
  const double eff = t.eff[0] + (t.eff[1] - t.eff[0]) * (t.occ > 1 ? (r - 1) / (t.occ - 1) : 1);
  const double work = t.BM * t.BN * nkt * BK / 64.0 / 1.9e3;  // us per tile, 64 FMA/cycle
  return per_sm * work / eff + 2.0 * std::ceil(per_sm / t.occ);
}

// Tile shape and split-K slice count of one product, by that estimate; a split
// pays the write and read of its partials and a reduction launch.  part_cap:
// doubles of split-K workspace available.
struct F64Plan {
  int tile = kT64, Z = 1;
};
F64Plan plan_f64(int M, int N, int nkt, size_t part_cap) {
  F64Plan best;
  double tbest = 1e300;
  for (int id = 0; id < kTiles; ++id) {
    const TileInfo &t = kTile[id];
    const double tiles = (double)((M + t.BM - 1) / t.BM) * ((N + t.BN - 1) / t.BN);
    const int zmax = (int)std::min<double>(nkt / 8, std::ceil(4.0 * kSms * t.occ / tiles));
    for (int z = 1; z <= std::max(1, zmax); z += z < 16 ? 1 : z / 8) {
      if (z > 1 && (double)z * M * N > (double)part_cap) break;
      const int kc = (nkt + z - 1) / z;
      double us = est_us(t, tiles * z, kc);
      // a short side: the long operand's bytes at the rate the copies reach
      us = std::max(us, 8.0 * BK * nkt * (double)std::max(M, N) / 5.0e6);
      if (z > 1) us += 4.0 + 16.0 * z * M * (double)N / 4.0e6;
      if (us < tbest * 0.999) {
        tbest = us;
        best.tile = id;
        best.Z = z;
      }
    }
  }
  return best;
}

template <int VEC>
int launch_id(int id, const F64Launch &L, unsigned tiles, unsigned z, cudaStream_t st) {
  switch (id) {
    case kT64: return launch_tile<T64, VEC>(L, tiles, z, st);
    case kT32: return launch_tile<T32, VEC>(L, tiles, z, st);
    case kT6432: return launch_tile<T6432, VEC>(L, tiles, z, st);
    default: return launch_tile<T6416, VEC>(L, tiles, z, st);
  }
}
// 16-byte copies: aligned operands with even leading dimensions and K
bool vec2_ok(const F64Task &t) {
  for (int s = 0; s < t.nseg; ++s) {
    const F64Seg &g = t.seg[s];
    if (g.lda % 2 || g.ldb % 2 || g.K % 2 || ((uintptr_t)g.A & 15) || ((uintptr_t)g.B & 15))
      return false;
  }
  return true;
}

// The dispatch of gemm_nt_f64 and gemm_nt_f64_scratch: `ws` is the caller's
// workspace of `cap` doubles, or null for the library's own.
int gemm_dispatch(int M, int N, int K, double alpha, const double *A, long long lda,
                  const double *B, long long ldb, double beta, const CView &C, double *ws,
                  size_t cap, cudaStream_t st) {
  if (M <= 0 || N <= 0) return ACES_OK;
  // a few thousand outputs: one warp each (no tiles, no split K)
  if ((long long)M * N <= kTinyOut && K > 0 && K <= 8192) {
    launch_after(k_gemm_tiny_f64, (unsigned)(((long long)M * N * 32 + 255) / 256), 256, 0, st, M, N,
                 K, alpha, A, lda, B, ldb, beta, C);
    count_launch();
    ACES_CUDA(cudaGetLastError());
    return ACES_OK;
  }
  // K <= 32: output-bound low-rank update
  if (K <= LR_K) return launch_lowrank(M, N, K, alpha, A, lda, B, ldb, beta, C, st);
  F64Launch L{};
  F64Task &t = L.one;
  t.nseg = 1;
  t.M = M;
  t.N = N;
  t.seg[0] = F64Seg{A, B, lda, ldb, K};
  t.C = C;
  if (M < N) {  // the longer side takes the tile's longer edge
    std::swap(t.M, t.N);
    t.seg[0] = F64Seg{B, A, ldb, lda, K};
    t.C = CView{C.p, C.ndiv, C.sn1, C.sn0, C.mdiv, C.sm1, C.sm0};
  }
  L.alpha = alpha;
  L.beta = beta;
  const int nkt = f64_ktiles(t);
  const size_t kOwn = size_t(1) << 25;  // of the library's own workspace: 256 MB
  F64Plan p = plan_f64(t.M, t.N, nkt, ws ? cap : kOwn);
  if (p.Z > 1) {
    L.part = ws ? ws : splitk_workspace((size_t)p.Z * t.M * t.N);
    if (!L.part) p = plan_f64(t.M, t.N, nkt, 0);  // no room for the partials: unsplit
  }
  const long long tiles = (long long)((t.M + kTile[p.tile].BM - 1) / kTile[p.tile].BM) *
                          ((t.N + kTile[p.tile].BN - 1) / kTile[p.tile].BN);
  if (tiles > 0x7fffffffLL) {
    set_error("gemm_nt_f64: %lld output tiles", tiles);
    return ACES_ERR_ARG;
  }
  int Z = p.Z;
  if (Z > 1) {
    L.kchunk = (nkt + Z - 1) / Z;
    Z = (nkt + L.kchunk - 1) / L.kchunk;
  }
  if (vec2_ok(t))
    ACES_TRY(launch_id<2>(p.tile, L, (unsigned)tiles, (unsigned)Z, st));
  else
    ACES_TRY(launch_id<1>(p.tile, L, (unsigned)tiles, (unsigned)Z, st));
  if (L.part) return splitk_reduce(t.C, L.part, t.M, t.N, Z, alpha, beta, st);
  return ACES_OK;
}
}  // namespace

int gemm_nt_f64(int M, int N, int K, double alpha, const double *A, long long lda,
                const double *B, long long ldb, double beta, const CView &C, cudaStream_t st) {
  return gemm_dispatch(M, N, K, alpha, A, lda, B, ldb, beta, C, nullptr, 0, st);
}

// The same dispatch with the split-K partials taken from caller-provided
// device memory `ws` (capacity `cap` doubles) instead of the library's
// workspace; where they do not fit the product runs unsplit.
int gemm_nt_f64_scratch(int M, int N, int K, double alpha, const double *A, long long lda,
                        const double *B, long long ldb, double beta, const CView &C,
                        double *ws, size_t cap, cudaStream_t st) {
  return gemm_dispatch(M, N, K, alpha, A, lda, B, ldb, beta, C, ws, cap, st);
}

// ---- task tables --------------------------------------------------------------
// 64 x 64 tiles unless 32 x 32 ones are estimated faster (triangular tasks
// need a square tile, and a table mixes both kinds)
int f64_tasks_plan(F64Task *tasks, int n, F64TaskPlan *plan) {
  *plan = F64TaskPlan{};
  double work[2] = {0.0, 0.0};
  long long total[2] = {0, 0};
  bool same = true, vec2 = true;
  for (int i = 0; i < n; ++i) {
    const F64Task &t = tasks[i];
    if (t.M < 1 || t.N < 1 || t.nseg < 1 || t.nseg > 4 || (t.tri && t.M != t.N)) {
      set_error("f64 tasks: task %d is %d x %d with %d segments", i, t.M, t.N, t.nseg);
      return ACES_ERR_ARG;
    }
    for (int s = 0; s < t.nseg; ++s)  // the kernel steps from one segment to the next
      if (t.seg[s].K < 1) {
        set_error("f64 tasks: segment %d of task %d has K = %d", s, i, t.seg[s].K);
        return ACES_ERR_ARG;
      }
    const int nkt = f64_ktiles(t);
    for (int b = 0; b < 2; ++b) {
      const int nt = f64_tiles(t.M, t.N, t.tri, kTile[b].BM, kTile[b].BN);
      total[b] += nt;
      work[b] += (double)nt * nkt;
    }
    same = same && t.M == tasks[0].M && t.N == tasks[0].N && t.tri == tasks[0].tri;
    vec2 = vec2 && vec2_ok(t);
  }
  if (n == 0) return ACES_OK;
  int b = 0;
  if (est_us(kTile[kT32], (double)total[1], work[1] / total[1]) <
      est_us(kTile[kT64], (double)total[0], work[0] / total[0]))
    b = 1;
  if (total[b] > 0x7fffffffLL) {
    set_error("f64 tasks: %lld output tiles", total[b]);
    return ACES_ERR_ARG;
  }
  long long at = 0;
  for (int i = 0; i < n; ++i) {
    tasks[i].tile0 = (int)at;
    at += f64_tiles(tasks[i].M, tasks[i].N, tasks[i].tri, kTile[b].BM, kTile[b].BN);
  }
  plan->tile = b;
  plan->tiles = (int)at;
  plan->per_task = same ? (int)(at / n) : 0;
  plan->vec2 = vec2;
  return ACES_OK;
}

int f64_tasks_run(const F64Task *dev, int n, const F64TaskPlan &plan, double alpha, double beta,
                  cudaStream_t st) {
  if (n == 0 || plan.tiles == 0) return ACES_OK;
  F64Launch L{};
  L.table = dev;
  L.ntask = n;
  L.per_task = plan.per_task;
  L.alpha = alpha;
  L.beta = beta;
  return plan.vec2 ? launch_id<2>(plan.tile, L, (unsigned)plan.tiles, 1, st)
                   : launch_id<1>(plan.tile, L, (unsigned)plan.tiles, 1, st);
}

}  // namespace acesb200
