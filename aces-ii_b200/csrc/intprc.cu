// intprc.cu -- the MO-integral list producer on the device: the six lists the
// closed-shell CC programs read, from density-fitted (or Cholesky) factors of
// the MO two-electron integrals.
//
// The reference's integral chain is vtran (AO -> MO transformation,
// vtran/vtran.F) followed by intprc, which sorts the transformed integrals
// into the irrep-blocked MOINTS lists (intprc/clmoio.F:46-260 creates lists
// 13, 10, 16, 25, 30, 233 with the pair types used here).  This entry point
// takes the MO factors B^L_pq, (pq|rs) = sum_L B^L_pq B^L_rs; a list element
// (row (p,q), column (r,s)) is <pq|rs> = (pr|qs).
//
// The FP64 tensor cores bound this step (2 v^4 naux operations for the
// dense <Ab|Cd> alone), so only distinct integrals are computed: the pairs
// (pr) and (qs) are packed (p <= r) and grouped by pair irrep, one product
// G_h = F_h F_h'^T per pair irrep h over the packed rows F[(pr)][L], and only
// the lower triangle of tiles where both sides are the same pairs (lists 13,
// 16 and 233).  Bandwidth-bound kernels then write the list blocks from G.
// o = 20, v = 180, naux = 600: 52.4 ms of dense products became 7.5 ms of
// packed ones (32 TFLOP/s) and 3.2 ms of expansion; with 8 irreps the products
// shrink by another factor of 64 at most.
//
// That takes factors equal to their transposes bit for bit.  Others, symmetric
// to rounding only or not at all, take dense products over all ordered pairs,
// as they are; so do systems whose packed G does not fit beside the lists.
#include <algorithm>
#include <cmath>
#include <vector>

#include "engine.cuh"

using namespace acesb200;

namespace {
struct ListSpec {
  int list, typeL, typeR;
  char P, Q, R, S;
};
// intprc/clmoio.F: list, row pair type, column pair type, index spaces
const ListSpec kLists[6] = {
    {13, 14, 14, 'o', 'o', 'o', 'o'},    // <Ij|Kl>
    {10, 14, 18, 'o', 'o', 'o', 'v'},    // <Ij|Ka>
    {16, 13, 14, 'v', 'v', 'o', 'o'},    // <Ab|Ij>
    {25, 11, 11, 'v', 'o', 'v', 'o'},    // <Ai|Bj>
    {30, 13, 11, 'v', 'v', 'v', 'o'},    // <Ab|Ci>
    {233, 13, 13, 'v', 'v', 'v', 'v'},   // <Ab|Cd>
};

// ---- symmetric factors --------------------------------------------------------
// stats[0] = max |B|, stats[1] = max |B[L][p][q] - B[L][q][p]| as the bit
// patterns of non-negative doubles (ordered like integers; a NaN is above
// every number).  One block per 32 x 32 tile pair of (p, q) and slab of L.
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffULL;
}
__global__ void __launch_bounds__(256)
    k_factor_stats(const double *__restrict__ B, int naux, int n,
                   unsigned long long *__restrict__ stats) {
  after_previous();
  __shared__ double T[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int tiles = (n + 31) / 32;
  int tp = blockIdx.x, td = 0;
  while ((td + 1) * (td + 2) / 2 <= tp) ++td;
  const int tc = tp - td * (td + 1) / 2;
  if (td >= tiles) return;
  unsigned long long big = 0, dif = 0;
  for (int L = blockIdx.y; L < naux; L += gridDim.y) {
    const double *X = B + (size_t)L * n * n;
    double y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = ty + 8 * k, p = td * 32 + r, q = tc * 32 + tx;   // tile (td, tc)
      y[k] = (p < n && q < n) ? X[(size_t)p * n + q] : 0.0;
      const int p2 = tc * 32 + r, q2 = td * 32 + tx;                 // tile (tc, td)
      T[r][tx] = (p2 < n && q2 < n) ? X[(size_t)p2 * n + q2] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double z = T[tx][ty + 8 * k];
      big = max(big, max(abs_bits(y[k]), abs_bits(z)));
      if (!(y[k] == z)) dif = max(dif, abs_bits(y[k] - z));   // a NaN differs from itself
    }
    __syncthreads();
  }
  for (int off = 16; off; off >>= 1) {
    big = max(big, __shfl_xor_sync(0xffffffffu, big, off));
    dif = max(dif, __shfl_xor_sync(0xffffffffu, dif, off));
  }
  if (tx == 0) {
    atomicMax(stats, big);
    if (dif) atomicMax(stats + 1, dif);
  }
}

// F[row][L] = B[L][p][q] of the row's orbital pair (p >= q), L < kp (zero past
// naux): 32 rows x 32 L per block through a shared-memory transpose; the rows
// of a tile are neighbours in q, so the reads coalesce but for the ends of
// the runs.
__global__ void __launch_bounds__(256)
    k_factor_pack(double *__restrict__ F, const double *__restrict__ B,
                  const int2 *__restrict__ rows, int nrows, int naux, int kp, int n) {
  after_previous();
  __shared__ double T[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int r0 = blockIdx.x * 32, L0 = blockIdx.y * 32;
  const int r = r0 + tx;
  size_t at = 0;
  if (r < nrows) {
    const int2 pq = rows[r];
    at = (size_t)pq.x * n + pq.y;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int L = L0 + ty + 8 * k;
    T[ty + 8 * k][tx] = (r < nrows && L < naux) ? B[(size_t)L * n * n + at] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int rr = r0 + ty + 8 * k, L = L0 + tx;
    if (rr < nrows && L < kp) F[(size_t)rr * kp + L] = T[tx][ty + 8 * k];
  }
}

// One irrep: the packed rows of G to the list.  Row R of G holds the packed
// symmetric n x n matrix of its pair (x, y) = rows[R] at c(c+1)/2 + a, a <= c;
// it goes to out[base + c sc + a] for all (c, a), base = x sx + y sy, and with
// swap to base = y sx + x sy as well (the other order of the pair).  A block
// walks the 32 x 32 tile pairs of its row; the packed tile is read once with
// lanes along a, and both orders of (c, a) are written with lanes along the
// unit stride.  Write bound.
__global__ void __launch_bounds__(256)
    k_expand_pairs(double *__restrict__ out, const double *__restrict__ G, long long ldg,
                   const int2 *__restrict__ rows, int x0, int y0, int n, long long sx,
                   long long sy, long long sc, int swap) {
  after_previous();
  __shared__ double X[32][33];   // [c local][a local]
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int2 pr = rows[blockIdx.x];
  const long long x = pr.x - x0, y = pr.y - y0;
  const double *row = G + (long long)blockIdx.x * ldg;
  const int tiles = (n + 31) / 32, ntp = tiles * (tiles + 1) / 2;
  for (int tp = blockIdx.y; tp < ntp; tp += gridDim.y) {
    int td = (int)((sqrtf(8.0f * tp + 1.0f) - 1.0f) * 0.5f);
    while (td * (td + 1) / 2 > tp) --td;
    while ((td + 1) * (td + 2) / 2 <= tp) ++td;
    const int c0 = td * 32, a0 = (tp - td * (td + 1) / 2) * 32;
    __syncthreads();  // the previous tile's reads are done
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int cl = ty + 8 * k, c = c0 + cl, a = a0 + tx;
      if (c < n && a <= c) {
        const double v = __ldcs(row + (long long)c * (c + 1) / 2 + a);
        X[cl][tx] = v;
        if (c0 == a0) X[tx][cl] = v;
      }
    }
    __syncthreads();
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      if (o == 1 && (!swap || x == y)) break;
      double *z = out + (o == 0 ? x * sx + y * sy : y * sx + x * sy);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int l = ty + 8 * k;
        if (c0 + l < n && a0 + tx < n) z[(long long)(c0 + l) * sc + a0 + tx] = X[l][tx];
        if (c0 != a0 && a0 + l < n && c0 + tx < n)
          z[(long long)(a0 + l) * sc + c0 + tx] = X[tx][l];
      }
    }
  }
}

// Several irreps: list block element (row (p,q), column (r,s)) of the block's
// pair irrep from G[(qs)][(pr)] of the irrep of (p,r).  Lanes run along the
// rows, p fastest: the stores coalesce, and so do the reads for p <= r.
struct GBlocks {
  const double *G[8];   // by pair irrep of (p,r)
  long long ld[8];
};
__global__ void __launch_bounds__(256)
    k_expand_irrep(double *__restrict__ out, GBlocks g, const int2 *__restrict__ rowtab,
                   const int2 *__restrict__ coltab, int nrows, int ncols,
                   const int *__restrict__ pidx, const int *__restrict__ irr, int n) {
  after_previous();
  const int ri = blockIdx.x * 256 + threadIdx.x;
  if (ri >= nrows) return;
  const int2 pq = rowtab[ri];
  const int hp = irr[pq.x];
  for (int ci = blockIdx.y; ci < ncols; ci += gridDim.y) {
    const int2 rs = coltab[ci];
    const int h = hp ^ irr[rs.x];
    out[(size_t)ci * nrows + ri] =
        g.G[h][pidx[pq.y * n + rs.y] * g.ld[h] + pidx[pq.x * n + rs.x]];
  }
}

int tri_tiles(int n) {
  const int t = (n + 31) / 32;
  return t * (t + 1) / 2;
}

// Device memory of one call, given back at its end.
struct Scratch {
  std::vector<void *> p;
  ~Scratch() {
    for (void *q : p) dev_free(q);
  }
  void *get(size_t bytes) {
    void *q = nullptr;
    if (dev_alloc(&q, std::max<size_t>(bytes, 8)) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    p.push_back(q);
    return q;
  }
};

// The symmetric path; *done = false when the factors are not symmetric or
// the scratch does not fit (no list has been written then).
int produce_packed(const double *dB, int naux, const std::vector<int> &irr_o,
                   const std::vector<int> &irr_v, cudaStream_t st, bool *done) {
  *done = false;
  const SymInfo &s = state().sym;
  const int g = s.nirrep, o = (int)irr_o.size(), v = (int)irr_v.size(), n = o + v;
  const int kp = (naux + 1) / 2 * 2;  // even rows: 16-byte copies
  // ---- pair rows by set (0: oo, 1: ov, 2: vv) and pair irrep, and their index
  std::vector<int> irr(irr_o);
  irr.insert(irr.end(), irr_v.begin(), irr_v.end());
  std::vector<int2> rows;
  std::vector<int> pidx((size_t)n * n, -1);
  int off[3][9], cnt[3][8];
  for (int set = 0; set < 3; ++set)
    for (int h = 0; h < 8; ++h) {
      off[set][h] = (int)rows.size();
      cnt[set][h] = 0;
      if (h < g) {
        // p >= q: oo and vv packed (p slow), ov with the virtual index fastest
        const int p0 = set == 2 ? o : 0, p1 = set == 2 ? n : o;
        for (int p = p0; p < p1; ++p) {
          const int q0 = set == 0 ? 0 : o, q1 = set == 1 ? n : p + 1;
          for (int q = q0; q < q1; ++q) {
            if ((irr[p] ^ irr[q]) != h) continue;
            pidx[(size_t)p * n + q] = pidx[(size_t)q * n + p] = cnt[set][h]++;
            rows.push_back(make_int2(p, q));
          }
        }
      }
      off[set][h + 1] = (int)rows.size();
    }
  const int nrows = (int)rows.size();
  // ---- the products: list, row set, column set (of G[(qs)][(pr)]); list 233's
  // G is the largest and has the scratch to itself
  struct Prod {
    int list, R, C;
  };
  const Prod prods[6] = {{13, 0, 0}, {10, 1, 0}, {16, 1, 1}, {25, 0, 2}, {30, 1, 2}, {233, 2, 2}};
  const bool direct16 = g == 1;  // <Ab|Ij> without symmetry is G itself, in place
  size_t goff[6][8], need_small = 0, need_vv = 0;
  for (int k = 0; k < 6; ++k)
    for (int h = 0; h < g; ++h) {
      const size_t sz = prods[k].list == 16 && direct16
                            ? 0
                            : (size_t)cnt[prods[k].R][h] * cnt[prods[k].C][h];
      size_t &at = k < 5 ? need_small : need_vv;
      goff[k][h] = at;
      at += (sz + 1) / 2 * 2;
    }
  // ---- scratch (after the lists, so that it never takes their room), and the
  // symmetry of the factors
  Scratch mem;
  auto *d_stats = (unsigned long long *)mem.get(16);
  if (!d_stats) return ACES_OK;
  ACES_CUDA(cudaMemsetAsync(d_stats, 0, 16, st));
  launch_after(k_factor_stats, dim3(tri_tiles(n), std::min(naux, 64)), 256, 0, st, dB, naux, n,
               d_stats);
  count_launch();
  ACES_CUDA(cudaGetLastError());
  double stats[2];
  ACES_CUDA(cudaMemcpyAsync(stats, d_stats, 16, cudaMemcpyDeviceToHost, st));
  ACES_CUDA(cudaStreamSynchronize(st));
  if (!std::isfinite(stats[0]) || stats[1] != 0.0) return ACES_OK;   // (a NaN too)
  double *F = (double *)mem.get((size_t)nrows * kp * 8);
  double *G = (double *)mem.get(std::max(need_small, need_vv) * 8);
  // one upload: rows, the pair-type tables of the irrep blocks, indices
  std::vector<int2> tab(rows);
  int tab_at[2][2];  // [space of p][space of q]: pairs in list order, all irreps
  std::vector<int> first[2];
  if (g > 1) {
    const std::vector<int> *ir[2] = {&irr_o, &irr_v};
    for (int a = 0; a < 2; ++a)
      for (int b = 0; b < 2; ++b) {
        tab_at[a][b] = (int)tab.size();
        for (int h = 0; h < g; ++h)
          for (int hq = 0; hq < g; ++hq)
            for (size_t q = 0; q < ir[b]->size(); ++q) {
              if ((*ir[b])[q] != hq) continue;
              for (size_t p = 0; p < ir[a]->size(); ++p)
                if (((*ir[a])[p] ^ hq) == h)
                  tab.push_back(make_int2((int)p + (a ? o : 0), (int)q + (b ? o : 0)));
            }
      }
  }
  std::vector<int> ints(pidx);
  ints.insert(ints.end(), irr.begin(), irr.end());
  std::vector<F64Task> tasks;
  int task_k[6] = {0};
  const size_t bytes_tab = tab.size() * sizeof(int2), bytes_int = (ints.size() + 3) / 4 * 16;
  char *up = (char *)mem.get(bytes_tab + 16 + bytes_int + 48 * sizeof(F64Task));
  if (!F || !G || !up) return ACES_OK;
  int2 *d_tab = (int2 *)up;
  int *d_ints = (int *)(up + (bytes_tab + 15) / 16 * 16);
  F64Task *d_tasks = (F64Task *)((char *)d_ints + bytes_int);
  double *base[6];
  for (int k = 0; k < 6; ++k) base[k] = aces_list_devptr(1, prods[k].list);
  const long long O = o, V = v;
  F64TaskPlan plan[2];
  for (int k = 0; k < 6; ++k) {
    if (k == 5) ACES_TRY(f64_tasks_plan(tasks.data(), (int)tasks.size(), &plan[0]));
    task_k[k] = (int)tasks.size();
    for (int h = 0; h < g; ++h) {
      const int M = cnt[prods[k].R][h], N = cnt[prods[k].C][h];
      if (M == 0 || N == 0) continue;
      F64Task t{};
      t.nseg = 1;
      t.M = M;
      t.N = N;
      t.tri = prods[k].R == prods[k].C;
      t.seg[0] = F64Seg{F + (size_t)off[prods[k].R][h] * kp, F + (size_t)off[prods[k].C][h] * kp,
                        kp, kp, kp};
      if (k == 2 && direct16)  // m = (j,b), n = (i,a): a + b v + i v^2 + j v^2 o
        t.C = CView{base[k], V, V * V * O, V, V, V * V, 1};
      else
        t.C = cview_rowmajor(G + goff[k][h], N);
      tasks.push_back(t);
    }
  }
  const int n_small = task_k[5], n_vv = (int)tasks.size() - n_small;
  ACES_TRY(f64_tasks_plan(tasks.data() + n_small, n_vv, &plan[1]));
  ACES_CUDA(cudaMemcpyAsync(d_tab, tab.data(), bytes_tab, cudaMemcpyHostToDevice, st));
  ACES_CUDA(cudaMemcpyAsync(d_ints, ints.data(), ints.size() * 4, cudaMemcpyHostToDevice, st));
  ACES_CUDA(cudaMemcpyAsync(d_tasks, tasks.data(), tasks.size() * sizeof(F64Task),
                            cudaMemcpyHostToDevice, st));
  launch_after(k_factor_pack, dim3((nrows + 31) / 32, (kp + 31) / 32), 256, 0, st, F, dB, d_tab,
               nrows, naux, kp, n);
  count_launch();
  ACES_CUDA(cudaGetLastError());
  // ---- one irrep: list offset of (pair (x,y) of the row, matrix (c,a) of the columns)
  auto expand = [&](int k) -> int {
    const Prod &P = prods[k];
    if (g == 1) {
      if (k == 2) return ACES_OK;
      long long sx = 0, sy = 0, sc = 0;
      int x0 = 0, y0 = 0, m = 0;
      switch (k) {
        case 0: m = o; sx = O * O * O; sy = O; sc = O * O; break;               // (j,l) x (k,i)
        case 1: m = o; y0 = o; sx = O; sy = O * O * O; sc = O * O; break;       // (j,a) x (k,i)
        case 3: m = v; sx = V * V * O; sy = V; sc = V * O; break;               // (j,i) x (b,a)
        case 4: m = v; y0 = o; sx = V * V * V; sy = V; sc = V * V; break;       // (i,b) x (c,a)
        default: m = v; x0 = y0 = o; sx = V * V * V; sy = V; sc = V * V;        // (d,b) x (c,a)
      }
      const int R = cnt[P.R][0], tp = tri_tiles(m);
      // enough blocks for the machine, few tile pairs each when there are many rows
      const int ny = std::max(1, std::min(tp, (148 * 16 + R - 1) / R));
      launch_after(k_expand_pairs, dim3(R, ny), 256, 0, st, base[k], G + goff[k][0], cnt[P.C][0],
                   d_tab + off[P.R][0], x0, y0, m, sx, sy, sc, P.R != 1);
      count_launch();
    } else {
      GBlocks gb{};
      for (int h = 0; h < g; ++h) {
        gb.G[h] = G + goff[k][h];
        gb.ld[h] = cnt[P.C][h];
      }
      const ListSpec *L = kLists;
      while (L->list != P.list) ++L;
      const int sp[4] = {L->P == 'v', L->Q == 'v', L->R == 'v', L->S == 'v'};
      size_t ra = tab_at[sp[0]][sp[1]], ca = tab_at[sp[2]][sp[3]];
      for (int h = 0; h < g; ++h) {
        int nc = 0, nr = 0;
        aces_list_dims(h + 1, P.list, &nc, &nr);
        if (nc > 0 && nr > 0) {
          launch_after(k_expand_irrep, dim3((nr + 255) / 256, std::min(nc, 32768)), 256, 0, st,
                       aces_list_devptr(h + 1, P.list), gb, d_tab + ra, d_tab + ca, nr, nc, d_ints,
                       d_ints + (size_t)n * n, n);
          count_launch();
        }
        ra += nr;
        ca += nc;
      }
    }
    ACES_CUDA(cudaGetLastError());
    return ACES_OK;
  };
  ACES_TRY(f64_tasks_run(d_tasks, n_small, plan[0], 1.0, 0.0, st));
  for (int k = 0; k < 5; ++k) ACES_TRY(expand(k));
  ACES_TRY(f64_tasks_run(d_tasks + n_small, n_vv, plan[1], 1.0, 0.0, st));
  ACES_TRY(expand(5));
  ACES_CUDA(cudaStreamSynchronize(st));
  *done = true;
  return ACES_OK;
}
}  // namespace

extern "C" int aces_intprc_df(const double *B, int naux, int on_device) {
  State &stt = state();
  std::lock_guard<std::recursive_mutex> lk(stt.mu);
  const SymInfo &s = stt.sym;
  if (!s.ready) {
    set_error("aces_intprc_df: symmetry not initialised (aces_sym_init)");
    return ACES_ERR_NOSYM;
  }
  if (!B || naux < 1) {
    set_error("aces_intprc_df: null factors or naux %d < 1", naux);
    return ACES_ERR_ARG;
  }
  std::vector<int> irr_o, irr_v;
  for (int h = 0; h < s.nirrep; ++h) {
    for (int k = 0; k < s.pop[h]; ++k) irr_o.push_back(h);
    for (int k = 0; k < s.vrt[h]; ++k) irr_v.push_back(h);
  }
  const long long o = (long long)irr_o.size(), v = (long long)irr_v.size(), n = o + v;
  if (o == 0 || v == 0) {
    set_error("aces_intprc_df: empty occupied or virtual space");
    return ACES_ERR_ARG;
  }
  CallScope call;
  cudaStream_t st = 0;
  std::vector<void *> owned;
  struct Free {
    std::vector<void *> &p;
    ~Free() {
      for (void *q : p) dev_free(q);
    }
  } release{owned};
  auto get = [&](double **out, size_t doubles) -> int {
    if (dev_alloc((void **)out, std::max<size_t>(doubles, 1) * 8) != cudaSuccess) {
      cudaGetLastError();
      set_error("aces_intprc_df: device allocation of %zu doubles failed", doubles);
      return ACES_ERR_NOMEM;
    }
    owned.push_back(*out);
    return ACES_OK;
  };
  const double *dB = B;
  if (!on_device) {
    double *t = nullptr;
    ACES_TRY(get(&t, (size_t)naux * n * n));
    ACES_CUDA(cudaMemcpyAsync(t, B, (size_t)naux * n * n * 8, cudaMemcpyHostToDevice, st));
    dB = t;
  }
  // every irrep of the lists, without the zero fill: all their pair types are
  // FULL, so each element is written below
  UnfilledLists unfilled[6];   // by list
  for (int k = 0; k < 6; ++k)
    ACES_TRY(list_inipck(1, kLists[k].typeL, kLists[k].typeR, kLists[k].list, 1, &unfilled[k]));
  {
    bool done = false;
    ACES_TRY(produce_packed(dB, naux, irr_o, irr_v, st, &done));
    if (done) {
      for (auto &u : unfilled) u.written();
      return ACES_OK;
    }
  }
  // ---- any factors: dense products over all ordered pairs,
  //   <pq|rs> = sum_L B_RP[r][p][L] B_SQ[s][q][L]
  // without symmetry straight into the list's column-major block (m = (r,p)
  // with p fastest has unit stride there), with irreps to a dense [r][p][s][q]
  // scratch that k_scatter_rpsq distributes over the irrep blocks.
  // K-contiguous factor blocks XY[x][y][L] = B[L][X0 + x][Y0 + y]
  double *blk[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
  const long long dim[2] = {o, v}, off[2] = {0, o};
  for (int X = 0; X < 2; ++X)
    for (int Y = 0; Y < 2; ++Y) {
      ACES_TRY(get(&blk[X][Y], (size_t)(dim[X] * dim[Y] * naux)));
      PermSpec ps;
      ps.n[0] = 1; ps.n[1] = (int)dim[X]; ps.n[2] = (int)dim[Y]; ps.n[3] = naux;
      ps.nterms = 1;
      ps.beta = 0.0;
      ps.t[0].src = dB + off[X] * n + off[Y];
      ps.t[0].alpha = 1.0;
      ps.t[0].s[0] = 0; ps.t[0].s[1] = n; ps.t[0].s[2] = 1; ps.t[0].s[3] = n * n;
      ACES_TRY(permute(blk[X][Y], ps, st));
    }
  auto sp = [](char c) { return c == 'o' ? 0 : 1; };
  double *X = nullptr;
  size_t xcap = 0;
  for (const ListSpec &L : kLists) {
    const long long np = dim[sp(L.P)], nq = dim[sp(L.Q)], nr = dim[sp(L.R)],
                    ns = dim[sp(L.S)];
    const double *A = blk[sp(L.R)][sp(L.P)], *Bm = blk[sp(L.S)][sp(L.Q)];
    const int M = (int)(nr * np), N = (int)(ns * nq);
    DevMap dm;
    ACES_TRY(make_map(dm, L.list, L.typeL, L.typeR, irr_o, irr_v, false));
    if (s.nirrep == 1) {
      double *lp = aces_list_devptr(1, L.list);
      const long long nrows = np * nq;
      // m = (r, p), n = (s, q): offset p + q np + (r + s nr) nrows
      const CView C{lp, np, nrows, 1, nq, nr * nrows, np};
      ACES_TRY(gemm_nt_f64(M, N, naux, 1.0, A, naux, Bm, naux, 0.0, C, st));
    } else {
      const size_t need = (size_t)M * N;
      if (need > xcap) {
        ACES_TRY(get(&X, need));
        xcap = need;
      }
      ACES_TRY(gemm_nt_f64(M, N, naux, 1.0, A, naux, Bm, naux, 0.0, cview_rowmajor(X, N), st));
      launch_scatter_rpsq(X, dm.m, st);
      ACES_CUDA(cudaGetLastError());
    }
    ACES_CUDA(cudaStreamSynchronize(st));
    unfilled[&L - kLists].written();
  }
  return ACES_OK;
}
