// triples.cu -- the (T) correction (trp/trps.F -> trp/trps2.F, trp/d1t2new.F,
// librt3/rmd314.f, trp/e4tijk.F, trp/t1t32n.f) on the device.
//
// For every occupied triplet i >= j >= k the connected triples
//   W_ijk^abc = sum over the 6 simultaneous permutations of (ia)(jb)(kc) of
//     X_ijk^abc = sum_d t(ij,ad) (bd|ck) - sum_l t(il,ab) (ck|jl)
// are built in a v^3 slot per triplet by three tensor-core launches (the 12
// contractions grouped by output orientation, four K segments each) whose
// outputs land in place through coalesced two-level views.  The energy kernel
// then sums, for the distinct permutations of (i,j,k) and all orderings of
// every virtual set {a>=b>=c}, the closed-shell expression
//   E[4]T  = 1/3 sum (4W_abc + W_bca + W_cab)(W_abc - W_cba)/D_ijk^abc
//   E[5]ST = 1/3 sum (4W_abc + W_bca + W_cab)(V_abc - V_cba)/D_ijk^abc,
//   V - W = t_i^a (jb|kc) + t_j^b (ia|kc) + t_k^c (ia|jb),
// reading every W element once per triplet.  Partial sums are kept per
// (triplet, block) and reduced in a fixed order: the FP64 energy sum is
// deterministic.
#include <algorithm>
#include <cmath>
#include <functional>
#include <vector>

#include "engine.cuh"

namespace acesb200 {

namespace {
// The six orderings s of a virtual set x = (x0, x1, x2): ordering s reads
// W at (x[kOrd[s][0]], x[kOrd[s][1]], x[kOrd[s][2]]).
constexpr int kOrd[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};

// The energy of a virtual set.  With the ordering s of the set read as an
// element of the permutation group, the terms of E[4]T over all orderings of
// the set and all permutations of (i,j,k),
//   sum_{q,p} (4 u_s0 + u_s1 + u_s2)(u_s0 - u_s3)
// (s0..s3: the orderings of W_abc, W_bca, W_cab, W_cba under q and p), are the
// bilinear form u^T M u with M[s][s] = 24, M[s][s'] = 6 where s' is a cyclic
// permutation of s (the orderings 0, 3, 4 and 1, 2, 5) and -12 otherwise, and
// E[5]ST is u^T M vd.  So (M u)_s = 18 u_s + 6 E - 12 O on the even orderings
// and 18 u_s + 6 O - 12 E on the odd ones, E and O the sums over 0, 3, 4 and
// 1, 2, 5.  A repeated virtual makes orderings coincide in pairs (or all six):
// their distinct ones contribute half (a sixth) of the form.

// a >= b >= c from the flat index n of the set in the order
// (a, then b <= a, then c <= b): n = a(a+1)(a+2)/6 + b(b+1)/2 + c
__device__ __forceinline__ void decode_set(int n, int &a, int &b, int &c) {
  int x = (int)cbrtf(6.0f * (float)n);
  while ((long long)x * (x + 1) * (x + 2) / 6 > n) --x;
  while ((long long)(x + 1) * (x + 2) * (x + 3) / 6 <= n) ++x;
  a = x;
  int r = n - (int)((long long)x * (x + 1) * (x + 2) / 6);
  int y = (int)((sqrtf(8.0f * (float)r + 1.0f) - 1.0f) * 0.5f);
  while (y * (y + 1) / 2 > r) --y;
  while ((y + 1) * (y + 2) / 2 <= r) ++y;
  b = y;
  c = r - y * (y + 1) / 2;
}

// One batch entry's contribution to E[4]T and E[5]ST, every set {a >= b >= c}
// of virtuals evaluated once.  Block (blockIdx.x, blockIdx.y = e) takes one
// tile triple A >= B >= C of 8-wide virtual tiles (decoded like a set) of
// triplet e and stages in shared memory, with sector-complete row reads, the
// six permuted 8x8x8 cubes of W (tiles (A,B,C), (A,C,B), ..., one per
// ordering), the 8x8 tiles of the <jk|..>, <ik|..>, <ij|..> slabs for every
// ordered pair of the three tiles, and the t1 rows and orbital energies of the
// three tiles.  Each of its 128 threads then evaluates four sets that share
// (b, c): what depends on these alone is read once.
// Instruction bound (W is read once, at 16 % of the DRAM rate, the issue slots
// two thirds full): with index splits per staged element, 36 shared-memory reads
// and a general 6 x 6 form per set, and a per-ordering sum for repeated virtuals
// o = 14, v = 170 took 14.0 ms; with the form above and these loop orders 8.3.
constexpr int kTile = 8;
// triplets of one FP64 batch (the energy launch's grid.y holds 65535)
constexpr int kMaxTasks = 32768;
// kOrd[s][r] in device code: the first position is s / 2, the other two
// follow in increasing order for even s and swapped for odd s
__host__ __device__ __forceinline__ constexpr int ordpos(int s, int r) {
  const int f = s >> 1, lo = f == 0 ? 1 : 0, hi = f == 2 ? 1 : 2;
  return r == 0 ? f : (r == 1 ? ((s & 1) ? hi : lo) : ((s & 1) ? lo : hi));
}
static_assert(ordpos(0, 2) == kOrd[0][2] && ordpos(3, 1) == kOrd[3][1] &&
                  ordpos(4, 2) == kOrd[4][2] && ordpos(5, 0) == kOrd[5][0] &&
                  ordpos(1, 1) == kOrd[1][1] && ordpos(2, 1) == kOrd[2][1],
              "ordpos restates kOrd");
// index of the ordered pair (x, y) of tile positions, x != y
__host__ __device__ __forceinline__ constexpr int pairpos(int x, int y) {
  return x * 2 + (y > x ? y - 1 : y);
}
template <typename TW>
__global__ void __launch_bounds__(128)
    k_triples_energy_tiled(const TW *__restrict__ Wbase, long long wstride,
                           const int *__restrict__ trip3, const double *__restrict__ t1,
                           const double *__restrict__ Ioovv, const double *__restrict__ eo,
                           const double *__restrict__ ev, int o, int v,
                           double *__restrict__ part) {
  after_previous();
  __shared__ TW cube[6][kTile][kTile + 1][kTile + 1];
  __shared__ double It[3][6][kTile][kTile + 1];
  __shared__ double ts[3][3][kTile];   // [t_i, t_j, t_k][tile position][local]
  __shared__ double es[3][kTile];      // ev of the three tiles
  __shared__ double sh[2][4];
  const int e = blockIdx.y;
  const int i = trip3[3 * e], j = trip3[3 * e + 1], k = trip3[3 * e + 2];
  const TW *__restrict__ W = Wbase + (long long)e * wstride;
  const int mult = (i == j && j == k) ? 6 : ((i == j || j == k) ? 2 : 1);
  const double scale = 1.0 / (3.0 * mult);
  const int v2 = v * v;
  int T[3];
  decode_set((int)blockIdx.x, T[0], T[1], T[2]);
  const int b0[3] = {T[0] * kTile, T[1] * kTile, T[2] * kTile};
  const int tid = threadIdx.x;
  // this thread's place in an 8 x 8 tile and which half of the third index
  const int half = tid >> 6, l1 = (tid >> 3) & 7, l2 = tid & 7;
  // six cubes: cube s spans tiles (T[kOrd[s][0]], T[kOrd[s][1]], T[kOrd[s][2]]);
  // the thread loads (x, y, z) = (half + 2 q, l1, l2)
#pragma unroll
  for (int s = 0; s < 6; ++s) {
    const int gx = b0[ordpos(s, 0)] + half, gy = b0[ordpos(s, 1)] + l1,
              gz = b0[ordpos(s, 2)] + l2;
    const TW *w = W + ((long long)gx * v2 + (gy * v + gz));
    const bool in = gy < v && gz < v;
    TW x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = in && gx + 2 * q < v ? w[(long long)(2 * q) * v2] : (TW)0;
#pragma unroll
    for (int q = 0; q < 4; ++q) cube[s][half + 2 * q][l1][l2] = x[q];
  }
  // integral tiles: slab 0 = <jk|..>, 1 = <ik|..>, 2 = <ij|..>; the two halves
  // of the block take the two pairs (x, .) of each x
  const double *slab[3] = {Ioovv + ((long long)j * o + k) * v2, Ioovv + ((long long)i * o + k) * v2,
                           Ioovv + ((long long)i * o + j) * v2};
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const int y = half < x ? half : half + 1;
    const int gr = b0[x] + l1, gc = (y == 0 ? b0[0] : (y == 1 ? b0[1] : b0[2])) + l2;
    const bool in = gr < v && gc < v;
    const int at = gr * v + gc;
#pragma unroll
    for (int sl = 0; sl < 3; ++sl) It[sl][2 * x + half][l1][l2] = in ? slab[sl][at] : 0.0;
  }
  if (tid < 72) {
    const int w = tid / 24, pos = (tid / 8) % 3, l = tid & 7;
    const int occ = w == 0 ? i : (w == 1 ? j : k), g = b0[pos] + l;
    ts[w][pos][l] = g < v ? t1[(long long)occ * v + g] : 0.0;
  } else if (tid < 96) {
    const int pos = (tid - 72) / 8, l = tid & 7, g = b0[pos] + l;
    es[pos][l] = g < v ? ev[g] : 0.0;
  }
  __syncthreads();
  double s4 = 0.0, s5 = 0.0;
  const int b = b0[1] + l1, c = b0[2] + l2;
  if (b < v && c <= b) {
    // t1 values by [occupied][tile position] and integrals by [slab][pair]
    double t[3][3], I[3][6];
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      t[w][1] = ts[w][1][l1];
      t[w][2] = ts[w][2][l2];
      I[w][pairpos(1, 2)] = It[w][pairpos(1, 2)][l1][l2];
      I[w][pairpos(2, 1)] = It[w][pairpos(2, 1)][l2][l1];
    }
    const double dbc = eo[i] + eo[j] + eo[k] - es[1][l1] - es[2][l2];
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      const int l0 = half + 2 * q, a = b0[0] + l0;
      if (a >= v || a < b) continue;
      const int l[3] = {l0, l1, l2};
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        t[w][0] = ts[w][0][l0];
        I[w][pairpos(0, 1)] = It[w][pairpos(0, 1)][l0][l1];
        I[w][pairpos(0, 2)] = It[w][pairpos(0, 2)][l0][l2];
        I[w][pairpos(1, 0)] = It[w][pairpos(1, 0)][l1][l0];
        I[w][pairpos(2, 0)] = It[w][pairpos(2, 0)][l2][l0];
      }
      double u[6];
#pragma unroll
      for (int s = 0; s < 6; ++s)
        u[s] = (double)cube[s][l[ordpos(s, 0)]][l[ordpos(s, 1)]][l[ordpos(s, 2)]];
      const double E = u[0] + u[3] + u[4], O = u[1] + u[2] + u[5];
      const double pe = 6.0 * E - 12.0 * O, po = 6.0 * O - 12.0 * E;
      double g4 = 0.0, g5 = 0.0;
#pragma unroll
      for (int s = 0; s < 6; ++s) {
        const int P0 = ordpos(s, 0), P1 = ordpos(s, 1), P2 = ordpos(s, 2);
        // V - W at (p0,p1,p2): t_i^p0 <jk|p1p2> + t_j^p1 <ik|p0p2> + t_k^p2 <ij|p0p1>
        const double vd = t[0][P0] * I[0][pairpos(P1, P2)] + t[1][P1] * I[1][pairpos(P0, P2)] +
                          t[2][P2] * I[2][pairpos(P0, P1)];
        const double y = 18.0 * u[s] + (s == 0 || s == 3 || s == 4 ? pe : po);
        g4 += y * u[s];
        g5 += y * vd;
      }
      const bool ab = a == b, bc = b == c;
      const double inv = (ab && bc ? 1.0 / 6.0 : (ab || bc ? 0.5 : 1.0)) / (dbc - es[0][l0]);
      s4 += g4 * inv;
      s5 += g5 * inv;
    }
  }
  for (int off = 16; off; off >>= 1) {
    s4 += __shfl_down_sync(0xffffffffu, s4, off);
    s5 += __shfl_down_sync(0xffffffffu, s5, off);
  }
  const int lane = tid & 31, wid = tid >> 5;
  if (lane == 0) {
    sh[0][wid] = s4;
    sh[1][wid] = s5;
  }
  __syncthreads();
  if (tid == 0) {
    double a4 = 0.0, a5 = 0.0;
    for (int w = 0; w < 4; ++w) {
      a4 += sh[0][w];
      a5 += sh[1][w];
    }
    const long long slot = (long long)e * gridDim.x + blockIdx.x;
    part[2 * slot] = scale * a4;
    part[2 * slot + 1] = scale * a5;
  }
}

// sum of n (E4, E5) partial pairs: 1024 threads stride the list, then a
// fixed-shape tree; the order of additions does not depend on timing
__global__ void __launch_bounds__(1024) k_sum_pairs(double *out, const double *part, long long n) {
  after_previous();
  double a = 0.0, b = 0.0;
  for (long long t = threadIdx.x; t < n; t += blockDim.x) {
    a += part[2 * t];
    b += part[2 * t + 1];
  }
  for (int off = 16; off; off >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, off);
    b += __shfl_down_sync(0xffffffffu, b, off);
  }
  __shared__ double sa[32], sb[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { sa[wid] = a; sb[wid] = b; }
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    a = lane < nw ? sa[lane] : 0.0;
    b = lane < nw ? sb[lane] : 0.0;
    for (int off = 16; off; off >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, off);
      b += __shfl_down_sync(0xffffffffu, b, off);
    }
    if (lane == 0) { out[0] = a; out[1] = b; }
  }
}
// Batch size of `slot`-byte W slots: up to 4 GB, and within a quarter of the
// free memory unless the buffer is already in the allocator's cache (asking the
// driver takes 0.1 to 70 ms on a machine that other processes allocate on: (T)
// of o = 8, v = 70 3.0 ms, but 3 to 77 from run to run with the question).
int batch_slots(double slot, int most) {
  int nb = (int)std::max(1.0, std::min((double)most, 4.0e9 / slot));
  if (dev_cached((size_t)(slot * nb))) return nb;
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    fr = 0;
  }
  return (int)std::max(1.0, std::min((double)nb, 0.25 * (double)fr / slot));
}
}  // namespace

// The 12 contractions of a triplet (6 permutations x 2 terms) fall into three
// classes by the position of the virtual that is not a pair index of the
// pair-side operands: class c (W index c on the t2/H side, pairs (a,b)),
// class a (pairs (b,c), index a) and class b (pairs (a,c), index b).  All four
// terms of a class share one output orientation, so each class is ONE
// tensor-core product with four K segments (2 x K = v, 2 x K = o); every
// output view has unit stride along m, the first class stores and the other
// two accumulate with RED.  Per class and segment (P = permutation of (ijk)):
//   class c:  t2[k,i] x Gv[j] (P4)   t2[k,j] x GvT[i] (P5)   -H[j,k] x t2P[i] (P0)   -H[i,k] x t2Q[j] (P2)
//   class a:  Gv[k] x t2[i,j] (P0)   GvT[j] x t2[i,k] (P1)   t2P[j] x -H[k,i] (P3)   t2Q[k] x -H[j,i] (P5)
//   class b:  Gv[k] x t2[j,i] (P2)   GvT[i] x t2[j,k] (P3)   t2P[i] x -H[k,j] (P1)   t2Q[k] x -H[i,j] (P4)
// with Gv[z][(b,c),d] = (bd|cz), GvT[z][(c,b),d] = Gv[z][(b,c),d],
// t2P[x][(a,b),l] = t2[x,l,a,b], t2Q[x][(b,a),l] = t2[x,l,a,b] and
// H[y,z][c,l] = (cz|yl).
//
// Split precision: the triplets run in batches.  Every operand of a class is a
// row window of one of six pre-split parent arrays, so a batch's class is ONE
// persistent tcgen05 launch over the tiles of all its triplets (the triplets'
// windows in a device table, W in FP32 -- below the BF16x3 products' own
// rounding), and one energy launch covers the batch.  The tile order (small
// side, then triplet, then large side) makes the concurrently running CTAs
// share the large operand's rows: a window used by several triplets of the
// batch (Gv[j] for every k of a pair (i,j), Gv[k] across pairs) is read from
// DRAM about once per launch instead of once per triplet.  Four launches per
// batch replace four per triplet.  The FP64 path batches the same way (FP64
// W slots, task tables of the FP64 contraction kernel).
int CCEngine::triples(double *e4, double *e5, double *seconds, int rank, int nranks) {
  const long long O = o, V = v;
  const long long V2 = V * V, V3 = V * V * V;
  cudaEvent_t t0 = nullptr, t1e = nullptr;
  DBuf Gv, GvT, t2P, t2Q, Hn, Wb, part, outp, dtrip, dent;
  SplitOperand sT2, sGv, sGvT, sHn, sT2P, sT2Q;
  // every exit, the error returns included, gives back the scratch and events
  struct Release {
    std::function<void()> f;
    ~Release() { f(); }
  } release_scratch{[&] {
    for (DBuf *b : {&Gv, &GvT, &t2P, &t2Q, &Hn, &Wb, &part, &outp, &dtrip, &dent}) {
      if (b->p) dev_free(b->p);
      b->p = nullptr;
    }
    for (SplitOperand *sp : {&sT2, &sGv, &sGvT, &sHn, &sT2P, &sT2Q}) {
      if (sp->hi) dev_free(sp->hi);
      sp->hi = sp->lo = nullptr;
    }
    if (t0) cudaEventDestroy(t0);
    if (t1e) cudaEventDestroy(t1e);
  }};
  ACES_CUDA(cudaEventCreate(&t0));
  ACES_CUDA(cudaEventCreate(&t1e));
  ACES_CUDA(cudaEventRecord(t0, st));
  const long long sv[4] = {V * V * V, V * V, V, 1};      // I_ovvv[m,a,e,f]
  const long long s3[4] = {O * O * V, O * V, V, 1};      // I_ooov[m,n,i,e]
  const long long st2[4] = {O * V * V, V * V, V, 1};     // t2[i,j,a,b]
  // Gv[k,b,c,d] = (bd|ck) = <bc|dk> = I_ovvv[k,d,c,b]; GvT[k,c,b,d] = Gv[k,b,c,d]
  ACES_TRY(alloc(Gv, O * V3, false));
  ACES_TRY(perm(Gv.p, o, v, v, v, 0.0, {PermTerm{I_ovvv.p, 1.0, {sv[0], sv[3], sv[2], sv[1]}}}));
  ACES_TRY(alloc(GvT, O * V3, false));
  ACES_TRY(perm(GvT.p, o, v, v, v, 0.0, {PermTerm{I_ovvv.p, 1.0, {sv[0], sv[2], sv[3], sv[1]}}}));
  // t2P[i,a,b,l] = t2[i,l,a,b]; t2Q[i,b,a,l] = t2[i,l,a,b]
  ACES_TRY(alloc(t2P, O * O * V2, false));
  ACES_TRY(perm(t2P.p, o, v, v, o, 0.0, {PermTerm{t2(), 1.0, {st2[0], st2[2], st2[3], st2[1]}}}));
  ACES_TRY(alloc(t2Q, O * O * V2, false));
  ACES_TRY(perm(t2Q.p, o, v, v, o, 0.0, {PermTerm{t2(), 1.0, {st2[0], st2[3], st2[2], st2[1]}}}));
  // Hn[j,k,c,l] = -(ck|jl) = -I_ooov[l,k,j,c] (the second terms enter with a minus sign)
  ACES_TRY(alloc(Hn, O * O * O * V, false));
  ACES_TRY(perm(Hn.p, o, o, v, o, 0.0, {PermTerm{I_ooov.p, -1.0, {s3[2], s3[1], s3[3], s3[0]}}}));
  // triplets i >= j >= k of this shard: index t (i, then j <= i, then k <= j)
  // with t % nranks == rank
  std::vector<int> trip;
  long long tix = 0;
  for (int i = 0; i < o; ++i)
    for (int j = 0; j <= i; ++j)
      for (int k = 0; k <= j; ++k, ++tix)
        if (tix % nranks == rank) {
          trip.push_back(i);
          trip.push_back(j);
          trip.push_back(k);
        }
  const int ntrip = (int)trip.size() / 3;
  ACES_TRY(alloc(outp, 2));
  ACES_TRY(alloc(dtrip, (trip.size() + 1) / 2 + 1));
  if (!trip.empty())
    ACES_CUDA(cudaMemcpyAsync(dtrip.p, trip.data(), trip.size() * sizeof(int),
                              cudaMemcpyHostToDevice, st));
  const int *d_trip = reinterpret_cast<const int *>(dtrip.p);
  const bool use_split = prec == ACES_PREC_BF16X3 && v >= 128;
  const CView vc{nullptr, kHugeView, 0, 1, V, V2, V};   // m = c, n = (a,b)
  const CView vcT{nullptr, kHugeView, 0, V, kHugeView, 0, 1};  // m = (a,b), n = c
  const CView va{nullptr, V, V, 1, kHugeView, 0, V2};   // m = (b,c), n = a
  const CView vb{nullptr, V, V2, 1, kHugeView, 0, V};   // m = (a,c), n = b
  long long nparts = 0;

  if (use_split) {
    ACES_TRY(split_pack(sT2, t2(), V, o * o * v, v, st));       // rows (x,y,alpha), K = d
    ACES_TRY(split_pack(sGv, Gv.p, V, o * v * v, v, st));       // rows (z,beta,gamma), K = d
    ACES_TRY(split_pack(sGvT, GvT.p, V, o * v * v, v, st));     // rows (z,gamma,beta), K = d
    ACES_TRY(split_pack(sHn, Hn.p, O, o * o * v, o, st));       // rows (y,z,gamma), K = l
    ACES_TRY(split_pack(sT2P, t2P.p, O, o * v * v, o, st));     // rows (x,alpha,beta), K = l
    ACES_TRY(split_pack(sT2Q, t2Q.p, O, o * v * v, o, st));     // rows (x,beta,alpha), K = l
    // the FP64 copies are not read again
    ACES_CUDA(cudaStreamSynchronize(st));
    for (DBuf *b : {&Gv, &GvT, &t2P, &t2Q}) {
      dev_free(b->p);
      b->p = nullptr;
    }
    const int nb = batch_slots((double)V3 * sizeof(float), std::max(ntrip, 1));
    ACES_TRY(alloc(Wb, (size_t)((V3 * nb + 1) / 2), false));  // FP32 slots in a double buffer
    // class c runs transposed on the 256 x 192 tiles (M = (a,b), N = c: the
    // ragged side is the one whose MMA N is cut to the live columns, where on
    // 128-row tiles M = c = v would leave 256 - v rows idle), and stores W
    // rows of v contiguous floats
    const SplitOperand Ac[4] = {sT2, sT2, sHn, sHn}, Bc[4] = {sGv, sGvT, sT2P, sT2Q};
    const bool c_wide = bf16x3_wide_applies(Bc, 4, v);
    // one entry per triplet and class: the windows of the four segments
    auto T2r = [&](int x, int y) { return (x * o + y) * v; };   // rows of sT2 / sHn
    auto Pr = [&](int z) { return z * v * v; };                  // rows of sGv/sGvT/sT2P/sT2Q
    std::vector<BatchEntry> ent((size_t)3 * ntrip);
    for (int t = 0; t < ntrip; ++t) {
      const int i = trip[3 * t], j = trip[3 * t + 1], k = trip[3 * t + 2];
      const long long coff = (long long)(t % nb) * V3;
      BatchEntry &c = ent[(size_t)3 * t], &a = ent[(size_t)3 * t + 1],
                 &b = ent[(size_t)3 * t + 2];
      c = c_wide ? BatchEntry{{Pr(j), Pr(i), Pr(i), Pr(j)},
                              {T2r(k, i), T2r(k, j), T2r(j, k), T2r(i, k)}, coff}
                 : BatchEntry{{T2r(k, i), T2r(k, j), T2r(j, k), T2r(i, k)},
                              {Pr(j), Pr(i), Pr(i), Pr(j)}, coff};
      a = BatchEntry{{Pr(k), Pr(j), Pr(j), Pr(k)},
                     {T2r(i, j), T2r(i, k), T2r(k, i), T2r(j, i)}, coff};
      b = BatchEntry{{Pr(k), Pr(i), Pr(i), Pr(k)},
                     {T2r(j, i), T2r(j, k), T2r(k, j), T2r(i, j)}, coff};
    }
    // entries of class q for triplets [t0, t0 + n) stored contiguously:
    // [class][triplet] on the device
    std::vector<BatchEntry> byclass((size_t)3 * ntrip);
    for (int q = 0; q < 3; ++q)
      for (int t = 0; t < ntrip; ++t) byclass[(size_t)q * ntrip + t] = ent[(size_t)3 * t + q];
    ACES_TRY(alloc(dent, (byclass.size() * sizeof(BatchEntry) + 7) / 8 + 1));
    if (!byclass.empty())
      ACES_CUDA(cudaMemcpyAsync(dent.p, byclass.data(), byclass.size() * sizeof(BatchEntry),
                                cudaMemcpyHostToDevice, st));
    const BatchEntry *d_ent = reinterpret_cast<const BatchEntry *>(dent.p);
    const SplitOperand Aa[4] = {sGv, sGvT, sT2P, sT2Q}, Ba[4] = {sT2, sT2, sHn, sHn};
    const int nt = (v + kTile - 1) / kTile;
    const int nblk = nt * (nt + 1) * (nt + 2) / 6;   // tile triples A >= B >= C
    ACES_TRY(alloc(part, (size_t)std::max(ntrip, 1) * nblk * 2, false));
    for (int t0b = 0; t0b < ntrip; t0b += nb) {
      const int n = std::min(nb, ntrip - t0b);
      CView cv = c_wide ? vcT : vc;
      cv.p = Wb.p;
      if (c_wide)
        ACES_TRY(gemm_nt_bf16x3_batched(Bc, Ac, 4, v * v, v, &byclass[(size_t)t0b], d_ent + t0b,
                                        n, 1.0, 0.0, cv, true, st));
      else
        ACES_TRY(gemm_nt_bf16x3_batched(Ac, Bc, 4, v, v * v, &byclass[(size_t)t0b],
                                        d_ent + t0b, n, 1.0, 0.0, cv, true, st));
      cv = va;
      cv.p = Wb.p;
      ACES_TRY(gemm_nt_bf16x3_batched(Aa, Ba, 4, v * v, v, &byclass[(size_t)ntrip + t0b],
                                      d_ent + ntrip + t0b, n, 1.0, 1.0, cv, true, st));
      cv = vb;
      cv.p = Wb.p;
      ACES_TRY(gemm_nt_bf16x3_batched(Aa, Ba, 4, v * v, v, &byclass[(size_t)2 * ntrip + t0b],
                                      d_ent + 2 * ntrip + t0b, n, 1.0, 1.0, cv, true, st));
      launch_after(k_triples_energy_tiled<float>, dim3(nblk, n), 128, 0, st,
                   reinterpret_cast<const float *>(Wb.p), V3, d_trip + 3 * t0b, t1(), I_oovv.p,
                   eo.p, ev.p, o, v, part.p + (size_t)t0b * nblk * 2);
      count_launch();
      ACES_CUDA(cudaGetLastError());
    }
    nparts = (long long)ntrip * nblk;
  } else {
    // FP64: the triplets in batches as above, W in FP64 slots; a class of a
    // batch is one launch over a table of tasks (four K segments each).  One
    // triplet at a time took 13 launches of about 10 us each at o = 8, v = 70:
    // 13.5 ms of kernels and 7 ms of gaps between them.
    const int nb =
        batch_slots((double)V3 * sizeof(double), std::min(std::max(ntrip, 1), kMaxTasks));
    ACES_TRY(alloc(Wb, V3 * nb, false));
    const int nt = (v + kTile - 1) / kTile;
    const int nblk = nt * (nt + 1) * (nt + 2) / 6;
    ACES_TRY(alloc(part, (size_t)std::max(ntrip, 1) * nblk * 2, false));
    auto T2p = [&](int x, int y) { return t2() + ((long long)x * o + y) * V * V; };
    auto Hp = [&](int y, int z) { return Hn.p + ((long long)y * o + z) * V * O; };
    auto Gp = [&](int z) { return Gv.p + (long long)z * V2 * V; };
    auto GTp = [&](int z) { return GvT.p + (long long)z * V2 * V; };
    auto Pp = [&](int x) { return t2P.p + (long long)x * V2 * O; };
    auto Qp = [&](int x) { return t2Q.p + (long long)x * V2 * O; };
    // C(view) = beta C + sum_s A_s B_s^T (K = v for the t2 x (bd|ck) segments, o
    // for the others)
    auto task = [&](const double *const (&A)[4], const double *const (&B)[4], int M, int N,
                    const CView &view, double *W) {
      F64Task t{};
      t.nseg = 4;
      t.M = M;
      t.N = N;
      t.C = view;
      t.C.p = W;
      for (int g = 0; g < 4; ++g) {
        const int K = g < 2 ? v : o;
        t.seg[g] = F64Seg{A[g], B[g], K, K, K};
      }
      return t;
    };
    std::vector<F64Task> tasks;
    ACES_TRY(alloc(dent, ((size_t)3 * nb * sizeof(F64Task) + 7) / 8));
    F64Task *d_tasks = reinterpret_cast<F64Task *>(dent.p);
    for (int t0b = 0; t0b < ntrip; t0b += nb) {
      const int n = std::min(nb, ntrip - t0b);
      tasks.resize((size_t)3 * n);
      for (int e = 0; e < n; ++e) {
        const int *x = &trip[3 * (size_t)(t0b + e)], i = x[0], j = x[1], k = x[2];
        double *W = Wb.p + (size_t)e * V3;
        tasks[e] = task({T2p(k, i), T2p(k, j), Hp(j, k), Hp(i, k)}, {Gp(j), GTp(i), Pp(i), Qp(j)},
                        v, v * v, vc, W);
        tasks[n + e] = task({Gp(k), GTp(j), Pp(j), Qp(k)}, {T2p(i, j), T2p(i, k), Hp(k, i), Hp(j, i)},
                            v * v, v, va, W);
        tasks[2 * n + e] = task({Gp(k), GTp(i), Pp(i), Qp(k)},
                                {T2p(j, i), T2p(j, k), Hp(k, j), Hp(i, j)}, v * v, v, vb, W);
      }
      F64TaskPlan plan[3];
      for (int q = 0; q < 3; ++q)
        ACES_TRY(f64_tasks_plan(tasks.data() + (size_t)q * n, n, &plan[q]));
      // the table is read by this batch's launches only: the copy waits for the
      // previous batch's (stream order), and the host vector is copied out
      ACES_CUDA(cudaMemcpyAsync(d_tasks, tasks.data(), tasks.size() * sizeof(F64Task),
                                cudaMemcpyHostToDevice, st));
      for (int q = 0; q < 3; ++q)
        ACES_TRY(f64_tasks_run(d_tasks + (size_t)q * n, n, plan[q], 1.0, q ? 1.0 : 0.0, st));
      launch_after(k_triples_energy_tiled<double>, dim3(nblk, n), 128, 0, st, Wb.p, V3,
                   d_trip + 3 * (size_t)t0b, t1(), I_oovv.p, eo.p, ev.p, o, v,
                   part.p + (size_t)t0b * nblk * 2);
      count_launch();
      ACES_CUDA(cudaGetLastError());
    }
    nparts = (long long)ntrip * nblk;
  }
  launch_after(k_sum_pairs, 1, 1024, 0, st, outp.p, part.p, nparts);
  count_launch();
  double h[2];
  ACES_CUDA(cudaMemcpyAsync(h, outp.p, 16, cudaMemcpyDeviceToHost, st));
  ACES_CUDA(cudaEventRecord(t1e, st));
  ACES_CUDA(cudaStreamSynchronize(st));
  if (int tcs = tc_status_and_clear()) {
    set_error("(T): tensor-core contraction gave up waiting (code %d)", tcs);
    return ACES_ERR_TIMEOUT;
  }
  float ms = 0.f;
  cudaEventElapsedTime(&ms, t0, t1e);
  *seconds = ms * 1e-3;
  *e4 = h[0];
  *e5 = h[1];
  if (!std::isfinite(*e4) || !std::isfinite(*e5)) {
    set_error("(T): non-finite energy");
    return ACES_ERR_NAN;
  }
  return ACES_OK;
}

}  // namespace acesb200
