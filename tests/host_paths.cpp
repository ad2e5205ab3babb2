// Cases of test_host_paths.py: one function each, run by name; 0 = passed.
#include "host_cuda.h"

#include <unistd.h>

#include <string>
#include <thread>

using namespace acesb200;

// dummy operand addresses: no kernel runs
static double *addr(size_t k) { return (double *)(0x100000000ull + (k << 32)); }

// launches of one product with `budget` bytes of device memory left; -1: it failed
static int product(int precision, int m, int n, int k, size_t budget) {
  host::launches.clear();
  pool_trim();
  host::budget = host::live + budget;
  const int rc = aces_xgemm('T', 'N', m, n, k, 1.0, addr(0), k, addr(1), k, 0.0, addr(2), m, precision);
  host::budget = ~size_t(0);
  return rc == ACES_OK ? (int)host::launches.size() : -1;
}

// Split products whose last wave is cut along K, and FP64 products with split
// K, run whole when their partial sums find no memory.
static int no_room_for_partials() {
  const size_t MB = size_t(1) << 20;
  // operand planes of 1300 x 4032 and 2200 x 4032 pairs of BF16, a little room
  const size_t planes = (1300 + 2200) * size_t(4032) * 4 + 4 * MB;
  CHECK(product(ACES_PREC_BF16X3, 1300, 2200, 4000, planes) == 3);
  CHECK(product(ACES_PREC_BF16X3, 1300, 2200, 4000, 8 * planes) == 4);   // and the reduction
  CHECK(product(ACES_PREC_FP64, 200, 150, 6000, 0) == 1);
  CHECK(product(ACES_PREC_FP64, 200, 150, 6000, 256 * MB) == 2);
  // the grouped launch, on operands at hand
  SplitOperand a, b;
  for (SplitOperand *x : {&a, &b}) {
    x->hi = addr(3);
    x->lo = addr(4);
    x->rows = x->rows_pad = 2200;
    x->k = x->k_pad = 4032;
  }
  const GroupedProblem pr[2] = {{&a, &b, 1, 1300, 2200, cview_colmajor(addr(5), 1300)},
                                {&a, &b, 1, 1300, 2200, cview_colmajor(addr(6), 1300)}};
  for (int room = 0; room < 2; ++room) {
    host::launches.clear();
    pool_trim();
    host::budget = host::live + (room ? 256 * MB : 0);
    int rc = 0;
    {
      CallScope call;
      rc = gemm_nt_bf16x3_grouped(pr, 2, 1.0, 0.0, 0);
    }
    CHECK(rc == ACES_OK);
    CHECK((int)host::launches.size() == 1 + room);
    host::budget = ~size_t(0);
  }
  return 0;
}

// Blocks given back during a call stay with its thread until the call has
// waited for its streams.
static int blocks_stay_with_their_call() {
  const size_t MB = size_t(1) << 20;
  cudaStream_t st;
  cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  void *q = nullptr, *own = nullptr, *a = nullptr, *b = nullptr;
  double *p = nullptr;
  {
    CallScope call;
    call.also(&st);
    p = splitk_workspace(1000);
    CHECK(p && dev_alloc(&q, MB) == cudaSuccess);
    host::launch(nullptr, st, dim3(1), true);   // reads both
    CHECK(splitk_workspace(1000) == p && splitk_workspace(8 * MB) != p);
    dev_free(q);
    std::thread([&] {
      dev_alloc(&a, 8000);
      dev_alloc(&b, MB);
    }).join();
    CHECK(a && b && a != p && b != q);
    CHECK(dev_alloc(&own, MB) == cudaSuccess && own == q);
    dev_free(own);
    CHECK(host::pending[st] == 1);
  }
  CHECK(host::pending[st] == 0);
  std::thread([&] { dev_alloc(&b, MB); }).join();
  CHECK(b == q);
  return 0;
}

// a system of o occupied and v virtual orbitals, its lists filled with zeros
static int small_system(int o, int v) {
  const int list[6][3] = {{13, 14, 14}, {10, 14, 18}, {16, 13, 14},
                          {25, 11, 11}, {30, 13, 11}, {233, 13, 13}};
  int rc = aces_init(0);
  if (rc == ACES_OK) rc = aces_sym_init(1, &o, &v);
  for (auto &l : list)
    if (rc == ACES_OK) rc = aces_inipck(1, l[1], l[2], l[0], 1);
  std::vector<double> eps(o + v);
  for (int i = 0; i < o + v; ++i) eps[i] = i < o ? -1.0 : 1.0 + i;
  return rc == ACES_OK ? aces_putrec("SCFEVALA", (long long)eps.size() * 8, eps.data()) : rc;
}

// Every entry point that launches does so inside a call, and no stream is left
// running when it returns, an error included.
static int entry_points_wait() {
  int outside = 0;
  host::on_launch = [&] { outside += call_workspace(1) == nullptr; };
  auto idle = [] {
    for (auto &s : host::pending)
      if (s.second) return false;
    return true;
  };
  std::vector<double> B(30 * 14 * 14, 0.1);
  aces_cc_config cc{};
  cc.cc_conv = 7;
  cc.cc_maxcyc = 5;
  cc.cc_exporder = 5;
  CHECK(small_system(4, 10) == ACES_OK);
  CHECK(aces_intprc_df(B.data(), 30, 0) == ACES_OK && idle());
  for (int prec : {ACES_PREC_FP64, ACES_PREC_BF16X3}) {
    cc.precision = prec;
    cc.triples = 1;
    CHECK(xvcc_run(&cc) == ACES_OK && idle());
    CHECK(xlambda_run(&cc) == ACES_OK && idle());
    CHECK(xdens_1pdm(&cc) == ACES_OK && idle());
    CHECK(aces_xgemm('N', 'T', 200, 150, 6000, 1.0, addr(0), 200, addr(1), 150, 0.0, addr(2), 200,
                     prec) == ACES_OK && idle());
  }
  aces_eom_config eom{};
  eom.nroots[0] = 1;
  eom.eom_conv = 5;
  eom.eom_maxcyc = 2;
  const int ee = xvee_run(&eom);
  CHECK((ee == ACES_OK || ee == ACES_ERR_NOCONV) && idle());
  CHECK(outside == 0);
  // out of memory somewhere in the solve
  const size_t n0 = host::launches.size();
  int failed = 0;
  for (size_t room = 1; room < 64; room += 4) {
    CHECK(small_system(8, 40) == ACES_OK);
    pool_trim();
    host::budget = host::live + (room << 20);
    failed += xvcc_run(&cc) == ACES_ERR_NOMEM;
    host::budget = ~size_t(0);
    CHECK(idle());
  }
  CHECK(failed > 2 && host::launches.size() > n0);
  host::on_launch = [] {};
  return 0;
}

// The first kernel of a call waits in plain stream order for whatever the
// caller launched before it; the later ones may be set up early.
static int first_launch_in_order() {
  auto ordered = [](size_t n) {
    if (host::launches.size() < n || host::launches[0].overlapped) return false;
    for (size_t i = 1; i < host::launches.size(); ++i)
      if (!host::launches[i].overlapped) return false;
    return true;
  };
  for (int prec : {ACES_PREC_FP64, ACES_PREC_BF16X3})
    for (int rep = 0; rep < 2; ++rep) {
      host::launches.clear();
      CHECK(aces_xgemm('N', 'T', 200, 150, 6000, 1.0, addr(0), 200, addr(1), 150, 0.0, addr(2), 200,
                       prec) == ACES_OK);
      CHECK(ordered(3));
      host::launches.clear();
      CHECK(aces_xgemm_static('N', 'T', 200, 150, 600, 1.0, addr(0), 200, addr(1), 150, 0.0,
                              addr(2), 200) == ACES_OK);
      CHECK(ordered(2));
    }
  std::vector<double> B(30 * 14 * 14, 0.0);
  CHECK(small_system(4, 10) == ACES_OK);
  host::launches.clear();
  CHECK(aces_intprc_df(B.data(), 30, 0) == ACES_OK);
  CHECK(ordered(3));
  return 0;
}

// A producer that fails leaves zeros in the lists it has created, not old
// device memory, and lists that were there as they were.
static int failed_producer_leaves_zeros() {
  const int o = 4, v = 30, n = o + v, naux = 30, list[6] = {13, 10, 16, 25, 30, 233};
  const size_t MB = size_t(1) << 20;
  std::vector<double> B((size_t)naux * n * n, 0.0);
  for (int there = 0; there < 2; ++there) {
    CHECK(aces_init(0) == ACES_OK && aces_sym_init(1, &o, &v) == ACES_OK);
    pool_trim();
    if (there) CHECK(small_system(o, v) == ACES_OK);
    std::vector<double> two((size_t)o * o, 2.0);
    if (there) CHECK(aces_putlst(two.data(), 1, 1, 1, 13) == ACES_OK);
    // room for the lists' memory and for nothing else of size
    host::budget = host::live + (there ? 0 : 256 * MB) + MB / 8;
    CHECK(aces_intprc_df(B.data(), naux, 1) == ACES_ERR_NOMEM);
    host::budget = ~size_t(0);
    for (int l : list) {
      int nc = 0, nr = 0;
      CHECK(aces_list_dims(1, l, &nc, &nr) == ACES_OK && nc > 0 && nr > 0);
      std::vector<double> x((size_t)nc * nr, 1.0);
      CHECK(aces_getlst(x.data(), 1, nc, 1, l) == ACES_OK);
      for (size_t i = 0; i < x.size(); ++i)
        CHECK(x[i] == (there && l == 13 && i < two.size() ? 2.0 : 0.0));
    }
  }
  return 0;
}

// a batched FP32-output launch of 40 entries with K = 64; the launch, or
// nullptr when it failed
static const host::Launch *batched(int N, const CView &C, double beta = 0.0) {
  SplitOperand a, b;
  for (SplitOperand *x : {&a, &b}) {
    x->hi = addr(3);
    x->lo = addr(4);
    x->rows = x->rows_pad = 40000;
    x->k = x->k_pad = 64;
  }
  std::vector<BatchEntry> e(40);
  for (int i = 0; i < 40; ++i) e[i] = BatchEntry{{i}, {i}, 0};
  host::launches.clear();
  CallScope call;
  const int rc = gemm_nt_bf16x3_batched(&a, &b, 1, 600, N, e.data(), e.data(), 40, 1.0, beta, C,
                                        true, 0);
  return rc == ACES_OK && !host::launches.empty() ? &host::launches.back() : nullptr;
}

// The wide tiles take outputs with unit m stride or whole contiguous rows; a
// view that splits n runs on the other tiles.
static int wide_tiles_need_plain_rows() {
  const long long plain = 1LL << 62;
  const CView rows{addr(5), plain, 0, 170, plain, 0, 1}, cols{addr(5), 600, 0, 1, plain, 0, 600},
      split{addr(5), plain, 0, 170, 10, 100, 1};
  const host::Launch *l;
  CHECK((l = batched(170, rows)) && l->cluster);
  CHECK((l = batched(170, cols)) && l->cluster);
  CHECK((l = batched(170, split)) && !l->cluster);
  return 0;
}

// Tile choices of batched launches: widths that the wide tiles serve and widths
// that they do not are different classes, and a saved choice of the wide tiles
// is not applied to the latter.
static int tile_choices_by_width() {
  const long long plain = 1LL << 62;
  const CView cols{addr(5), plain, 0, 1, plain, 0, 600};
  const int others[2][2] = {{100, 140}, {220, 170}};   // not served, served: as many 144-wide tiles
  for (auto &w : others) {
    aces_set_autotune(2);
    aces_set_autotune(1);
    long long n[3] = {0, 0, 0}, changed;
    double ms;
    CHECK(batched(w[0], cols));
    aces_autotune_stats(&n[0], &changed, &ms);
    CHECK(batched(w[1], cols));
    aces_autotune_stats(&n[1], &changed, &ms);
    CHECK(n[0] == 1 && n[1] == 2);
    // the file takes the choices through save and load, and one of the wide tiles
    // for every class of batched launches keeps to the widths they serve
    char path[] = "/tmp/tile_choicesXXXXXX";
    CHECK(mkstemp(path) >= 0 && aces_autotune_save(path) == ACES_OK);
    FILE *f = std::fopen(path, "r");
    std::string text;
    for (int c; (c = std::fgetc(f)) != EOF;) text += (char)c;
    std::fclose(f);
    for (size_t at; (at = text.find(" 1 0 0 0\n")) != std::string::npos;)
      text.replace(at, 9, " 1 256 0 1\n");
    f = std::fopen(path, "w");
    std::fputs(text.c_str(), f);
    std::fclose(f);
    aces_set_autotune(2);
    CHECK(aces_autotune_load(path) == ACES_OK);
    aces_autotune_stats(&n[2], &changed, &ms);
    CHECK(n[2] == 2 && changed == 2);
    const host::Launch *l;
    CHECK((l = batched(w[0], cols)) && !l->cluster);
    CHECK((l = batched(w[1], cols)) && l->cluster);
    std::remove(path);
    aces_set_autotune(0);
    aces_set_autotune(2);
  }
  return 0;
}

// A task table with an empty K segment is refused (the kernel would take a tile
// of the next segment for it).
static int empty_segments_are_refused() {
  for (int empty = -1; empty < 3; ++empty) {
    F64Task t{};
    t.nseg = 3;
    t.M = t.N = 40;
    t.C = cview_colmajor(addr(5), 40);
    for (int s = 0; s < 3; ++s) t.seg[s] = F64Seg{addr(0), addr(1), 50, 50, s == empty ? 0 : 50};
    F64TaskPlan plan;
    CHECK((f64_tasks_plan(&t, 1, &plan) == ACES_OK) == (empty < 0));
  }
  return 0;
}

struct Case {
  const char *name;
  int (*run)();
};
static const Case cases[] = {
    {"no_room_for_partials", no_room_for_partials},
    {"blocks_stay_with_their_call", blocks_stay_with_their_call},
    {"entry_points_wait", entry_points_wait},
    {"first_launch_in_order", first_launch_in_order},
    {"failed_producer_leaves_zeros", failed_producer_leaves_zeros},
    {"wide_tiles_need_plain_rows", wide_tiles_need_plain_rows},
    {"tile_choices_by_width", tile_choices_by_width},
    {"empty_segments_are_refused", empty_segments_are_refused},
};

int main(int argc, char **argv) {
  for (const Case &c : cases)
    if (argc == 2 && !std::strcmp(argv[1], c.name)) return c.run();
  return 2;
}
