// Cases of test_host_paths.py: one function each, run by name; 0 = passed.
#include "host_cuda.h"

#include <thread>

using namespace acesb200;

// dummy operand addresses: no kernel runs
static double *addr(size_t k) { return (double *)(0x100000000ull + (k << 32)); }

// launches of one product with `budget` bytes of device memory left; -1: it failed
static int product(int precision, int m, int n, int k, size_t budget) {
  host::launches.clear();
  pool_trim();
  host::budget = host::live + budget;
  int rc = 0;
  std::thread([&] {  // a thread that holds no workspace yet
    rc = aces_xgemm('T', 'N', m, n, k, 1.0, addr(0), k, addr(1), k, 0.0, addr(2), m, precision);
  }).join();
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
    std::thread([&] { rc = gemm_nt_bf16x3_grouped(pr, 2, 1.0, 0.0, 0); }).join();
    CHECK(rc == ACES_OK);
    CHECK((int)host::launches.size() == 1 + room);
    host::budget = ~size_t(0);
  }
  return 0;
}

struct Case {
  const char *name;
  int (*run)();
};
static const Case cases[] = {
    {"no_room_for_partials", no_room_for_partials},
};

int main(int argc, char **argv) {
  for (const Case &c : cases)
    if (argc == 2 && !std::strcmp(argv[1], c.name)) return c.run();
  return 2;
}
