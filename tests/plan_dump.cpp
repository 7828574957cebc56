// Prints the plan that a verify call would take, and the query lengths it
// admits, without a GPU: plan_dump <path 0|1> <min> <max> <candidates> <reads>
// <cut-off or -1> <multiprocessors> <PEQ entries> (min and max 0: no range announced). Or the lengths that a send
// sees in its queries, which are the given ones over and over: plan_dump lengths
// <queries> <mark each length 0|1> <length> <length> ..
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "myers_internal.h"

using namespace myers;

// Whether a candidate whose query has m rows is verified, as the kernels decide:
// in an unbucketed launch of one shape by its rows, else by its word count.
static bool admits(const PlanTable& p, bool unbucketed, uint32_t m) {
  if (p.row_limit > 0 && (m < p.row_min || m > p.row_limit)) return false;
  if (!unbucketed) return plan_cfg(p, m) != kNoCfg;
  const Shape s = p.shape[0];
  if (s.variant == kSlicedVariant) return p.row_limit > 0 || m <= (uint32_t)s.W << s.L;
  return m <= 32u * s.W * s.L;
}

static void print(const char* name, const PlanTable& p, bool unbucketed) {
  printf("\"%s\": {\"cfg\": %u, \"batched\": %u, \"sliced\": %u, \"spread\": %u, \"row_limit\": %u, \"unbucketed\": %d, \"shapes\": [", name,
         p.num_cfg, p.num_batched, p.num_sliced, p.spread, p.row_limit, (int)unbucketed);
  for (uint32_t c = 0; c < p.num_cfg; ++c) printf("%s[%u, %u, %u]", c ? ", " : "", p.shape[c].variant, p.shape[c].L, p.shape[c].W);
  printf("], \"admits\": [");  // first and last length of each run
  bool any = false;
  for (uint32_t m = 1, from = 0; m <= kMaxWords * 32 + 1; ++m) {
    const bool in = m <= kMaxWords * 32 && p.num_cfg > 0 && admits(p, unbucketed, m);
    if (in && from == 0) from = m;
    if (!in && from != 0) {
      printf("%s[%u, %u]", any ? ", " : "", from, m - 1);
      any = true;
      from = 0;
    }
  }
  printf("]}");
}

static int lengths(int argc, char** argv) {
  const uint32_t n = (uint32_t)atoi(argv[2]);
  const bool by_length = atoi(argv[3]) != 0;
  std::vector<qryInfo_t> queries(n);
  for (uint32_t q = 0; q < n; ++q) queries[q] = qryInfo_t{0, (uint32_t)strtoul(argv[4 + q % (argc - 4)], nullptr, 10)};
  std::vector<uint8_t> present(kMaxWords + 1, 7), present_m(kMaxWords * 32 + 1, 7);
  const Lengths l = scan_lengths(queries.data(), n, present.data(), present_m.data(), by_length);
  printf("{\"lo\": %u, \"hi\": %u, \"words\": [", l.lo, l.hi);
  for (uint32_t w = 0, any = 0; w <= kMaxWords; ++w)
    if (present[w]) printf("%s%u", any++ ? ", " : "", w);
  printf("], \"marked\": [");
  for (uint32_t m = 0, any = 0; by_length && m <= kMaxWords * 32; ++m)
    if (present_m[m]) printf("%s%u", any++ ? ", " : "", m);
  printf("]}\n");
  return 0;
}

int main(int argc, char** argv) {
  if (argc > 4 && strcmp(argv[1], "lengths") == 0) return lengths(argc, argv);
  if (argc != 9) return 2;
  const uint32_t sms = (uint32_t)atoi(argv[7]);
  const uint64_t entries = strtoull(argv[8], nullptr, 10);
  const bool batched = atoi(argv[1]) != 0;
  const uint32_t lo = (uint32_t)atoi(argv[2]), hi = (uint32_t)atoi(argv[3]);
  const uint64_t n = strtoull(argv[4], nullptr, 10), reads = strtoull(argv[5], nullptr, 10);
  const float cut = strtof(argv[6], nullptr);
  const uint32_t first = lo ? lo : 1, last = hi ? hi : kMaxWords * 32;
  PlanTable a, b;
  memset(&a, 0, sizeof(a));
  memset(&b, 0, sizeof(b));
  if (cut >= 0.0f) {
    std::vector<uint8_t> present(kMaxWords * 32 + 1, 0);
    for (uint32_t m = first; m <= last; ++m) present[m] = 1;
    if (cutoff_plans(a, b, present.data(), cut, cutoff_prefix_mult(), batched, n, sms, 0, hi == 0) != 0) return 1;
    const bool unbucketed = !batched && !a.bucketed;
    printf("{");
    print("first", a, unbucketed);
    printf(", ");
    print("second", b, unbucketed);
    printf("}\n");
    return 0;
  }
  if (plan_for_range(a, lo, hi, batched, n, reads, entries, sms) != 0) return 1;
  const bool unbucketed = sliced_alone(a) || (!batched && a.num_cfg == 1 && a.num_sliced == 0);
  printf("{");
  print("plan", a, unbucketed);
  printf("}\n");
  return 0;
}
