// Candidate list lengths the merge refuses: which ones (host), and, with the
// argument "gpu", that a merge over such lengths reads the other lists alone and
// reports the fault in the status word.
#include <cstdio>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "fused_knn.h"

using namespace curplsh_b200;

#define CHECK(x)                                             \
  do {                                                       \
    if (!(x)) {                                              \
      printf("failed at line %d: %s\n", __LINE__, #x);       \
      return 1;                                              \
    }                                                        \
  } while (0)

namespace {

constexpr int kCap = 64, kLists = 4, kDim = 8, kRows = 1024, kK = 4;

template <class T>
T* to_device(const std::vector<T>& v) {
  T* p = nullptr;
  if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess) return nullptr;
  cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return p;
}

// One query, four lists of capacity 64; list 0 holds rows 3 and 9, list 2 row 5.
int merge(const std::vector<int>& counts, std::vector<int>* idx, uint32_t* status) {
  std::vector<uint64_t> pools(kLists * kCap, 0);
  pools[0] = (uint64_t)0x80000000u << 32 | 3u;
  pools[1] = (uint64_t)0x80000000u << 32 | 9u;
  pools[2 * kCap] = (uint64_t)0x80000000u << 32 | 5u;
  std::vector<float> rows((size_t)kRows * kDim), query(kDim, 0.f);
  for (int i = 0; i < kRows; ++i)
    for (int c = 0; c < kDim; ++c) rows[(size_t)i * kDim + c] = (float)i;
  MergeLaunch m{};
  m.nq = 1;
  m.nb = kRows;
  m.d = kDim;
  m.k = kK;
  m.kprime = kK;
  m.pool_cap = kCap;
  m.plan.num_qblocks = 1;
  m.plan.num_tiles = kLists;
  m.plan.work_per_cta = kLists;
  m.plan.units_per_block = kLists;
  m.plan.split_tiles = 1;
  m.pools = to_device(pools);
  m.pool_counts = to_device(counts);
  m.q_bound = to_device(std::vector<uint32_t>(1, 0xFFFFFFFFu));
  m.queries = to_device(query);
  m.db = to_device(rows);
  m.ld_db = kDim;
  m.out_idx = to_device(std::vector<int>(kK, -7));
  m.out_dist = to_device(std::vector<float>(kK, -7.f));
  m.status = to_device(std::vector<uint32_t>(1, 0u));
  CHECK(m.pools && m.pool_counts && m.q_bound && m.queries && m.db && m.out_idx && m.out_dist && m.status);
  CHECK(launch_merge_rerank(m, nullptr) == cudaSuccess);
  CHECK(cudaDeviceSynchronize() == cudaSuccess);
  idx->resize(kK);
  cudaMemcpy(idx->data(), m.out_idx, kK * sizeof(int), cudaMemcpyDeviceToHost);
  cudaMemcpy(status, m.status, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  CHECK(pool_count_valid(0, kCap) && pool_count_valid(1, kCap) && pool_count_valid(kCap, kCap));
  CHECK(!pool_count_valid(-1, kCap) && !pool_count_valid(kCap + 1, kCap));
  CHECK(!pool_count_valid(0x7fffffff, kCap) && !pool_count_valid((int)0x80000000u, kCap));
  if (argc > 1 && !strcmp(argv[1], "gpu")) {
    std::vector<int> idx;
    uint32_t status = 0;
    CHECK(merge({2, 0, 1, 0}, &idx, &status) == 0);
    CHECK(status == kErrNone && idx == std::vector<int>({3, 5, 9, -1}));
    CHECK(merge({2, -1, 0x7fffffff, kCap + 1}, &idx, &status) == 0);
    CHECK(status == kErrBadSchedule && idx == std::vector<int>({3, 9, -1, -1}));
  }
  printf("merge counts ok\n");
  return 0;
}
