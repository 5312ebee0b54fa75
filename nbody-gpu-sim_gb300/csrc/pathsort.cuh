// pathsort.cuh -- bodies sorted by (segment, high path key, index) (pathsort.cu).
#pragma once

#include "bh_tree.cuh"
#include "pathkey.cuh"

namespace nbgb {

// Sorts of at most this many bodies; larger builds use the radix sort: beyond it the
// 1,024 buckets outgrow the shared memory of ps_local one by one, first in clustered
// sets.  Keys, sort and order, us, sample / radix sort (Plummer sphere; cube): 1M
// 174 / 227; 171 / 250, 1.31M 236 / 290; 214 / 342, 1.4M 242 / 306; 219 / 350, 1.7M
// 391 / 329; 282 / 382, 2M 427 / 356; 325 / 407.
constexpr int64_t kPathSortMax = 1310720;
constexpr int kPsMaxBuckets = 1024;
constexpr int64_t kPsMean = 192;  // bodies per bucket, until the buckets run out

// First bucket of each segment (nseg + 1 entries); the number of buckets, or 0
// where the radix sort has to be used (too many bodies or segments).
int path_sort_buckets(const int64_t* n_per, int nseg, int32_t* first);

struct PathSortBuffers {
  char* ws;            // path_sort_ws_bytes()
  u64* key;            // n, scratch: keys by body
  uint32_t* bucket;    // n, scratch
  u64* skey;           // n, scratch: keys by bucket
  uint32_t* sidx;      // n, scratch
  // results by sorted position
  uint32_t* body;
  int32_t* kseg;
  u64* hi;
  float4* spm;
};

size_t path_sort_ws_bytes();
size_t path_sort_zero_words();  // leading words of ws that are zero before a sort
// first: path_sort_buckets' table on the device, nb their number (above 0).
void path_sort(const float4* pm, const SegView& sv, const int32_t* first, int nb, int64_t n,
               int nseg, const PathSortBuffers& b, StageTimer* timer, cudaStream_t st);

}  // namespace nbgb
