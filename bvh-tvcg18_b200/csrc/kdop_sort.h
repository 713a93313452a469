// kdop_sort.h -- sizes of the device radix sort (kdop_sort.cuh), the exclusive
// scan and the ordering of a traversal's results (kdop_sort.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace kdop {

constexpr int64_t kSortTile = 4096;  // keys per block and pass

// Words of scratch a radix sort of n keys needs.
size_t radix_scratch_words(int64_t n);
// Words of scratch exclusive_scan_u32 needs for n counts (8-byte aligned).
size_t scan_scratch_words(int64_t n);
// out[i] = in[0] + ... + in[i-1] (in == out allowed).
cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* scratch, cudaStream_t st);

}  // namespace kdop

struct kdop_scene;
namespace kdop {
// Sorts the last traversal's n candidate rows by (pair, tet of A, tet of B)
// and, after kdop_contacts, regroups the n_contacts contact rows and the
// records in that order.  work: sort_results_bytes(n, n_contacts) bytes.  A
// bounded wait that gave up sets DEV_ERR_TIMEOUT in the scene's control block;
// the results are then lost.
cudaError_t sort_results(kdop_scene* s, int64_t n, int64_t n_contacts, void* work);
size_t sort_results_bytes(int64_t n, int64_t n_contacts);
}  // namespace kdop
