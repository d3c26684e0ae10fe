// Stable radix sort of (key, 32-bit payload) pairs (sort_reduce.cu).
#pragma once
#include <cstdint>

#include "vlr_host.hpp"

namespace vlr {

// Scratch bytes of a sort of n pairs with keys of key_bytes (4 or 8).
size_t radix_scratch_bytes(int n, int key_bytes);
// Stable LSD radix sort by the low `bits` bits of the keys, enqueued on the
// context stream.  The sorted pairs end in either the input arrays or the
// scratch, as *keys_out / *vals_out report.
int radix_sort(vlr_ctx* ctx, unsigned* keys, unsigned* vals, int n, int bits, void* scratch, unsigned** keys_out,
               unsigned** vals_out);
int radix_sort(vlr_ctx* ctx, uint64_t* keys, unsigned* vals, int n, int bits, void* scratch, uint64_t** keys_out,
               unsigned** vals_out);

}  // namespace vlr
