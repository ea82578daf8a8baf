// Stable LSD radix sort of (uint64 key, uint32 value) pairs (sort.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <utility>
#include <cuda_runtime.h>

namespace nbg
{
    // What launching the sorts takes on the current device: made once by each context that
    // sorts. A kernel's shared-memory limit belongs to a device and a CUDA context, so one opt-in
    // a process would leave the sorts of a second device without it.
    struct SortSetup
    {
        int sms = 0;            // 0: not made yet
        int whole_per_sm = 0;   // resident CTAs of the sort in one launch
    };
    cudaError_t setup_sort(SortSetup* setup);

    // Temporary bytes radix_sort_pairs needs for n pairs.
    size_t sort_temp_bytes(size_t n);

    // The bytes at its start (a multiple of 16) that are zero before a sort of n pairs.
    size_t sort_zero_bytes(size_t n);

    // Sort by bits [begin_bit, end_bit) of the key, 9 bits per pass, ping-ponging between
    // (keys, vals) and (keys_alt, vals_alt). *in_alt tells which pair holds the result.
    // n < 2^31. A look-back wait that gives up (it cannot, unless the device is broken) ORs
    // DEV_ERR_TIMEOUT into *err. early: as in launch_after.
    cudaError_t radix_sort_pairs(uint64_t* keys, uint32_t* vals, uint64_t* keys_alt, uint32_t* vals_alt,
                                 size_t n, int begin_bit, int end_bit, void* temp, cudaStream_t stream,
                                 uint64_t* launches, bool* in_alt, unsigned* err, bool early,
                                 const SortSetup& setup);

    // The same sort in one launch, done only when *run_if is not 0 on the device (the host
    // need not know); the result is in (keys, vals). For a call after radix_sort_pairs on the
    // same temp and n, with at most pass_base passes: both use the 16 passes' tickets,
    // histograms and published counts.
    cudaError_t radix_sort_if(uint64_t* keys, uint32_t* vals, uint64_t* keys_alt, uint32_t* vals_alt, size_t n,
                              int begin_bit, int end_bit, void* temp, int pass_base, cudaStream_t stream,
                              uint64_t* launches, unsigned* err, const unsigned* run_if, const SortSetup& setup);
}
