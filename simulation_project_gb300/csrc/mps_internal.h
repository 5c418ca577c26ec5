// mps_internal.h - declarations shared between the translation units of the library.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "../../include/mps_types.h"

namespace mps {

// radix sort (sort.cu).  Scratch: barrier words, key ranges, digit totals, digit counts of
// every CTA, alternate key and value arrays.
constexpr int kRadixDigitBits = 9;
constexpr int kRadixMaxCtas = 304;
constexpr long long kRadixTwoPerSm = 2500000;
// CTAs of a sort: up to 4,096 keys one (no grid barriers), then one per 1,024 keys, one per SM
// at most, or two where memory bounds it
constexpr int radix_ctas_for(long long n) {
    const int most = n < kRadixTwoPerSm ? kRadixMaxCtas / 2 : kRadixMaxCtas;
    return n <= 4096 ? 1 : (n + 1023) / 1024 < most ? (int)((n + 1023) / 1024) : most;
}
constexpr size_t radix_scratch_bytes_for(long long n, int max_ctas = kRadixMaxCtas) {
    const size_t ctas = (size_t)(radix_ctas_for(n) < max_ctas ? radix_ctas_for(n) : max_ctas);
    return sizeof(unsigned) * (8 + 2 * ctas + ((size_t)1 << kRadixDigitBits) * (ctas + 1)) +
           sizeof(int) * 2 * (size_t)(n > 0 ? n : 0);
}
inline size_t radix_scratch_bytes(int n) { return radix_scratch_bytes_for(n); }
// bits of the keys 0 .. range
int radix_bits(unsigned range);
// Bits of a solver's error word that its host side keeps to itself (not MPS_ERR_*): a grid
// barrier of the sort of its particles, of its wall bins ran out.
constexpr unsigned kErrSortParticles = 1u << 30, kErrSortBins = 1u << 29;
// stable sort of (keys, vals) by key; bits: the keys lie in [0, 2^bits), < 0: any int range.
// *err gets `bit` if a grid barrier runs out.  The arrays' contents are then undefined (pairs
// lost, repeated or never written): nothing may use them as indexes before it has seen that
// *err is clear.
cudaError_t radix_sort_pairs(int n, int* keys, int* vals, int bits, void* scratch, unsigned* err, unsigned bit,
                             cudaStream_t st, int max_ctas = kRadixMaxCtas);
// polls of a grid barrier's wait, in the kernels of sort.cu and of solver.cu
cudaError_t sort_barrier_polls(int polls);
cudaError_t solver_barrier_polls(int polls);
// in-place exclusive scan of len unsigned values, total to *total_dev (if not NULL);
// tile_sums (scan_tile_sums_capacity() values, or NULL: single-CTA scan) lets it
// run on many CTAs
cudaError_t scan_exclusive(unsigned* a, int len, unsigned* total_dev, cudaStream_t st, unsigned* tile_sums = nullptr);
size_t scan_tile_sums_capacity();

// library-owned scratch for the reference-named entry points, which take no scratch
// argument (runtime.cu).  Grows on demand; one buffer per slot, and no slot belongs to two
// of the users below.
void* scratch_get(int slot, size_t bytes);
// A call's turn with its user's scratch: one host thread at a time, and on the GPU after the
// work that the turn before queued on its own stream, so calls on several streams do not
// overwrite each other's buffers.  Without a stream only the host threads take turns (the
// call has waited for its own work by then).  A turn lasts through the call's host waits, so
// each user has its own: a thread that sorts does not wait for one that bins triangles.
class ScratchTurn {
public:
    enum User { kSort, kOutside, kTriangles, kUsers };
    explicit ScratchTurn(User user);
    ScratchTurn(User user, cudaStream_t st);
    ~ScratchTurn();
    ScratchTurn(const ScratchTurn&) = delete;
    ScratchTurn& operator=(const ScratchTurn&) = delete;

private:
    User user_;
    cudaStream_t st_ = nullptr;
    bool on_stream_ = false;
};
// records "where: CUDA error string" for mps_last_error()
void note_error(const char* where, cudaError_t e);
// records a message of the library's own for mps_last_error()
void note_message(const char* msg);

// Kernel launches issued by this library since load (every launch site is written as
// MPS_COUNT_LAUNCH k<<<...>>>(...); read by mps_kernel_launches()).
extern unsigned long long g_kernel_launches;
#define MPS_COUNT_LAUNCH __atomic_fetch_add(&::mps::g_kernel_launches, 1ull, __ATOMIC_RELAXED),
void scratch_release_all();

// a cooperative launch that its stream or context has no room for (its SMs are a part of the
// GPU's) or does not do: not an error of the call, which then takes another way
inline bool coop_refused(cudaError_t e) {
    if (e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorNotSupported) return false;
    cudaGetLastError();
    return true;
}

inline CCTStatusType cuda_status(cudaError_t e) { return e == cudaSuccess ? CCT_NOERR : CCT_CUDAERR; }

}  // namespace mps

#define MPS_CUDA_TRY(expr)                                  \
    do {                                                    \
        cudaError_t _e = (expr);                            \
        if (_e != cudaSuccess) return CCT_CUDAERR;          \
    } while (0)
