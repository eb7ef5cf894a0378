// Hole fill after a move (removal compaction).
//
// Holes are the set bits of the removal bitmap the move kernels write (one 32-bit
// word per warp of particles).  The k-th hole in ascending order is paired with the
// k-th live particle counted from the back; pairs are kept while the live particle
// lies behind the hole and k < remove_count.  Both sequences are monotone, so the
// kept pairs are a prefix: exactly the pairs of the reference's sequential loop
// (opp_lib/src/core/opp_particle_organize_core.cpp:124-218).
//   1. per-block hole counts over the bitmap,
//   2. emit hole[k] and mover[k] for k < remove_count (ranks from the counts, which every block
//      sums itself up to kHfDirectBlocks blocks, else from an exclusive scan of them),
//   3. copy every dat element mover[k] -> hole[k] for the kept pairs.

#include <climits>
#include <mutex>

#include "oppb_graph.h"
#include "scan.cuh"

namespace oppb {
namespace {

constexpr int kHfBlock = 256;
constexpr int kHfWordsPerThread = 2;
constexpr int kHfWords = kHfBlock * kHfWordsPerThread;  // words per block (16,384 particles)
constexpr int kMaxDats = 16;

struct DatList {
    int32_t n;
    int32_t total_cols;
    void* data[kMaxDats];
    int32_t dim[kMaxDats];
    int32_t bytes[kMaxDats];
};

// A count of a launch: the host's value, or (dev != nullptr) the value in device memory plus
// `add`, capped by the host's value, which is then its upper bound (include/oppb_graph.h).
struct CountArg {
    int32_t host;
    const int32_t* dev;
    int32_t add;
};

__device__ __forceinline__ int32_t resolve(const CountArg& c) {
    if (!c.dev) return c.host;
    const int32_t v = *c.dev + c.add;
    return v < 0 ? 0 : (v < c.host ? v : c.host);
}

// Bitmap word w restricted to particles < size.
__device__ __forceinline__ uint32_t hole_word(const uint32_t* bits, int64_t w, int32_t size) {
    const int64_t first = w * 32;
    if (first >= size) return 0u;
    uint32_t v = bits[w];
    const int64_t valid = size - first;
    if (valid < 32) v &= (1u << valid) - 1u;
    return v;
}

__global__ void __launch_bounds__(kHfBlock) hf_count_kernel(const uint32_t* __restrict__ bits, CountArg size_arg,
                                                            int64_t n_words, int* __restrict__ block_holes) {
    __shared__ int sm[kHfBlock / 32 + 1];
    const int32_t size = resolve(size_arg);
    const int64_t w0 = (int64_t)blockIdx.x * kHfWords;
    int c = 0;
#pragma unroll
    for (int k = 0; k < kHfWordsPerThread; k++) {
        const int64_t w = w0 + (int64_t)k * kHfBlock + threadIdx.x;
        if (w < n_words) c += __popc(hole_word(bits, w, size));
    }
    int total;
    block_exclusive_scan(c, sm, &total);
    if (threadIdx.x == 0) block_holes[blockIdx.x] = total;
}

// Emits the pairs' two sides.  block_holes: with kScanned the exclusive hole prefix per block and,
// at [n_blocks], the total H; else the blocks' hole counts, which every block sums up to itself
// (and to H): up to kHfDirectBlocks blocks that costs less than the scan's launch.  *total_out
// receives H for the copy kernel.
//
// Latency-bound: thousands of threads do nothing but the few over the holes and the last live
// particles, so what counts is the longest thread.  After the block's scan the words' prefixes go
// through shared memory and each thread takes single bytes: at most eight particles one after
// the other instead of 64 (460k particles, 2,000 removals: 4.4 us instead of 6.0).
template <bool kScanned>
__global__ void __launch_bounds__(kHfBlock) hf_emit_kernel(const uint32_t* __restrict__ bits, CountArg size_arg,
                                                           int64_t n_words, const int* __restrict__ block_holes,
                                                           int n_blocks, CountArg remove_arg,
                                                           int32_t* __restrict__ hole_list,
                                                           int32_t* __restrict__ mover_list, int* total_out) {
    __shared__ int sm[kHfBlock / 32 + 1];
    __shared__ uint32_t s_word[kHfWords];
    __shared__ int s_before[kHfWords];  // holes of the set before the word
    const int32_t size = resolve(size_arg);
    const int32_t remove_count = resolve(remove_arg);
    int base, H;
    if (kScanned) {
        base = block_holes[blockIdx.x];
        H = block_holes[n_blocks];
    } else {
        int before = 0, all = 0;
        for (int b = threadIdx.x; b < n_blocks; b += kHfBlock) {
            const int c = block_holes[b];
            all += c;
            before += b < (int)blockIdx.x ? c : 0;
        }
        block_exclusive_scan(before, sm, &base);
        block_exclusive_scan(all, sm, &H);
        if (blockIdx.x == 0 && threadIdx.x == 0) *total_out = H;
    }
    // Thread t owns kHfWordsPerThread consecutive words (blocked, so ranks follow index order).
    const int64_t w0 = (int64_t)blockIdx.x * kHfWords;
    const int t0 = threadIdx.x * kHfWordsPerThread;
    uint32_t w[kHfWordsPerThread];
    int c = 0;
#pragma unroll
    for (int k = 0; k < kHfWordsPerThread; k++) {
        w[k] = (w0 + t0 + k < n_words) ? hole_word(bits, w0 + t0 + k, size) : 0u;
        c += __popc(w[k]);
    }
    int total;
    int before = block_exclusive_scan(c, sm, &total) + base;
    // No pair lies in this block: no hole, and its last particle is not among the last
    // remove_count live ones (live particles behind the block: all behind it less its holes).
    const int64_t live_total = (int64_t)size - H;
    const int64_t first0 = w0 * 32;
    const int64_t behind = first0 + (int64_t)kHfWords * 32 < size ? size - (first0 + (int64_t)kHfWords * 32) : 0;
    const int64_t live_behind = behind - ((int64_t)H - base - total);
    if ((total == 0 || base >= remove_count) && live_behind >= remove_count) return;
#pragma unroll
    for (int k = 0; k < kHfWordsPerThread; k++) {
        s_word[t0 + k] = w[k];
        s_before[t0 + k] = before;
        before += __popc(w[k]);
    }
    __syncthreads();
#pragma unroll 1
    for (int e = threadIdx.x; e < kHfWords * 4; e += kHfBlock) {
        const uint32_t word = s_word[e >> 2];
        const int shift = (e & 3) * 8;
        const int64_t first = first0 + (int64_t)(e >> 2) * 32 + shift;
        if (first >= size) continue;
        const uint32_t valid = size - first < 8 ? (1u << (int)(size - first)) - 1u : 0xffu;
        const int holes_before = s_before[e >> 2] + __popc(word & ((1u << shift) - 1u));
        uint32_t hb = (word >> shift) & valid;
        uint32_t lb = ~(word >> shift) & valid;
        // Holes: ascending rank.
        for (int h = holes_before; hb && h < remove_count; h++) {
            hole_list[h] = (int32_t)(first + (__ffs(hb) - 1));
            hb &= hb - 1;
        }
        // Live particles: back rank = live_total - 1 - front rank, front rank = index - holes
        // before it; the byte's last one has the smallest.
        int64_t back = live_total - 1 - (first - holes_before);
        if (back - __popc(lb) + 1 < remove_count) {
            for (; lb; back--) {
                if (back < remove_count) mover_list[back] = (int32_t)(first + (__ffs(lb) - 1));
                lb &= lb - 1;
            }
        }
    }
}

// One (pair, column) per thread and pass of a grid-stride loop: copies the element of column
// col of the mover to the hole.  The pair index runs fastest, so a warp reads consecutive
// entries of the two lists and, the movers being the last live particles in descending order,
// neighbouring elements of one column; only the writes to the holes scatter.
__global__ void hf_copy_kernel(CountArg pairs_arg, const int32_t* __restrict__ hole_list,
                               const int32_t* __restrict__ mover_list, const int* __restrict__ totals,
                               CountArg size_arg, int32_t stride, DatList dats) {
    const int64_t n_pairs_max = resolve(pairs_arg);
    const int64_t size = resolve(size_arg);
    const int64_t H = totals[0];
    const int64_t n_items = n_pairs_max * dats.total_cols;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_items;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int col = (int)(t / n_pairs_max);
        const int64_t k = t - (int64_t)col * n_pairs_max;
        if (k >= H || k >= size - H) continue;
        const int32_t to = hole_list[k], from = mover_list[k];
        if (from <= to) continue;
        int d = 0, c = col;
        while (d < dats.n && c >= dats.dim[d]) {
            c -= dats.dim[d];
            d++;
        }
        if (d >= dats.n) continue;
        const int64_t off = (int64_t)c * stride;
        if (dats.bytes[d] == 8) {
            int64_t* a = reinterpret_cast<int64_t*>(dats.data[d]) + off;
            a[to] = a[from];
        } else {
            int32_t* a = reinterpret_cast<int32_t*>(dats.data[d]) + off;
            a[to] = a[from];
        }
    }
}

// Closes a device-sized step (one thread): the step record, the first error, the new count.
__global__ void step_end_kernel(oppb_set_count* cnt, int32_t pending, const oppb_move_status* st,
                                oppb_step_record* records, int32_t n_records) {
    const int32_t n = cnt->size + pending;
    const int32_t removed = st->remove_count;
    oppb_step_record r;
    r.size_before_move = n;
    r.removed = removed;
    r.size = n - removed;
    r.max_visits = st->max_visits;
    r.total_visits = st->total_visits;
    r.recheck_count = st->recheck_count;
    r.error = st->error;
    const int32_t step = cnt->steps;
    if (records && n_records > 0) records[step % n_records] = r;
    if (st->error && !cnt->error) {
        cnt->error = st->error;
        cnt->error_step = step;
    }
    cnt->size = n - removed;
    cnt->steps = step + 1;
}

// bits[w] bit b = (p2c[32 w + b] == removed) over [0, size); a warp writes one word, bits past
// size are 0.
__global__ void __launch_bounds__(256) removal_bits_kernel(const int32_t* __restrict__ p2c, int32_t size,
                                                           uint32_t* __restrict__ bits) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const bool gone = i < size && __ldg(p2c + i) == kRemoved;
    const uint32_t w = __ballot_sync(kFullMask, gone);
    if ((threadIdx.x & 31) == 0 && i < size) bits[i >> 5] = w;
}

// Blocks up to which the emit kernel sums the blocks' counts itself instead of a scan launch (4.2 us
// and a gap): 4 loads a thread at the limit, 16.8M particles (at 57M particles, 3,517 blocks, the
// emit kernel takes 12 us longer so).  A captured ten-step cycle of 460k
// particles takes 714 us instead of 796, a step-by-step one 525 instead of 540 (four steps).
constexpr int kHfDirectBlocks = 1024;

// The hole fill's launches.  block_holes: n_blocks + 1 ints.
int launch_hole_fill(const uint32_t* remove_bits, const CountArg& sz, const CountArg& rc, int64_t n_words, int n_blocks,
                     int* block_holes, int32_t* hole_list, int32_t* mover_list, int32_t stride, const DatList& dl,
                     int copy_grid, cudaStream_t s) {
    int* total = block_holes + n_blocks;
    hf_count_kernel<<<n_blocks, kHfBlock, 0, s>>>(remove_bits, sz, n_words, block_holes);
    if (n_blocks <= kHfDirectBlocks) {
        hf_emit_kernel<false><<<n_blocks, kHfBlock, 0, s>>>(remove_bits, sz, n_words, block_holes, n_blocks, rc,
                                                            hole_list, mover_list, total);
    } else {
        scan_single_block_kernel<<<1, kScanBlock, 0, s>>>(block_holes, n_blocks);
        hf_emit_kernel<true><<<n_blocks, kHfBlock, 0, s>>>(remove_bits, sz, n_words, block_holes, n_blocks, rc,
                                                           hole_list, mover_list, total);
        count_launches(1);
    }
    count_launches(2);
    if (dl.total_cols > 0) {
        hf_copy_kernel<<<copy_grid, 256, 0, s>>>(rc, hole_list, mover_list, total, sz, stride, dl);
        count_launches(1);
    }
    return launch_status();
}

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace
}  // namespace oppb

extern "C" int oppb_removal_bits(const int32_t* p2c, int32_t size, uint32_t* remove_bits, void* stream) {
    using namespace oppb;
    if (size < 0 || (size > 0 && (!p2c || !remove_bits))) return OPPB_ERR_ARG;
    if (size == 0) return OPPB_OK;
    removal_bits_kernel<<<ceil_div(size, 256), 256, 0, as_stream(stream)>>>(p2c, size, remove_bits);
    count_launches(1);
    return launch_status();
}

extern "C" size_t oppb_hole_fill_workspace_bytes(int32_t size, int32_t remove_count) {
    using namespace oppb;
    if (size < 0 || remove_count < 0) return 0;
    const int64_t n_words = ceil_div(size, 32);
    const int n_blocks = ceil_div(n_words, kHfWords);
    return align256(sizeof(int) * (size_t)(n_blocks + 1)) + align256(sizeof(int) * scan_scratch_ints(n_blocks)) +
           2 * align256(sizeof(int32_t) * (size_t)(remove_count > 0 ? remove_count : 1));
}

extern "C" int oppb_hole_fill(int32_t size, int32_t remove_count, const uint32_t* remove_bits, int32_t stride,
                              int32_t n_dats, const oppb_dat* dats, void* workspace, size_t workspace_bytes,
                              void* stream) {
    using namespace oppb;
    if (size < 0 || remove_count < 0 || stride < size || n_dats < 0 || n_dats > kMaxDats) return OPPB_ERR_ARG;
    if (remove_count == 0 || size == 0) return OPPB_OK;
    if (!remove_bits || !dats || !workspace) return OPPB_ERR_ARG;
    if (workspace_bytes < oppb_hole_fill_workspace_bytes(size, remove_count)) return OPPB_ERR_WORKSPACE;
    DatList dl{};
    dl.n = n_dats;
    dl.total_cols = 0;
    for (int d = 0; d < n_dats; d++) {
        if (!dats[d].data || dats[d].dim <= 0 || (dats[d].elem_bytes != 4 && dats[d].elem_bytes != 8))
            return OPPB_ERR_ARG;
        dl.data[d] = dats[d].data;
        dl.dim[d] = dats[d].dim;
        dl.bytes[d] = dats[d].elem_bytes;
        dl.total_cols += dats[d].dim;
    }
    cudaStream_t s = as_stream(stream);
    const int64_t n_words = ceil_div(size, 32);
    const int n_blocks = ceil_div(n_words, kHfWords);
    char* ws = static_cast<char*>(workspace);
    int* block_base = reinterpret_cast<int*>(ws);
    ws += align256(sizeof(int) * (size_t)(n_blocks + 1));
    ws += align256(sizeof(int) * scan_scratch_ints(n_blocks));
    int32_t* hole_list = reinterpret_cast<int32_t*>(ws);
    ws += align256(sizeof(int32_t) * (size_t)remove_count);
    int32_t* mover_list = reinterpret_cast<int32_t*>(ws);

    const CountArg sz{size, nullptr, 0}, rc{remove_count, nullptr, 0};
    return launch_hole_fill(remove_bits, sz, rc, n_words, n_blocks, block_base, hole_list, mover_list, stride, dl,
                            ceil_div((int64_t)remove_count * dl.total_cols, 256), s);
}

extern "C" size_t oppb_hole_fill_dev_workspace_bytes(int32_t size_bound) {
    return oppb_hole_fill_workspace_bytes(size_bound, size_bound);
}

extern "C" int oppb_hole_fill_dev(int32_t size_bound, const oppb_set_count* count, int32_t pending,
                                  const oppb_move_status* status, const uint32_t* remove_bits, int32_t stride,
                                  int32_t n_dats, const oppb_dat* dats, void* workspace, size_t workspace_bytes,
                                  void* stream) {
    using namespace oppb;
    if (size_bound < 0 || pending < 0 || stride < size_bound || n_dats < 0 || n_dats > kMaxDats) return OPPB_ERR_ARG;
    if (!count || !status) return OPPB_ERR_ARG;
    if (size_bound == 0) return OPPB_OK;
    if (!remove_bits || !dats || !workspace) return OPPB_ERR_ARG;
    if (workspace_bytes < oppb_hole_fill_dev_workspace_bytes(size_bound)) return OPPB_ERR_WORKSPACE;
    DatList dl{};
    dl.n = n_dats;
    dl.total_cols = 0;
    for (int d = 0; d < n_dats; d++) {
        if (!dats[d].data || dats[d].dim <= 0 || (dats[d].elem_bytes != 4 && dats[d].elem_bytes != 8))
            return OPPB_ERR_ARG;
        dl.data[d] = dats[d].data;
        dl.dim[d] = dats[d].dim;
        dl.bytes[d] = dats[d].elem_bytes;
        dl.total_cols += dats[d].dim;
    }
    cudaStream_t s = as_stream(stream);
    const int64_t n_words = ceil_div(size_bound, 32);
    const int n_blocks = ceil_div(n_words, kHfWords);
    char* ws = static_cast<char*>(workspace);
    int* block_base = reinterpret_cast<int*>(ws);
    ws += align256(sizeof(int) * (size_t)(n_blocks + 1));
    ws += align256(sizeof(int) * scan_scratch_ints(n_blocks));
    int32_t* hole_list = reinterpret_cast<int32_t*>(ws);
    ws += align256(sizeof(int32_t) * (size_t)size_bound);
    int32_t* mover_list = reinterpret_cast<int32_t*>(ws);
    // The count and the move's remove count are read on the device; the lists hold up to
    // size_bound pairs, and no more than the count can be removed.
    const CountArg sz{size_bound, &count->size, pending};
    const CountArg rc{size_bound, &status->remove_count, 0};
    const int64_t copy_blocks = ceil_div((int64_t)size_bound * dl.total_cols, 256);
    return launch_hole_fill(remove_bits, sz, rc, n_words, n_blocks, block_base, hole_list, mover_list, stride, dl,
                            (int)(copy_blocks < 148 * 16 ? copy_blocks : 148 * 16), s);
}

extern "C" int oppb_step_end_dev(oppb_set_count* count, int32_t pending, const oppb_move_status* status,
                                 oppb_step_record* records, int32_t n_records, void* stream) {
    using namespace oppb;
    if (!count || !status || pending < 0 || n_records < 0 || (n_records > 0 && !records)) return OPPB_ERR_ARG;
    step_end_kernel<<<1, 1, 0, as_stream(stream)>>>(count, pending, status, records, n_records);
    count_launches(1);
    return launch_status();
}

// ------------------------------------------------------- allocation-free hole fill
//
// oppb_hole_fill_static runs the same four kernels as oppb_hole_fill with its scratch in
// a fixed array of this library instead of a caller workspace, for callers that cannot
// allocate device memory where they move particles (a plugin that sees only the dats'
// device pointers while another runtime owns the memory, or a loop that cannot afford
// the device-wide synchronisation of cudaMalloc / cudaFree).
//
// Layout of the array (int32 words): per-block hole counts for the largest possible
// particle count (their scan leaves the total at [n_blocks]), then the hole list and the
// mover list of OPPB_HOLE_FILL_STATIC_MAX_REMOVES entries each.  Every word a call reads
// was written earlier in the same call, so nothing has to start at zero and the contents
// left by the previous call are harmless.  All calls on a device share the array: calls
// that overlap on the GPU race.

namespace oppb {
namespace {

constexpr int64_t kStaticMaxBlocks = (((int64_t)INT_MAX + 31) / 32 + kHfWords - 1) / kHfWords;  // 131,072
constexpr int64_t kStaticBaseWords = (kStaticMaxBlocks + 1 + 63) / 64 * 64;  // whole 256-B lines
constexpr int64_t kStaticListWords = OPPB_HOLE_FILL_STATIC_MAX_REMOVES;
constexpr int64_t kStaticWords = kStaticBaseWords + 2 * kStaticListWords;  // about 8.5 MiB

}  // namespace

// Held by every GPU that loads the library, until the process exits.
static __device__ __align__(256) int32_t g_hole_fill_scratch[kStaticWords];

namespace {

constexpr int kStaticMaxDevices = 64;
std::mutex g_static_mu;
int32_t* g_static_addr[kStaticMaxDevices];  // device address of g_hole_fill_scratch, per device

// Device address of the scratch array on the current device.  In host code the array's name
// only stands in for the symbol; a kernel must be given this address instead.  It is looked
// up again on every call made outside a stream capture (cheap once the module is loaded), so
// that a device reset, which unloads the module and may place the array elsewhere when it is
// loaded again, never leaves a stale address behind; a call inside a capture uses the address
// found by the last call outside one.
int static_scratch(cudaStream_t stream, int32_t** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return OPPB_ERR_NO_DEVICE;
    }
    if (dev < 0 || dev >= kStaticMaxDevices) return OPPB_ERR_NO_DEVICE;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
        cudaGetLastError();
        return OPPB_ERR_LAUNCH;
    }
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_addr[dev] || cap == cudaStreamCaptureStatusNone) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_hole_fill_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            return OPPB_ERR_LAUNCH;
        }
        g_static_addr[dev] = static_cast<int32_t*>(p);
    }
    *out = g_static_addr[dev];
    return OPPB_OK;
}

}  // namespace
}  // namespace oppb

extern "C" int oppb_hole_fill_static(int32_t size, int32_t remove_count, const uint32_t* remove_bits,
                                     int32_t stride, int32_t n_dats, const oppb_dat* dats, void* stream) {
    using namespace oppb;
    if (size < 0 || remove_count < 0 || stride < size || n_dats < 0 || n_dats > kMaxDats) return OPPB_ERR_ARG;
    if (remove_count > OPPB_HOLE_FILL_STATIC_MAX_REMOVES) return OPPB_ERR_SCRATCH_LIMIT;
    if (remove_count == 0 || size == 0) return OPPB_OK;
    if (!remove_bits || !dats) return OPPB_ERR_ARG;
    DatList dl{};
    dl.n = n_dats;
    dl.total_cols = 0;
    for (int d = 0; d < n_dats; d++) {
        if (!dats[d].data || dats[d].dim <= 0 || (dats[d].elem_bytes != 4 && dats[d].elem_bytes != 8))
            return OPPB_ERR_ARG;
        dl.data[d] = dats[d].data;
        dl.dim[d] = dats[d].dim;
        dl.bytes[d] = dats[d].elem_bytes;
        dl.total_cols += dats[d].dim;
    }
    cudaStream_t s = as_stream(stream);
    int32_t* scratch = nullptr;
    const int lookup = static_scratch(s, &scratch);
    if (lookup != OPPB_OK) return lookup;
    const int64_t n_words = ceil_div(size, 32);
    const int n_blocks = ceil_div(n_words, kHfWords);  // <= kStaticMaxBlocks for any int32 size
    int* block_base = scratch;
    int32_t* hole_list = scratch + kStaticBaseWords;
    int32_t* mover_list = hole_list + kStaticListWords;

    const CountArg sz{size, nullptr, 0}, rc{remove_count, nullptr, 0};
    return launch_hole_fill(remove_bits, sz, rc, n_words, n_blocks, block_base, hole_list, mover_list, stride, dl,
                            ceil_div((int64_t)remove_count * dl.total_cols, 256), s);
}
