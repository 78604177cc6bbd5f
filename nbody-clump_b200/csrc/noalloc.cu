// noalloc.cu -- a cell sort that allocates no device memory.
//
// Some callers cannot call cudaMalloc: a host program whose device memory
// is owned by another framework's pool, or code running where allocation is
// forbidden once a run has started (a memory budget fixed at start-up).
// nbc_cell_sort_noalloc gives them the engine's cell hash and a stable radix
// sort by cell (the order of the first half of a list rebuild) using only
// buffers the caller passes plus one scratch array compiled into this library.
//
// A hash and one launch per digit: the hash counts the first digit of each
// tile of keys, each pass finds its own offsets from the counts of all tiles
// and counts the next digit where the keys land.
//
// Scratch: `g_sort_scratch` below, NBC_NOALLOC_MAX_N elements of key/value
// ping-pong plus the digit counts of three passes, about 2.5 MB, held on every
// GPU that loads the library until the process exits.  Every call on a device
// shares it and it keeps the previous call's contents (the counts are rebuilt
// from zero by each call, the ping-pong halves are fully overwritten), so
// calls whose work overlaps on the GPU -- on two streams, or from two host
// threads -- race on it and must be serialised by the caller.
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "../../include/nbc.h"
#include "kernels.cuh"

namespace nbc {
extern thread_local std::string g_last_error;
}

namespace {

constexpr int MAX_N = NBC_NOALLOC_MAX_N;
// 512 threads a block, 4 keys a thread.  A digit has up to 9 bits (two passes
// for the grids of up to 262,144 cells where 8 bits need three; with 10 the
// counts of a tile, which every block reads, are twice as long).  The counts
// of a tile are at most TILE, so two digits share a word.
constexpr int CS_THREADS = 512;
constexpr int CS_ITEMS = 4;
constexpr int CS_TILE = CS_THREADS * CS_ITEMS;
constexpr int CS_BITS = 9;
constexpr int CS_DIGITS = 1 << CS_BITS;
constexpr int CS_WORDS = CS_DIGITS / 2;   // of a tile's counts
constexpr int CS_WARPS = CS_THREADS / 32;
static_assert(CS_DIGITS == CS_THREADS && CS_TILE < 65536, "a thread per digit, 16-bit counts");

constexpr int MAX_TILES = (MAX_N + CS_TILE - 1) / CS_TILE;
constexpr int CS_PARTS = 8;               // of the tiles, whose counts a pass sums side by side
static_assert((MAX_TILES + CS_PARTS - 1) / CS_PARTS * CS_TILE < 65536, "the sum of a part stays in 16 bits");
constexpr size_t CS_COUNTS = (size_t)MAX_TILES * CS_WORDS;
constexpr size_t SCRATCH_INTS = 2 * (size_t)MAX_N + 3 * CS_COUNTS;

// the scratch array; host code must not pass its name to a kernel (in host
// code it is only a stand-in), it uses the device address looked up below
__device__ __align__(256) int g_sort_scratch[SCRATCH_INTS];

constexpr int MAX_DEVICES = 64;
int* g_scratch_addr[MAX_DEVICES] = {nullptr};
std::mutex g_scratch_mu;

nbc_status fail(nbc_status code, const std::string& m) {
    nbc::g_last_error = m;
    return code;
}

__device__ __forceinline__ void count_digit(unsigned* cnt, int dig) { atomicAdd(cnt + (dig >> 1), 1u << (16 * (dig & 1))); }

// GetParticleCellIndex_cuk (src/dem_grid.cu:155-202) on caller buffers, a tile
// per block, with the counts of the tile's first digits; clears the counts
// that the first pass adds to.
__global__ void __launch_bounds__(CS_THREADS) k_cs_hash(const double* __restrict__ pos, int n, nbc_grid_desc g, int mask,
                                                        int* __restrict__ keys, unsigned* __restrict__ cnt,
                                                        unsigned* __restrict__ cnt_next) {
    __shared__ unsigned h[CS_WORDS];
    const int tid = threadIdx.x;
    if (tid < CS_WORDS) h[tid] = 0;
    __syncthreads();
    const int cellnum = g.dims[0] * g.dims[1] * g.dims[2];
#pragma unroll
    for (int it = 0; it < CS_ITEMS; it++) {
        const int i = blockIdx.x * CS_TILE + it * CS_THREADS + tid;
        if (i >= n) break;
        const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
        int local;
        if (z >= g.box_hi[2] || y >= g.box_hi[1] || x >= g.box_hi[0] || z < g.box_lo[2] || y < g.box_lo[1] ||
            x < g.box_lo[0]) {
            local = cellnum - 1;
        } else {
            int cx = nbc::clampi((int)floor((x - g.origin[0]) / g.cell), 0, g.dims[0] - 1);
            int cy = nbc::clampi((int)floor((y - g.origin[1]) / g.cell), 0, g.dims[1] - 1);
            int cz = nbc::clampi((int)floor((z - g.origin[2]) / g.cell), 0, g.dims[2] - 1);
            local = nbc::clampi(cz * g.dims[1] * g.dims[0] + cy * g.dims[0] + cx, 0, cellnum - 1);
        }
        keys[i] = local;
        count_digit(h, local & mask);
    }
    __syncthreads();
    cudaTriggerProgrammaticLaunchCompletion();
    if (tid < CS_WORDS) {
        cnt[blockIdx.x * CS_WORDS + tid] = h[tid];
        cnt_next[blockIdx.x * CS_WORDS + tid] = 0;
    }
}

// One stable pass by the digit at `shift`.  cnt: this digit's counts per tile;
// cnt_next (null in the last pass): the next digit's, counted here by the tile
// a key lands in; cnt_clear (null when no pass follows the next): cleared for
// the pass after.  vin null: a key's value is its index.
//
// A block sums every tile's counts for itself (a digit's total, and its part
// of the tiles before), 88 KB from the L2 at 180,000 keys, where a scan would
// be three more launches: eight tiles side by side, 16 bytes a thread, so that
// all loads of a thread are in flight (two tiles at a time and 4 bytes: 33 us
// for the call below).  A warp takes 128 consecutive keys, 32 at a time; the
// lanes with an equal digit are found by a vote per bit, and a warp keeps
// counts of its own, so that the block waits a few times a pass and not three
// times per 256 keys.  A pass is launched while the one before it writes its
// keys (triggered any earlier, the waiting blocks take their place on the SMs
// unevenly: 24.6 us, as without).  The call is bound by the latency of three
// short launches: 180,001 keys of 17 bits 20.5 us, before 96 in 16 launches;
// 262,144 of 21 bits 33; 500 keys 14.  Tiles of 1,024 keys: 25% slower, the
// counts of twice as many tiles weigh more than the idle SMs.
__global__ void __launch_bounds__(CS_THREADS)
    k_cs_pass(const int* kin, const int* vin, int* __restrict__ kout, int* __restrict__ vout, int n, int shift, int bits,
              const unsigned* cnt, unsigned* __restrict__ cnt_next, unsigned* __restrict__ cnt_clear) {
    __shared__ __align__(16) unsigned short wcnt[CS_WARPS][CS_DIGITS];
    __shared__ __align__(16) unsigned s_all[CS_PARTS][CS_WORDS], s_bef[CS_PARTS][CS_WORDS];
    __shared__ int s_base[CS_DIGITS], s_warp[CS_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x, tiles = gridDim.x, mask = (1 << bits) - 1;
    constexpr unsigned FULL = 0xffffffffu;
    int k[CS_ITEMS], v[CS_ITEMS], rank[CS_ITEMS];
    for (int u = tid; u < CS_WARPS * CS_DIGITS / 2; u += CS_THREADS) ((unsigned*)wcnt)[u] = 0;
    // what the launch before wrote (kin, vin, cnt: not __restrict__, or their
    // loads could move up) is complete from here on
    cudaGridDependencySynchronize();
    const int at = tile * CS_TILE + warp * (CS_TILE / CS_WARPS) + lane;
#pragma unroll
    for (int it = 0; it < CS_ITEMS; it++) {
        const int i = at + 32 * it;
        k[it] = i < n ? kin[i] : 0;
        v[it] = vin && i < n ? vin[i] : i;
    }
    if (cnt_clear && tid < CS_WORDS) cnt_clear[tile * CS_WORDS + tid] = 0;
    // the counts of every eighth tile, eight digits a thread
    const int part = tid / (CS_WORDS / 4), col = tid % (CS_WORDS / 4);
    uint4 all = make_uint4(0, 0, 0, 0), bef = all;
#pragma unroll 8
    for (int t = part; t < tiles; t += CS_PARTS) {
        const uint4 c = ((const uint4*)cnt)[t * (CS_WORDS / 4) + col];
        all.x += c.x; all.y += c.y; all.z += c.z; all.w += c.w;
        if (t < tile) { bef.x += c.x; bef.y += c.y; bef.z += c.z; bef.w += c.w; }
    }
    ((uint4*)s_all[part])[col] = all;
    ((uint4*)s_bef[part])[col] = bef;
    __syncthreads();
    // each key's place among the warp's keys of its digit
#pragma unroll
    for (int it = 0; it < CS_ITEMS; it++) {
        const bool valid = at + 32 * it < n;
        const int dig = (k[it] >> shift) & mask;
        unsigned peers = __ballot_sync(FULL, valid);
#pragma unroll
        for (int b = 0; b < CS_BITS; b++) {
            const bool bit = (dig >> b) & 1;
            const unsigned m = __ballot_sync(FULL, bit);
            peers &= bit ? m : ~m;
        }
        const unsigned below = peers & ((1u << lane) - 1u);
        const int had = wcnt[warp][dig];
        rank[it] = had + __popc(below);
        __syncwarp();
        if (valid && !below) wcnt[warp][dig] = (unsigned short)(had + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // digit tid: exclusive sum of the totals, the tiles before, and the warps before
    int tot = 0, base = 0;
#pragma unroll
    for (int p = 0; p < CS_PARTS; p++) {
        tot += (s_all[p][tid >> 1] >> (16 * (tid & 1))) & 0xffff;
        base += (s_bef[p][tid >> 1] >> (16 * (tid & 1))) & 0xffff;
    }
    int inc = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += x;
    }
    if (lane == 31) s_warp[warp] = inc;
    int acc = 0;
#pragma unroll
    for (int x = 0; x < CS_WARPS; x++) {
        const int c = wcnt[x][tid];
        wcnt[x][tid] = (unsigned short)acc;
        acc += c;
    }
    __syncthreads();
    base += inc - tot;
#pragma unroll
    for (int x = 0; x < CS_WARPS; x++) base += x < warp ? s_warp[x] : 0;
    s_base[tid] = base;
    cudaTriggerProgrammaticLaunchCompletion();
    __syncthreads();
#pragma unroll
    for (int it = 0; it < CS_ITEMS; it++) {
        if (at + 32 * it >= n) continue;
        const int dig = (k[it] >> shift) & mask;
        const int q = s_base[dig] + wcnt[warp][dig] + rank[it];
        kout[q] = k[it];
        vout[q] = v[it];
        if (cnt_next) count_digit(cnt_next + q / CS_TILE * CS_WORDS, (k[it] >> (shift + bits)) & mask);
    }
}

}  // namespace

extern "C" nbc_status nbc_cell_sort_noalloc(const double* pos_dev, int n, const nbc_grid_desc* grid, int* perm_dev,
                                            int* key_dev, void* stream) {
    if (n < 0 || n > MAX_N)
        return fail(NBC_ERR_ARG, "nbc_cell_sort_noalloc: n = " + std::to_string(n) + " is outside 0.." +
                                     std::to_string(MAX_N) + " (the size of the library's scratch array)");
    if (!grid || (n > 0 && (!pos_dev || !perm_dev || !key_dev)))
        return fail(NBC_ERR_ARG, "nbc_cell_sort_noalloc: null argument");
    const long long cells = (long long)grid->dims[0] * grid->dims[1] * grid->dims[2];
    if (grid->dims[0] <= 0 || grid->dims[1] <= 0 || grid->dims[2] <= 0 || cells > (1LL << 30) || !(grid->cell > 0))
        return fail(NBC_ERR_ARG, "nbc_cell_sort_noalloc: bad grid");
    if (n == 0) return NBC_OK;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(NBC_ERR_NO_DEVICE, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= MAX_DEVICES) return fail(NBC_ERR_ARG, "device ordinal too large");
    cudaStream_t st = (cudaStream_t)stream;
    int* scratch;
    {
        // The scratch array's device address, with the device current.  It
        // is looked up again on every call made outside a stream capture (a
        // device reset rebuilds the context and may move the array); a call
        // inside a capture uses the address the last uncaptured call on this
        // device found, so the first call on a device must come before any
        // capture.
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        e = cudaStreamIsCapturing(st, &cs);
        if (e != cudaSuccess)
            return fail(NBC_ERR_CUDA, std::string("cudaStreamIsCapturing: ") + cudaGetErrorString(e));
        std::lock_guard<std::mutex> lock(g_scratch_mu);
        if (cs == cudaStreamCaptureStatusNone) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_sort_scratch);
            if (e != cudaSuccess)
                return fail(NBC_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
            g_scratch_addr[dev] = (int*)p;
        } else if (!g_scratch_addr[dev]) {
            return fail(NBC_ERR_STATE, "nbc_cell_sort_noalloc: the first call on a device must not be captured");
        }
        scratch = g_scratch_addr[dev];
    }
    int* kB = scratch;
    int* vB = kB + MAX_N;
    unsigned* cnt[3];
    for (int c = 0; c < 3; c++) cnt[c] = (unsigned*)(vB + MAX_N) + c * CS_COUNTS;
    int bits = 1;
    while ((1LL << bits) < cells) bits++;
    const int passes = (bits + CS_BITS - 1) / CS_BITS, dbits = (bits + passes - 1) / passes;
    const int tiles = (n + CS_TILE - 1) / CS_TILE;
    // the caller's output buffers are one side of the ping-pong; with an odd
    // pass count the first pass starts from the scratch side so the last
    // pass lands in the caller's buffers
    int *ki, *vi, *ko, *vo;
    if (passes % 2 == 1) { ki = kB; vi = vB; ko = key_dev; vo = perm_dev; }
    else { ki = key_dev; vi = perm_dev; ko = kB; vo = vB; }
    k_cs_hash<<<tiles, CS_THREADS, 0, st>>>(pos_dev, n, *grid, (1 << dbits) - 1, ki, cnt[0], cnt[1]);
    for (int p = 0; p < passes; p++) {
        // (launched while the one before it drains)
        cudaLaunchAttribute early[1];
        early[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        early[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(tiles);
        cfg.blockDim = dim3(CS_THREADS);
        cfg.stream = st;
        cfg.attrs = early;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, k_cs_pass, (const int*)ki, (const int*)(p ? vi : nullptr), ko, vo, n, dbits * p, dbits,
                               (const unsigned*)cnt[p % 3], p + 1 < passes ? cnt[(p + 1) % 3] : (unsigned*)nullptr,
                               p + 2 < passes ? cnt[(p + 2) % 3] : (unsigned*)nullptr);
        if (e != cudaSuccess) return fail(NBC_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
        int* t = ki; ki = ko; ko = t;
        t = vi; vi = vo; vo = t;
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(NBC_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    return NBC_OK;
}
