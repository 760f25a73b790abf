// prims.cu — exclusive scan and LSD radix sort (hand-written; no CUB).
#include "prims.cuh"

namespace psx {

namespace {
constexpr int kScanBlock = 1024;  // elements per block: 256 threads x 4

__device__ __forceinline__ int warp_incl_scan(int v) {
    const unsigned m = 0xffffffffu;
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(m, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// block-wide exclusive scan of one value per thread (256 threads); returns block total via *tot
__device__ __forceinline__ int block_excl_scan(int v, int* sh, int* tot) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int inc = warp_incl_scan(v);
    if (lane == 31) sh[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int s = (lane < (blockDim.x >> 5)) ? sh[lane] : 0;
        int si = warp_incl_scan(s);
        sh[lane] = si - s;
        if (lane == 31) sh[32] = si;
    }
    __syncthreads();
    int r = inc - v + sh[wid];
    if (tot) *tot = sh[32];
    __syncthreads();
    return r;
}

__global__ void k_scan_blocks(const int* in, int* out, int n, const int* n_dev, int* block_sums) {
    __shared__ int sh[33];
    if (n_dev) n = min(n, *n_dev);
    int base = blockIdx.x * kScanBlock + threadIdx.x * 4;
    int v[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) { v[k] = (base + k < n) ? in[base + k] : 0; s += v[k]; }
    int tot;
    int ex = block_excl_scan(s, sh, &tot);
#pragma unroll
    for (int k = 0; k < 4; ++k) { if (base + k < n) out[base + k] = ex; ex += v[k]; }
    if (threadIdx.x == 0) block_sums[blockIdx.x] = tot;
}

// single block scans the per-block sums (any count) in chunks of 1024
__global__ void k_scan_sums(int* sums, int nb, int* total) {
    __shared__ int sh[33];
    int carry = 0;
    for (int c = 0; c < nb; c += kScanBlock) {
        int base = c + threadIdx.x * 4;
        int v[4], s = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) { v[k] = (base + k < nb) ? sums[base + k] : 0; s += v[k]; }
        int tot;
        int ex = block_excl_scan(s, sh, &tot) + carry;
#pragma unroll
        for (int k = 0; k < 4; ++k) { if (base + k < nb) sums[base + k] = ex; ex += v[k]; }
        carry += tot;
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void k_scan_add(int* out, int n, const int* n_dev, const int* sums) {
    if (n_dev) n = min(n, *n_dev);
    int add = sums[blockIdx.x];
    int base = blockIdx.x * kScanBlock + threadIdx.x * 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) if (base + k < n) out[base + k] += add;
}
}  // namespace

namespace {
// The whole scan in one block: below kSmallScan elements three launches cost more than
// their work (about 2.5 us each in a frame's chain; up to eight rounds of 4096 here).
constexpr int kSmallScan = 32768;
__global__ void __launch_bounds__(1024) k_scan_small(const int* in, int* out, int n, const int* n_dev, int* total) {
    __shared__ int sums[33];
    if (n_dev) n = min(n, *n_dev);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int carry = 0;
    for (int c = 0; c < n; c += 4096) {
        const int base = c + threadIdx.x * 4;
        int v[4], t = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) { v[k] = base + k < n ? in[base + k] : 0; t += v[k]; }
        const int inc = warp_incl_scan(t);
        if (lane == 31) sums[wid] = inc;
        __syncthreads();
        if (wid == 0) {
            const int w = sums[lane], wi = warp_incl_scan(w);
            sums[lane] = wi - w;
            if (lane == 31) sums[32] = wi;
        }
        __syncthreads();
        int ex = carry + sums[wid] + inc - t;
#pragma unroll
        for (int k = 0; k < 4; ++k) { if (base + k < n) out[base + k] = ex; ex += v[k]; }
        carry += sums[32];
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = carry;
}
}  // namespace

size_t scan_scratch_ints(int n) { return (size_t)(n + kScanBlock - 1) / kScanBlock + 1; }

static int scan_impl(const int* in, int* out, int n, const int* n_dev, int* total, int* scratch, cudaStream_t s) {
    if (n <= kSmallScan) {
        k_scan_small<<<1, 1024, 0, s>>>(in, out, n, n_dev, total);
        return 1;
    }
    int nb = (n + kScanBlock - 1) / kScanBlock;
    if (nb == 0) nb = 1;
    k_scan_blocks<<<nb, 256, 0, s>>>(in, out, n, n_dev, scratch);
    k_scan_sums<<<1, 256, 0, s>>>(scratch, nb, total);
    k_scan_add<<<nb, 256, 0, s>>>(out, n, n_dev, scratch);
    return 3;
}

int scan_exclusive(const int* in, int* out, int n, int* total, int* scratch, cudaStream_t s) {
    return scan_impl(in, out, n, nullptr, total, scratch, s);
}
int scan_exclusive_dev(const int* in, int* out, const int* n_dev, int n_max, int* total, int* scratch, cudaStream_t s) {
    return scan_impl(in, out, n_max, n_dev, total, scratch, s);
}

// ---------------------------------------------------------------- radix sort
//
// One 8-bit digit per pass.  A tile of keys is split into 8 contiguous
// warp chunks; per-warp digit counters make the ranking stable: a key's rank is
// (keys of the same digit in earlier tiles) + (in earlier warps of this tile) +
// (earlier in this warp's chunk), the last counted 32 keys at a time with
// __match_any_sync.
namespace {
constexpr int kRadixThreads = 256;
constexpr int kWarps = kRadixThreads / 32;
// A warp ranks its chunk 32 keys at a time, one round after another, so the tile sets the
// chain's length.  4096 keys a tile leave 65,537 keys to 17 blocks (25.6 us a scatter); up
// to 2^18 keys, 1024 a tile fill the chip's SMs (65 blocks).  Above, larger tiles keep
// the histogram small.
int radix_tile(int n) { return n <= (1 << 18) ? 1024 : 4096; }

template <int kTile>
__global__ void k_radix_hist(const uint32_t* keys, int n, int shift, int* hist, int ntiles) {
    __shared__ int h[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    int base = blockIdx.x * kTile;
    for (int i = threadIdx.x; i < kTile; i += blockDim.x) {
        int k = base + i;
        if (k < n) atomicAdd(&h[(keys[k] >> shift) & 255], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < 256; d += blockDim.x) hist[d * ntiles + blockIdx.x] = h[d];
}

template <int kTile>
__global__ void k_radix_scatter(const uint32_t* keys, const int* vals, uint32_t* ok, int* ov, int n, int shift,
                                const int* offs, int ntiles) {
    constexpr int kPerWarp = kTile / kWarps;
    __shared__ int wc[kWarps][256];   // per-warp running counters, then per-warp base offsets
    int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = lane; i < 256; i += 32) wc[wid][i] = 0;
    __syncwarp();
    int cbase = blockIdx.x * kTile + wid * kPerWarp;
    // pass 1: per-warp digit histogram
    for (int r = 0; r < kPerWarp; r += 32) {
        int k = cbase + r + lane;
        if (k < n) atomicAdd(&wc[wid][(keys[k] >> shift) & 255], 1);
    }
    __syncthreads();
    // exclusive scan across warps per digit, plus the global tile offset
    for (int d = threadIdx.x; d < 256; d += blockDim.x) {
        int run = offs[d * ntiles + blockIdx.x];
        for (int w = 0; w < kWarps; ++w) { int c = wc[w][d]; wc[w][d] = run; run += c; }
    }
    __syncthreads();
    // pass 2: stable scatter, 32 keys at a time
    for (int r = 0; r < kPerWarp; r += 32) {
        int k = cbase + r + lane;
        bool valid = k < n;
        uint32_t key = valid ? keys[k] : 0xffffffffu;
        int d = valid ? (int)((key >> shift) & 255) : 256 + lane;  // invalid lanes match nobody
        unsigned peers = __match_any_sync(0xffffffffu, d);
        int rank = __popc(peers & ((1u << lane) - 1));
        int cnt = __popc(peers);
        int leader = __ffs(peers) - 1;
        int basev = 0;
        if (valid && lane == leader) basev = wc[wid][d];
        basev = __shfl_sync(0xffffffffu, basev, leader);
        if (valid) {
            int dst = basev + rank;
            ok[dst] = key;
            ov[dst] = vals[k];
        }
        __syncwarp();
        if (valid && lane == leader) wc[wid][d] = basev + cnt;
        __syncwarp();
    }
}
}  // namespace

size_t radix_hist_ints(int n) {
    int ntiles = (n + radix_tile(n) - 1) / radix_tile(n);
    if (ntiles == 0) ntiles = 1;
    size_t h = (size_t)256 * ntiles;
    return 2 * h + scan_scratch_ints((int)h) + 1;
}

int radix_sort_pairs(uint32_t* keys, int* vals, uint32_t* tmpk, int* tmpv, int n, int bits, int* hist, cudaStream_t s) {
    if (n <= 0) return 0;
    const int tile = radix_tile(n), ntiles = (n + tile - 1) / tile;
    int h = 256 * ntiles;
    int* offs = hist + h;
    int* scratch = offs + h;
    uint32_t* ka = keys; int* va = vals;
    uint32_t* kb = tmpk; int* vb = tmpv;
    int passes = (bits + 7) / 8, launches = 0;
    for (int p = 0; p < passes; ++p) {
        int shift = 8 * p;
        if (tile == 1024) k_radix_hist<1024><<<ntiles, kRadixThreads, 0, s>>>(ka, n, shift, hist, ntiles);
        else k_radix_hist<4096><<<ntiles, kRadixThreads, 0, s>>>(ka, n, shift, hist, ntiles);
        launches += 2 + scan_exclusive(hist, offs, h, nullptr, scratch, s);
        if (tile == 1024) k_radix_scatter<1024><<<ntiles, kRadixThreads, 0, s>>>(ka, va, kb, vb, n, shift, offs, ntiles);
        else k_radix_scatter<4096><<<ntiles, kRadixThreads, 0, s>>>(ka, va, kb, vb, n, shift, offs, ntiles);
        uint32_t* tk = ka; ka = kb; kb = tk;
        int* tv = va; va = vb; vb = tv;
    }
    if (ka != keys) {
        cudaMemcpyAsync(keys, ka, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(vals, va, sizeof(int) * n, cudaMemcpyDeviceToDevice, s);
    }
    return launches;
}

}  // namespace psx
