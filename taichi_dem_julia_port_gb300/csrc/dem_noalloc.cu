// dem_noalloc.cu — the broad-phase bucket sort for callers that cannot
// allocate device memory.
//
// Some embedders cannot call cudaMalloc: a host that pre-allocates every
// device buffer once and forbids allocation afterwards (a real-time or
// certified control loop), a process whose allocator is owned by another
// framework, or a step that runs while allocation is blocked.  They pass their
// own input and output buffers, and the temporary memory the sort needs lives
// in one file-scope device array below, reserved on every GPU that loads this
// library until the process exits.
//
// The sort: cell + hashcode per particle (src/utils.jl:1-2), then a stable
// least-significant-digit radix sort of the particle indices by bucket, 10
// bits per pass (one pass for tables of up to 1,024 buckets, two above).
// Stability keeps ascending index inside each bucket, which is the order the
// library's regular broad phase gives (the reference leaves it free,
// src/kernels.jl:15-22).  The work is O(n + H) whatever the bucket
// occupancy: one bucket holding every particle costs the same as many small
// ones.
//
// Three launches per pass, none of which waits on another block: the digit
// counts of every chunk of 4,096 particles (the first pass counts while it
// hashes), each digit's running sum over the chunks, and the scatter, which
// scans the 1,024 digit totals itself.
//
// Limits: n <= 1,048,576 particles and hash_table_size <= 1,048,576 buckets;
// the array is 9.4 MB (the first pass's keys and indices, the per-chunk
// digit counts, and the digit totals).
#include <cmath>
#include <mutex>

#include "dem_device.cuh"
#include "dem_gb300.h"

namespace {

constexpr long long kMaxN = 1 << 20;
constexpr long long kMaxH = 1 << 20;
constexpr int kBlock = 512;
constexpr int kWarps = kBlock / 32;
constexpr int kItems = 8;
constexpr int kChunk = kBlock * kItems;  // particles per block of a radix pass
constexpr int kDigitBits = 10;
constexpr int kBins = 1 << kDigitBits;
constexpr long long kMaxBlocks = kMaxN / kChunk;
constexpr long long kHistWords = kBins * kMaxBlocks;
constexpr size_t kKeysOff = 0;
constexpr size_t kValsOff = kKeysOff + kMaxN;
constexpr size_t kHistOff = kValsOff + kMaxN;
constexpr size_t kTotalsOff = kHistOff + kHistWords;
constexpr size_t kWords = kTotalsOff + kBins;
constexpr int kMaxDevices = 64;

// The scratch: the first pass's output keys (0-based buckets) and particle
// indices, the digit counts of every chunk (scanned in place over the chunks)
// and the digits' totals.
// Every word a call reads is written earlier in the same call, so nothing
// needs clearing between calls.  Host code must not take this name as a
// device address; it uses the address from cudaGetSymbolAddress (see
// scratch_on()).
static __device__ __align__(256) uint32_t g_scratch[kWords];

struct Geometry {
    double dmin[3];
    double cell;
    float inv_cell32, dmin_cells;  // the FP32 screen of the cell (cell_screen)
    int screen;                    // 0: the cell size is beyond the screen's range
    uint32_t H;
    uint32_t mask;
};

__device__ __forceinline__ uint32_t na_bucket(int x, int y, int z, const Geometry& g) {
    const uint32_t m = dem::morton1(x, y, z);
    return g.mask ? (m & g.mask) : (m % g.H);
}
// What the screen leaves open, out of line: eight particles' cells unrolled
// with the exact divisions inline waited for instructions a third of the time
// (1,000,000 particles: 23 us).
static __device__ __noinline__ int na_cell_exact(double num, double cell) {
    return dem::ceil_i32(__ddiv_rn(num, cell));
}
__device__ __forceinline__ int na_cell(double x, int c, const Geometry& g) {
    const double num = __dsub_rn(x, g.dmin[c]);
    int k;
    if (g.screen && dem::cell_screen(num, g.inv_cell32, g.dmin_cells, &k)) return k;
    return na_cell_exact(num, g.cell);
}

// cell + hashcode (src/utils.jl:1-2) of one chunk, the reference's 1-based
// buckets, with the first pass's digit counts (hist[chunk · kBins + digit]).
// The three quotients per particle were the whole sort's largest cost as FP64
// divisions (1,000,000 particles: 74 us of 166 us; GB300 retires one FP64
// warp-instruction per 64 cycles and SM sub-partition); the FP32 screen decides all but the cells' edges.
__global__ void __launch_bounds__(kBlock)
    k_na_hash(const double* __restrict__ px, const double* __restrict__ py,
              const double* __restrict__ pz, int n, Geometry g, uint32_t* bucket_out,
              uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kBins];
    const int base = blockIdx.x * kChunk + (int)threadIdx.x;
    double x[kItems], y[kItems], z[kItems];
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int i = base + q * kBlock;
        x[q] = i < n ? px[i] : 0.0;
        y[q] = i < n ? py[i] : 0.0;
        z[q] = i < n ? pz[i] : 0.0;
    }
    for (int b = threadIdx.x; b < kBins; b += kBlock) h[b] = 0u;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int i = base + q * kBlock;
        if (i < n) {
            const uint32_t b = na_bucket(na_cell(x[q], 0, g), na_cell(y[q], 1, g),
                                         na_cell(z[q], 2, g), g);
            bucket_out[i] = b + 1u;
            atomicAdd(&h[b & (kBins - 1)], 1u);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < kBins; b += kBlock) hist[(size_t)blockIdx.x * kBins + b] = h[b];
}

// Digit counts of one chunk's keys for a later pass.
__global__ void __launch_bounds__(kBlock)
    k_na_digit_count(const uint32_t* __restrict__ keys, int n, int shift,
                     uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kBins];
    for (int b = threadIdx.x; b < kBins; b += kBlock) h[b] = 0u;
    __syncthreads();
    const int base = blockIdx.x * kChunk + (int)threadIdx.x;
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int k = base + q * kBlock;
        // equal digits of a warp are counted once: the keys come sorted by
        // their low digit, so many neighbours share the high one
        const uint32_t d = k < n ? (keys[k] >> shift) & (kBins - 1) : (uint32_t)kBins;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        if (k < n && (unsigned)(__ffs(peers) - 1) == (threadIdx.x & 31u))
            atomicAdd(&h[d], (uint32_t)__popc(peers));
    }
    __syncthreads();
    for (int b = threadIdx.x; b < kBins; b += kBlock) hist[(size_t)blockIdx.x * kBins + b] = h[b];
}

// Every digit's counts over the chunks become running sums, in place, and its
// total: 32 digits per block, one per lane (128-byte rows), the chunks split
// over the block's warps.
constexpr int kRowWarps = 16;
constexpr int kRowItems = (int)(kMaxBlocks / kRowWarps);
__global__ void __launch_bounds__(32 * kRowWarps)
    k_na_digit_rows(uint32_t* hist, int nblk, uint32_t* totals) {
    __shared__ uint32_t sums[kRowWarps][32];
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
    const int d = blockIdx.x * 32 + lane;
    const int per = (nblk + kRowWarps - 1) / kRowWarps, b0 = warp * per;
    uint32_t v[kRowItems];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kRowItems; ++k) {
        v[k] = k < per && b0 + k < nblk ? hist[(size_t)(b0 + k) * kBins + d] : 0u;
        sum += v[k];
    }
    sums[warp][lane] = sum;
    __syncthreads();
    uint32_t run = 0, all = 0;
    for (int w = 0; w < kRowWarps; ++w) {
        const uint32_t t = sums[w][lane];
        run += w < warp ? t : 0u;
        all += t;
    }
#pragma unroll
    for (int k = 0; k < kRowItems; ++k) {
        if (k < per && b0 + k < nblk) hist[(size_t)(b0 + k) * kBins + d] = run;
        run += v[k];
    }
    if (warp == 0) totals[d] = all;
}

// Exclusive scan of kBins values, two per thread (v: this thread's pair).
static_assert(kBins == 2 * kBlock, "two digits per thread");
__device__ __forceinline__ uint2 block_scan_bins(uint2 v, uint32_t* warp_sums) {
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v.x + v.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    uint32_t pre = 0;
    for (unsigned w = 0; w < warp; ++w) pre += warp_sums[w];
    __syncthreads();
    const uint32_t e = pre + x - (v.x + v.y);
    return make_uint2(e, e + v.x);
}

// Stable scatter of one chunk's (key, index) pairs by the digit at `shift`.
// Each warp ranks its own 256 consecutive elements, 32 per round
// (same_digit groups equal digits by one ballot per bit, 63 -> 59 us for the
// whole sort of 1,000,000 against __match_any_sync), in a digit table of its own; the
// tables' running sums over the warps, in order, then place every element
// after the earlier elements of its digit, so the order inside a digit is the
// input order.  The chunk is put in digit order in shared memory and written
// from there, runs of equal digits together.  (With one warp ranking 1,024
// elements and every element written from its own thread the two scatters of
// 1,000,000 particles took 26 and 13 us.)  idx_in == nullptr: the indices
// are the positions.
__device__ __forceinline__ unsigned same_digit(uint32_t d, bool valid) {
    unsigned m = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < kDigitBits; ++b) {
        const bool one = (d >> b) & 1u;
        const unsigned v = __ballot_sync(0xffffffffu, one);
        m &= one ? v : ~v;
    }
    return m;
}
struct ScatterShared {
    uint16_t cnt[kWarps][kBins];
    uint32_t key[kChunk], idx[kChunk];
    uint32_t dst[kBins];  // a digit's output position minus its position in the chunk
    uint32_t warp_sums[kWarps];
};
__global__ void __launch_bounds__(kBlock)
    k_na_digit_scatter(const uint32_t* __restrict__ keys, uint32_t bias,
                       const uint32_t* __restrict__ idx_in, int n, int shift,
                       const uint32_t* __restrict__ hist, const uint32_t* __restrict__ totals,
                       uint32_t* __restrict__ keys_out, uint32_t* __restrict__ idx_out) {
    extern __shared__ unsigned char raw[];
    ScatterShared& sh = *reinterpret_cast<ScatterShared*>(raw);
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const int base = blockIdx.x * kChunk;
    const int m = min(kChunk, n - base);
    uint32_t key[kItems], idx[kItems];
    const int e0 = (int)warp * (kItems * 32) + (int)lane;
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const int e = e0 + r * 32;
        key[r] = e < m ? keys[base + e] - bias : 0u;
        idx[r] = e < m ? (idx_in ? idx_in[base + e] : (uint32_t)(base + e)) : 0u;
    }
    const int d0 = 2 * (int)threadIdx.x;
    const uint2 tot = make_uint2(totals[d0], totals[d0 + 1]);
    const uint2 row = *reinterpret_cast<const uint2*>(hist + (size_t)blockIdx.x * kBins + d0);
    uint32_t* zero = reinterpret_cast<uint32_t*>(&sh.cnt[0][0]);
    for (int b = threadIdx.x; b < kWarps * kBins / 2; b += kBlock) zero[b] = 0u;
    __syncthreads();
    uint32_t rank[kItems];  // within the warp's elements of the same digit
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const bool valid = e0 + r * 32 < m;
        const uint32_t d = (key[r] >> shift) & (kBins - 1);
        const unsigned peers = same_digit(d, valid);
        uint32_t before = 0;
        if (valid) before = sh.cnt[warp][d];
        __syncwarp();
        rank[r] = before + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        if (valid && (unsigned)(__ffs(peers) - 1) == lane)
            sh.cnt[warp][d] = (uint16_t)(before + (uint32_t)__popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // the warps' counts of this thread's two digits become running sums
    uint2 c = make_uint2(0u, 0u);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const uint32_t u = reinterpret_cast<uint32_t*>(sh.cnt[w])[threadIdx.x];
        reinterpret_cast<uint32_t*>(sh.cnt[w])[threadIdx.x] = c.x | (c.y << 16);
        c.x += u & 0xffffu;
        c.y += u >> 16;
    }
    const uint2 local = block_scan_bins(c, sh.warp_sums);    // first place in the chunk
    const uint2 global = block_scan_bins(tot, sh.warp_sums);  // first place of the digit
    // the chunk's first place of each digit joins the warps' running sums
    // (at most kChunk, of a digit after all of them, so 16 bits hold it)
#pragma unroll
    for (int w = 0; w < kWarps; ++w)
        reinterpret_cast<uint32_t*>(sh.cnt[w])[threadIdx.x] += local.x | (local.y << 16);
    sh.dst[d0] = global.x + row.x - local.x;
    sh.dst[d0 + 1] = global.y + row.y - local.y;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        if (e0 + r * 32 < m) {
            const uint32_t at = sh.cnt[warp][(key[r] >> shift) & (kBins - 1)] + rank[r];
            sh.key[at] = key[r];
            sh.idx[at] = idx[r];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int e = q * kBlock + (int)threadIdx.x;
        if (e < m) {
            const uint32_t k = sh.key[e];
            const uint32_t dst = sh.dst[(k >> shift) & (kBins - 1)] + (uint32_t)e;
            idx_out[dst] = sh.idx[e];
            if (keys_out) keys_out[dst] = k;
        }
    }
}

std::mutex g_setup_mutex;
uint32_t* g_scratch_ptr[kMaxDevices] = {};

// Device address of g_scratch on the current device, looked up once per
// device (the first call on each device does this, so that call should come
// before any stream capture on that device).
int scratch_on(int device, uint32_t** out) {
    if (device < 0 || device >= kMaxDevices) return DEM_ERR_INVALID;
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_ptr[device]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_scratch) != cudaSuccess || !p) {
            cudaGetLastError();  // this call's own failure
            return DEM_ERR_CUDA;
        }
        // the scatter's shared memory is above the default limit
        if (cudaFuncSetAttribute(k_na_digit_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(ScatterShared)) != cudaSuccess) {
            cudaGetLastError();
            return DEM_ERR_CUDA;
        }
        g_scratch_ptr[device] = static_cast<uint32_t*>(p);
    }
    *out = g_scratch_ptr[device];
    return DEM_OK;
}

// The launch just queued: its configuration error, if any (a launch error is
// this call's own; the check at entry made sure none was pending before).
inline bool launched() { return cudaGetLastError() == cudaSuccess; }

}  // namespace

extern "C" int dem_bucket_sort_noalloc(const double* px, const double* py, const double* pz,
                                       int64_t n, const double* domain_min, double cell_size,
                                       int64_t hash_table_size, uint32_t* bucket,
                                       uint32_t* sorted, void* stream) {
    if (n < 0 || !domain_min || !(cell_size > 0) || hash_table_size < 1) return DEM_ERR_INVALID;
    if (n > kMaxN || hash_table_size > kMaxH) return DEM_ERR_CAPACITY;
    if (n > 0 && (!px || !py || !pz || !bucket || !sorted)) return DEM_ERR_INVALID;
    if (n == 0) return DEM_OK;
    // an error already pending on this thread belongs to someone else: it is
    // reported (DEM_ERR_CUDA) and left in place, and no work is queued
    if (cudaPeekAtLastError() != cudaSuccess) return DEM_ERR_CUDA;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return DEM_ERR_NO_DEVICE;
    uint32_t* scratch = nullptr;
    const int rc = scratch_on(device, &scratch);
    if (rc != DEM_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    uint32_t* keys_tmp = scratch + kKeysOff;
    uint32_t* idx_tmp = scratch + kValsOff;
    uint32_t* hist = scratch + kHistOff;
    uint32_t* totals = scratch + kTotalsOff;
    Geometry g;
    double dm = 0.0;
    for (int c = 0; c < 3; ++c) {
        g.dmin[c] = domain_min[c];  // host memory
        dm = std::fmax(dm, std::fabs(g.dmin[c]));
    }
    g.cell = cell_size;
    g.inv_cell32 = (float)(1.0 / cell_size);
    g.dmin_cells = (float)(dm / cell_size * 1.001);
    g.screen = cell_size > 0x1p-100 && cell_size < 0x1p100;
    g.H = (uint32_t)hash_table_size;
    g.mask = (g.H & (g.H - 1)) == 0 ? g.H - 1 : 0u;
    const int nn = (int)n;
    // buckets are 0 .. H-1 < 2^20: one 10-bit pass for H <= 1,024, else two
    const int passes = hash_table_size <= kBins ? 1 : 2;
    const int nblk = (nn + kChunk - 1) / kChunk;
    k_na_hash<<<nblk, kBlock, 0, s>>>(px, py, pz, nn, g, bucket, hist);
    if (!launched()) return DEM_ERR_CUDA;
    for (int pass = 0; pass < passes; ++pass) {
        const int shift = pass * kDigitBits;
        const bool last = pass == passes - 1;
        const uint32_t* kin = pass == 0 ? bucket : keys_tmp;
        const uint32_t bias = pass == 0 ? 1u : 0u;  // the outputs' buckets are 1-based
        const uint32_t* iin = pass == 0 ? nullptr : idx_tmp;
        if (pass > 0) {
            k_na_digit_count<<<nblk, kBlock, 0, s>>>(kin, nn, shift, hist);
            if (!launched()) return DEM_ERR_CUDA;
        }
        k_na_digit_rows<<<kBins / 32, 32 * kRowWarps, 0, s>>>(hist, nblk, totals);
        if (!launched()) return DEM_ERR_CUDA;
        k_na_digit_scatter<<<nblk, kBlock, sizeof(ScatterShared), s>>>(
            kin, bias, iin, nn, shift, hist, totals, last ? nullptr : keys_tmp,
            last ? sorted : idx_tmp);
        if (!launched()) return DEM_ERR_CUDA;
    }
    return DEM_OK;
}
