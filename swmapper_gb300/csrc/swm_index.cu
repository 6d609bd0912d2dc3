// swm_index.cu -- GPU k-mer index build, index files, device scan.
//
// Index build (serial_index.c:157-445, rebuilt for the GPU):
//   kb_encode   32 bases per thread -> lo/hi bit planes and N mask (get_seed,
//               serial_index.c:157-232)
//   kb_count    one thread per sampled position p = 4t: k-mer and N test
//               from the planes, atomic count (chromo_hash_index,
//               serial_index.c:253-269)
//   scan        start offsets (store_positions, serial_index.c:337-340)
//   kb_radix    the sampled positions ordered by k-mer: a stable radix sort
//               keeps each bucket in position order, the order the
//               reference's serial scatter produces (serial_index.c:343-352);
//               its last pass writes the resident index, positions (u32) and
//               flank codes (u16), the layout of .positions / .pos_lseeds
#include <errno.h>
#include <fcntl.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/stat.h>
#include <unistd.h>

#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "swm_common.cuh"
#include "swm_files.h"

// ----------------------------------------------------------------- errors

static thread_local char g_err[512] = "";

void swm_set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
}

extern "C" const char *swm_last_error(void) { return g_err; }

// ------------------------------------------------------------------- scan

#define SCAN_T 256
#define SCAN_V 8
#define SCAN_TILE (SCAN_T * SCAN_V)

uint64_t swm_scan_tmp_words(uint64_t n_cap) { return (n_cap + SCAN_TILE - 1) / SCAN_TILE + 64; }

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, d);
        if ((threadIdx.x & 31) >= d) v += t;
    }
    return v;
}

// exclusive block scan of one value per thread (blockDim.x == SCAN_T or 1024)
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *total) {
    __shared__ uint32_t wsum[33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    uint32_t inc = warp_incl_scan(v);
    if (lane == 31) wsum[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        uint32_t s = lane < nw ? wsum[lane] : 0u;
        uint32_t si = warp_incl_scan(s);
        if (lane < nw) wsum[lane] = si - s;
        if (lane == nw - 1) wsum[32] = si;
    }
    __syncthreads();
    uint32_t r = inc - v + wsum[wid];
    if (total) *total = wsum[32];
    __syncthreads();
    return r;
}

__device__ __forceinline__ uint64_t scan_n(const uint32_t *d_n, uint64_t n_host, uint64_t n_cap) {
    uint64_t n = d_n ? (uint64_t)*d_n : n_host;
    return n < n_cap ? n : n_cap;
}

// Sum of one 64-bit value per thread over the block (every thread gets it).
__device__ __forceinline__ uint64_t block_sum_u64(uint64_t v) {
    __shared__ unsigned long long wsum64[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if (lane == 0) wsum64[wid] = v;
    __syncthreads();
    uint64_t t = 0;
    for (int w = 0; w < nw; w++) t += wsum64[w];
    __syncthreads();
    return t;
}

// Totals are 32-bit: a sum that does not fit saturates to SWM_SCAN_SATURATED
// (each tile's partial, then the total), so callers see an overflow instead
// of a wrapped value.
__global__ void k_scan_reduce(const uint32_t *__restrict__ in, const uint32_t *d_n, uint64_t n_host, uint64_t n_cap,
                              uint32_t *__restrict__ part) {
    const uint64_t n = scan_n(d_n, n_host, n_cap);
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    uint64_t s = 0;
    if (base < n) {
#pragma unroll
        for (int v = 0; v < SCAN_V; v++) {
            uint64_t i = base + threadIdx.x + (uint64_t)v * SCAN_T;
            if (i < n) s += in[i];
        }
    }
    const uint64_t tot = block_sum_u64(s);
    if (threadIdx.x == 0)
        part[blockIdx.x] = (base < n) ? (tot < SWM_SCAN_SATURATED ? (uint32_t)tot : SWM_SCAN_SATURATED) : 0u;
}

__global__ void k_scan_top(uint32_t *part, const uint32_t *d_n, uint64_t n_host, uint64_t n_cap, uint32_t *out,
                           uint32_t *d_total) {
    const uint64_t n = scan_n(d_n, n_host, n_cap);
    const uint64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    const uint64_t per = (nb + blockDim.x - 1) / blockDim.x;
    const uint64_t b0 = threadIdx.x * per;
    uint32_t s = 0;
    uint64_t s64 = 0;
    for (uint64_t i = b0; i < b0 + per && i < nb; i++) {
        s += part[i];
        s64 += part[i];
    }
    const uint64_t tot64 = block_sum_u64(s64);
    uint32_t tot;
    uint32_t ex = block_excl_scan(s, &tot);
    for (uint64_t i = b0; i < b0 + per && i < nb; i++) {
        uint32_t v = part[i];
        part[i] = ex;
        ex += v;
    }
    if (threadIdx.x == 0) {
        if (tot64 >= SWM_SCAN_SATURATED) tot = SWM_SCAN_SATURATED;
        out[n] = tot;
        if (d_total) *d_total = tot;
    }
}

__global__ void k_scan_down(const uint32_t *__restrict__ in, const uint32_t *d_n, uint64_t n_host, uint64_t n_cap,
                            const uint32_t *__restrict__ part, uint32_t *__restrict__ out) {
    const uint64_t n = scan_n(d_n, n_host, n_cap);
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    if (base >= n) return;
    const uint64_t i0 = base + (uint64_t)threadIdx.x * SCAN_V;
    uint32_t v[SCAN_V];
    const bool whole = i0 + SCAN_V <= n && (((uintptr_t)in | (uintptr_t)out) & 15) == 0;
    if (whole) {
        const uint4 a = reinterpret_cast<const uint4 *>(in + i0)[0], b = reinterpret_cast<const uint4 *>(in + i0)[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < SCAN_V; j++) v[j] = (i0 + j < n) ? in[i0 + j] : 0u;
    }
    uint32_t s = 0;
#pragma unroll
    for (int j = 0; j < SCAN_V; j++) s += v[j];
    uint32_t ex = block_excl_scan(s, nullptr) + part[blockIdx.x];
#pragma unroll
    for (int j = 0; j < SCAN_V; j++) { // each becomes its exclusive prefix
        const uint32_t x = v[j];
        v[j] = ex;
        ex += x;
    }
    if (whole) {
        reinterpret_cast<uint4 *>(out + i0)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4 *>(out + i0)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int j = 0; j < SCAN_V; j++)
            if (i0 + j < n) out[i0 + j] = v[j];
    }
}

int swm_exclusive_scan(const uint32_t *d_in, uint32_t *d_out, const uint32_t *d_n, uint64_t n_host, uint64_t n_cap,
                       uint32_t *d_tmp, uint32_t *d_total, cudaStream_t st) {
    const uint64_t nb = (n_cap + SCAN_TILE - 1) / SCAN_TILE;
    const unsigned grid = (unsigned)(nb ? nb : 1);
    k_scan_reduce<<<grid, SCAN_T, 0, st>>>(d_in, d_n, n_host, n_cap, d_tmp);
    k_scan_top<<<1, 1024, 0, st>>>(d_tmp, d_n, n_host, n_cap, d_out, d_total);
    k_scan_down<<<grid, SCAN_T, 0, st>>>(d_in, d_n, n_host, n_cap, d_tmp, d_out);
    SWM_CUDA(cudaGetLastError());
    return SWM_OK;
}

// ------------------------------------------------------------ index build

// Four sequence bytes -> 4 lo bits, 4 hi bits, 4 "not A/C/G/T" bits, base j at
// bit j. Lower case counts as upper case (serial_index.c:152); the code
// ((c >> 1) ^ (c >> 2)) & 3 maps A C G T to 0 1 2 3, anything else encodes as 0.
// The letter of each byte's code (one byte permute) tells whether the byte was
// one of the four; almost always all are.
__device__ __forceinline__ void encode4(uint32_t w, uint32_t &lo, uint32_t &hi, uint32_t &nm) {
    w &= 0xdfdfdfdfu;
    uint32_t c = ((w >> 1) ^ (w >> 2)) & 0x03030303u;
    const uint32_t y = (c | (c >> 4)) & 0x00ff00ffu; // codes as permute selectors, a nibble each
    const uint32_t x = __byte_perm(0x54474341u, 0u, y | (y >> 8)) ^ w;
    nm = 0;
    if (x) {
        uint32_t bad = x | (x >> 4);
        bad |= bad >> 2;
        bad = (bad | (bad >> 1)) & 0x01010101u; // bytes that differ
        c &= ~(bad * 3u);
        nm = (bad * 0x10204080u) >> 28;
    }
    lo = ((c & 0x01010101u) * 0x10204080u) >> 28;
    hi = (((c >> 1) & 0x01010101u) * 0x10204080u) >> 28;
}

__global__ void kb_encode(const uint8_t *__restrict__ seq, uint64_t n, uint32_t *__restrict__ b2,
                          uint32_t *__restrict__ b3) {
    const uint64_t W = (n + 31) / 32;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < W; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t p0 = w * 32;
        const uint32_t cnt = (n - p0 >= 32) ? 32u : (uint32_t)(n - p0);
        uint32_t q[8];
        if (cnt == 32 && (((uintptr_t)(seq + p0)) & 15) == 0) {
            const uint4 *v = reinterpret_cast<const uint4 *>(seq + p0);
            const uint4 a = __ldcs(v), b = __ldcs(v + 1);
            q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
            q[4] = b.x; q[5] = b.y; q[6] = b.z; q[7] = b.w;
        } else { // unaligned sequence, or the last partial word
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) {
                q[j] = 0;
#pragma unroll
                for (uint32_t i = 0; i < 4; i++)
                    if (4 * j + i < cnt) q[j] |= (uint32_t)seq[p0 + 4 * j + i] << (8 * i);
            }
        }
        uint32_t lo = 0, hi = 0, nm = 0;
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) {
            uint32_t l, h, m;
            encode4(q[j], l, h, m);
            lo |= l << (4 * j);
            hi |= h << (4 * j);
            nm |= m << (4 * j);
        }
        if (cnt < 32) nm &= (1u << cnt) - 1u; // bases past the end are not N
        reinterpret_cast<uint2 *>(b2)[w] = make_uint2(lo, hi);
        b3[w] = nm;
    }
}

// k-mer at sampled position i (get_seed_from_enc_bits, serial_index.c:280-331);
// false when it holds an N. With FLANK also its flank code: 3 bases before
// (bases 0 .. 2 when i is 0) and 3 after, lo bits then hi bits. One 32-base
// window from i - 3 holds both (k <= 14).
template <bool FLANK>
__device__ __forceinline__ bool seed_at(const uint2 *__restrict__ b2p, const uint32_t *__restrict__ b3, uint64_t i,
                                        uint32_t k, uint32_t *seed, uint32_t *flank) {
    const uint32_t res = SWM_SEED_STEP - 1, rmask = (1u << res) - 1, mask = (1u << k) - 1;
    const uint64_t w = i / 32;
    const uint32_t sh = (uint32_t)(i % 32);
    if (swm_fsr(b3[w], b3[w + 1], sh) & mask) return false;
    const uint32_t f = i >= res ? res : 0u; // bases of the window before the k-mer
    const uint64_t q = (i - f) / 32;
    const uint32_t qs = (uint32_t)((i - f) % 32);
    const uint2 a = b2p[q], b = b2p[q + 1];
    const uint32_t lo = swm_fsr(a.x, b.x, qs), hi = swm_fsr(a.y, b.y, qs);
    *seed = swm_spread16((lo >> f) & mask) | (swm_spread16((hi >> f) & mask) << 1);
    if (FLANK)
        *flank = (lo & rmask) | ((lo >> (f + k)) & rmask) << res | (hi & rmask) << (2 * res) |
                 ((hi >> (f + k)) & rmask) << (3 * res);
    return true;
}

// ------------------------------------------------ ordering the positions
//
// The reference's scatter visits positions in ascending order, so a bucket's
// entries ascend. A stable least-significant-digit radix sort of the samples
// by k-mer gives that order with streaming passes only: 6.2 ms for 1 Gbp (250 M
// samples, k = 12) where an atomic scatter to 8-byte slots and a sort of every
// bucket took 35 ms (each entry's random write moved a whole DRAM burst, one
// atomic per bucket on three counters serialised the bucket lists, and the
// sorts read and wrote the buckets once more).
//
// An entry travels as one 64-bit key: flank code (12 bits), position / 4 (30)
// and the digits of the k-mer still to be sorted by (at most 21 bits: the first
// pass makes the key from the planes and sorts by the lowest digit right
// away). Every pass cuts its input into one contiguous chunk per resident
// block: the chunks' digit counts (kb_count for the first pass, kb_hist for
// the others), scanned digit by digit, give each chunk the place of its first
// key of every digit, and a block then moves its chunk tile by tile; no block
// waits for another. A middle pass over 1 Gbp takes 1.33 ms and its counts 0.26;
// one kernel whose tiles look back at the counts of the tiles before them took
// 1.64. The ALU pipe (65% busy: ranking, 32 keys a warp) and the latency of a
// tile's phases bound a pass, DRAM is at 3.1 TB/s; 4 blocks of 256 threads an
// SM (64 registers) were faster than 3 (80): 1.33 against 1.37 ms.
#define RADIX_BINS 256
#define RADIX_THREADS 256 // one thread per digit
#define RADIX_ITEMS 16
#define RADIX_TILE (RADIX_THREADS * RADIX_ITEMS)
#define RADIX_WARPS (RADIX_THREADS / 32)
#define RADIX_BLOCKS_PER_SM 4
#define RADIX_MAX_PASSES 4
#define RADIX_LS_BITS 12
#define RADIX_SEED_SHIFT 42 // flank code, then 30 bits of position / 4

// Bucket counts of every sample of [0, T), and the lowest digit's count per
// chunk of `chunk` samples (one per block) in hist[digit * gridDim.x + block].
__global__ void __launch_bounds__(512) kb_count(const uint2 *__restrict__ b2p, const uint32_t *__restrict__ b3,
                                                uint64_t T, uint64_t chunk, uint32_t k, uint32_t bits,
                                                uint32_t *__restrict__ count, uint32_t *__restrict__ hist) {
    __shared__ uint32_t h[RADIX_BINS];
    if (threadIdx.x < RADIX_BINS) h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t t0 = blockIdx.x * chunk, t1 = t0 + chunk < T ? t0 + chunk : T;
    for (uint64_t t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
        uint32_t sd;
        if (seed_at<false>(b2p, b3, t * SWM_SEED_STEP, k, &sd, nullptr)) {
            atomicAdd(&count[sd], 1u);
            atomicAdd(&h[sd & ((1u << bits) - 1)], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x < RADIX_BINS) hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// The same counts of one digit of *n keys, cut into gridDim.x chunks.
__device__ __forceinline__ uint64_t radix_chunk(uint64_t n, uint32_t chunks) {
    const uint64_t tiles = (n + RADIX_TILE - 1) / RADIX_TILE;
    return (tiles + chunks - 1) / chunks * RADIX_TILE;
}
__global__ void __launch_bounds__(512) kb_hist(const unsigned long long *__restrict__ in,
                                               const uint32_t *__restrict__ n, uint32_t shift, uint32_t bits,
                                               uint32_t *__restrict__ hist) {
    __shared__ uint32_t h[RADIX_BINS];
    if (threadIdx.x < RADIX_BINS) h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t total = *n, chunk = radix_chunk(total, gridDim.x);
    const uint64_t t0 = blockIdx.x * chunk, t1 = t0 + chunk < total ? t0 + chunk : total;
    const uint32_t dmask = (1u << bits) - 1;
    // chunks start at whole tiles: two keys per load
    for (uint64_t t = t0 + 2 * threadIdx.x; t < t1; t += 2 * blockDim.x) {
        const ulonglong2 v = __ldcs(reinterpret_cast<const ulonglong2 *>(in + t));
        atomicAdd(&h[(uint32_t)(v.x >> (RADIX_SEED_SHIFT + shift)) & dmask], 1u);
        if (t + 1 < t1) atomicAdd(&h[(uint32_t)(v.y >> (RADIX_SEED_SHIFT + shift)) & dmask], 1u);
    }
    __syncthreads();
    if (threadIdx.x < RADIX_BINS) hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

struct RadixSmem {
    union {
        unsigned long long key[RADIX_TILE];        // the tile in digit order
        uint32_t cnt[RADIX_WARPS][RADIX_BINS];     // before that: counts per warp and digit
    };
    uint32_t base[RADIX_BINS]; // first output index of the digit minus its first place in the tile
};

// One pass: the block's chunk in tiles. FIRST: the keys come from the planes
// (sample t of T at position 4 t; samples with an N are left out); otherwise
// from in, *n of them. LAST: the entries go to pos / ls instead of out. first:
// the scanned counts (see kb_count). A tile's keys are ranked by digit within
// their warp (one ballot per digit bit; match instructions took 40% longer, and
// masks made with shared-memory atomics moved the limit from the ALU to the
// shared-memory pipe) and written through shared memory, so that each digit's
// keys go out as one run of consecutive addresses. In shared memory a key of
// the first pass holds its place in the tile and its digit where the position
// goes, so that the digit can be read back.
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(RADIX_THREADS, RADIX_BLOCKS_PER_SM)
    kb_radix(const uint2 *__restrict__ b2p, const uint32_t *__restrict__ b3, uint64_t T, uint64_t chunk_first, uint32_t k,
             const unsigned long long *__restrict__ in, const uint32_t *__restrict__ n, uint32_t shift, uint32_t bits,
             const uint32_t *__restrict__ first, unsigned long long *__restrict__ out, uint32_t *__restrict__ pos,
             uint16_t *__restrict__ ls) {
    __shared__ RadixSmem S;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t total = FIRST ? T : (uint64_t)*n;
    const uint64_t chunk = FIRST ? chunk_first : radix_chunk(total, gridDim.x);
    const uint64_t t0 = blockIdx.x * chunk, t1 = t0 + chunk < total ? t0 + chunk : total;
    const uint32_t dmask = (1u << bits) - 1;
    const uint32_t dsh = RADIX_SEED_SHIFT - 32 + shift; // of the digit in a key's high word
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    uint32_t next = first[tid * gridDim.x + blockIdx.x]; // output index of the chunk's next key of digit tid
    uint32_t *cnt = S.cnt[warp];
    for (uint64_t base = t0; base < t1; base += RADIX_TILE) {
        // ---- the tile's keys: warp w holds its 512 in rows of 32
        const uint32_t left = t1 - base < RADIX_TILE ? (uint32_t)(t1 - base) : RADIX_TILE;
        const uint32_t w0 = warp * (32 * RADIX_ITEMS) + lane;
        unsigned long long key[RADIX_ITEMS];
        uint32_t at[RADIX_ITEMS]; // digit (RADIX_BINS: no key) | place << 16
#pragma unroll
        for (int j = 0; j < RADIX_ITEMS; j++) {
            const uint32_t i = w0 + 32 * j;
            at[j] = RADIX_BINS;
            key[j] = 0;
            if (i < left) {
                if (FIRST) {
                    uint32_t sd, fl;
                    if (seed_at<true>(b2p, b3, (base + i) * SWM_SEED_STEP, k, &sd, &fl)) {
                        at[j] = sd & dmask;
                        key[j] = (unsigned long long)(sd >> bits) << RADIX_SEED_SHIFT | i << RADIX_LS_BITS | fl;
                    }
                } else {
                    key[j] = __ldcs(in + base + i);
                    at[j] = ((uint32_t)(key[j] >> 32) >> dsh) & dmask;
                }
            }
        }
#pragma unroll
        for (int w = 0; w < RADIX_WARPS; w++) S.cnt[w][tid] = 0;
        __syncthreads();
        // ---- rank of each key among its warp's keys of the same digit
#pragma unroll
        for (int j = 0; j < RADIX_ITEMS; j++) {
            const uint32_t d = at[j];
            const bool have = d < RADIX_BINS;
            uint32_t mm = __ballot_sync(0xffffffffu, have); // lanes with the same digit
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const bool on = (d & (1u << q)) != 0;
                const uint32_t b = __ballot_sync(0xffffffffu, on);
                mm &= on ? b : ~b;
            }
            const uint32_t below = mm & lt;
            uint32_t c = 0;
            if (have) c = cnt[d];
            at[j] = d | (c + __popc(below)) << 16;
            __syncwarp();
            if (have && !below) cnt[d] = c + __popc(mm);
            __syncwarp();
        }
        __syncthreads();
        // ---- thread d owns digit d: the warps' counts become places in the tile
        uint32_t mine = 0;
#pragma unroll
        for (int w = 0; w < RADIX_WARPS; w++) {
            const uint32_t c = S.cnt[w][tid];
            S.cnt[w][tid] = mine;
            mine += c;
        }
        uint32_t tile_n;
        const uint32_t loc = block_excl_scan(mine, &tile_n);
        S.base[tid] = next - loc;
        next += mine;
#pragma unroll
        for (int w = 0; w < RADIX_WARPS; w++) S.cnt[w][tid] += loc;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < RADIX_ITEMS; j++) {
            const uint32_t d = at[j] & 0xffffu;
            if (d < RADIX_BINS) at[j] += cnt[d] << 16;
        }
        __syncthreads(); // the counts are read: the keys take their place
#pragma unroll
        for (int j = 0; j < RADIX_ITEMS; j++) {
            const uint32_t d = at[j] & 0xffffu;
            if (d < RADIX_BINS) S.key[at[j] >> 16] = FIRST ? key[j] | (unsigned long long)d << 32 : key[j];
        }
        __syncthreads();
#pragma unroll 4
        for (uint32_t i = tid; i < tile_n; i += RADIX_THREADS) {
            const unsigned long long v = S.key[i];
            const uint32_t hi = (uint32_t)(v >> 32);
            const uint32_t o = S.base[FIRST ? hi & (RADIX_BINS - 1) : (hi >> dsh) & dmask] + i;
            const uint32_t t = FIRST ? (uint32_t)base + ((uint32_t)v >> RADIX_LS_BITS)
                                     : (uint32_t)(v >> RADIX_LS_BITS) & 0x3fffffffu;
            if (LAST) {
                pos[o] = t * SWM_SEED_STEP;
                ls[o] = (uint16_t)(v & ((1u << RADIX_LS_BITS) - 1));
            } else if (FIRST) {
                const unsigned long long ends = (1ull << RADIX_LS_BITS) - 1 | ~0ull << RADIX_SEED_SHIFT;
                out[o] = (v & ends) | (unsigned long long)t << RADIX_LS_BITS;
            } else {
                out[o] = v;
            }
        }
        __syncthreads(); // the next tile's counts overwrite the keys
    }
}

// ---------------------------------------------------- candidate table
//
// long_seeds_filter (mapper_cpe.c:2090-2123) keeps an entry of a seed's
// bucket when the 3 flank bits of each plane at the seed's shift equal the
// read's, i.e. when the whole 15-base long seed matches. The table groups the
// genome's entries by 15-mer and, within one, by the shift t at which the
// entry's 12-mer lies in it (stable: ascending position inside a group), so
// that the entries one (seed, shift, read flank) keeps are one contiguous range
// of positions, found with a single offset lookup, and the four shifts of a
// long seed look up neighbouring offsets and read neighbouring ranges: a read's
// lookups touch one sector of the 17 GiB offset array per long seed instead of
// one per shift, and so do its positions (ordered by bucket, shift and flank,
// the table made the candidate stage 27% and the seed stage, which stored a key
// per seed, 32% slower: 2.18 and 0.80 against 1.72 and 0.61 ms per 524,288 reads of
// 150 bp on 3.1 Gbp). ctab_off[4 key15 + t] is where a
// group starts and ctab_off[4 key15 + t + 1] where it ends (the last entry
// holds 4 * n_seeds); swm_ctab_key15 gives the key.

#define CTAB_THREADS 512
#define CTAB_CORES (1u << 18)  // codes of the 9 bases every shift's 12-mer holds: one partition each
#define CTAB_KEYS_CORE (1u << 14)
#define CTAB_BUCKETS_CORE 256  // buckets that hold a core: 64 at each shift

// Bucket q of core c9: shift t = q / 64, and the 3 bases of its 12-mer outside
// the core from q % 64 (3 - t before it, t after).
__device__ __forceinline__ uint32_t ctab_bucket(uint32_t c9, uint32_t q) {
    const uint32_t t = q >> 6, w = q & 63u, nl = 2 * (3 - t);
    return (w & ((1u << nl) - 1)) | (c9 << nl) | ((w >> nl) << (24 - 2 * t));
}

// Key within the core's partition of an entry of its bucket q with flank value
// v (swm_ctab_flank at shift t): the 15-mer's 6 outer bases, then t.
__device__ __forceinline__ uint32_t ctab_local(uint32_t q, uint32_t v) {
    const uint32_t t = q >> 6, w = q & 63u, nl = 2 * (3 - t);
    const uint32_t f = (v & 1u) | (v & 8u) >> 2 | (v & 2u) << 1 | (v & 16u) >> 1 | (v & 4u) << 2 | (v & 32u); // 2 bits a base
    const uint32_t outer = (f & ((1u << (2 * t)) - 1)) | (w & ((1u << nl) - 1)) << (2 * t) | (w >> nl) << 6 |
                           (f >> (2 * t)) << (6 + 2 * t);
    return outer << 2 | t;
}

// entries of every partition (a warp each)
__global__ void __launch_bounds__(256) kb_ctab_sums(const uint32_t *__restrict__ count, uint32_t *__restrict__ sums) {
    const uint32_t lane = threadIdx.x & 31, c9 = (blockIdx.x * 256 + threadIdx.x) >> 5;
    if (c9 >= CTAB_CORES) return;
    uint32_t s = 0;
    for (uint32_t q = lane; q < CTAB_BUCKETS_CORE; q += 32) s += count[ctab_bucket(c9, q)];
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) sums[c9] = s;
}

// One block per core at a time: a histogram of the core's 16,384 keys over the
// entries of its 256 buckets in shared memory, its exclusive scan (written out
// as one 64 KB row of offsets), and a stable scatter of the positions. A
// bucket's entries have keys of their own, so one warp takes each bucket and
// its match masks keep the order.
__global__ void __launch_bounds__(CTAB_THREADS, 3) kb_ctab(const uint32_t *__restrict__ off,
                                                           const uint32_t *__restrict__ pos,
                                                           const uint16_t *__restrict__ ls,
                                                           const uint32_t *__restrict__ base,
                                                           uint32_t *__restrict__ ctab_off,
                                                           uint32_t *__restrict__ ctab_pos) {
    extern __shared__ __align__(16) uint32_t ctab_smem[];
    uint32_t *hist = ctab_smem;                       // CTAB_KEYS_CORE
    uint32_t *bo = ctab_smem + CTAB_KEYS_CORE;        // bucket starts
    uint32_t *bc = bo + CTAB_BUCKETS_CORE;            // bucket counts
    __shared__ uint32_t wtot[CTAB_THREADS / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nwarps = CTAB_THREADS / 32;
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    for (uint32_t c9 = blockIdx.x; c9 < CTAB_CORES; c9 += gridDim.x) {
        for (uint32_t i = tid; i < CTAB_KEYS_CORE / 4; i += CTAB_THREADS)
            reinterpret_cast<uint4 *>(hist)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (tid < CTAB_BUCKETS_CORE) {
            const uint32_t b = ctab_bucket(c9, tid), o = off[b];
            bo[tid] = o;
            bc[tid] = off[b + 1] - o;
        }
        __syncthreads();
        for (uint32_t q = warp; q < CTAB_BUCKETS_CORE; q += nwarps)
            for (uint32_t j = lane; j < bc[q]; j += 32)
                atomicAdd(&hist[ctab_local(q, swm_ctab_flank(ls[bo[q] + j], q >> 6))], 1u);
        __syncthreads();
        // exclusive scan, 1,024 keys per warp in rows of 32
        const uint32_t per = CTAB_KEYS_CORE / nwarps, k0 = warp * per;
        uint32_t run = 0;
        for (uint32_t j = 0; j < per; j += 32) {
            const uint32_t v = hist[k0 + j + lane], inc = warp_incl_scan(v);
            hist[k0 + j + lane] = run + inc - v;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) wtot[warp] = run;
        __syncthreads();
        uint32_t at = base[c9];
        for (uint32_t w = 0; w < warp; w++) at += wtot[w];
        uint32_t *row = ctab_off + (uint64_t)c9 * CTAB_KEYS_CORE;
        for (uint32_t j = lane; j < per; j += 32) {
            const uint32_t v = hist[k0 + j] + at;
            hist[k0 + j] = v; // now the running cursor of the key
            __stcs(row + k0 + j, v);
        }
        __syncthreads();
        for (uint32_t q = warp; q < CTAB_BUCKETS_CORE; q += nwarps) {
            const uint32_t o = bo[q], c = bc[q];
            for (uint32_t j0 = 0; j0 < c; j0 += 32) {
                const bool in = j0 + lane < c;
                const uint32_t p = in ? pos[o + j0 + lane] : 0u;
                const uint32_t k = in ? ctab_local(q, swm_ctab_flank(ls[o + j0 + lane], q >> 6)) : CTAB_KEYS_CORE + lane;
                const uint32_t mm = __match_any_sync(0xffffffffu, k); // lanes past the end match nobody
                uint32_t w = 0;
                if (in) w = hist[k] + __popc(mm & lt);
                __syncwarp();
                if (in) {
                    ctab_pos[w] = p;
                    if ((mm & lt) == 0) hist[k] += __popc(mm);
                }
                __syncwarp();
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------ refill schedule keys

// one thread per bucket (most have a few keys; a large one's are 128 bytes
// apart, so its thread's reads are no worse than others')
__global__ void __launch_bounds__(256) kb_keys32(const uint32_t *__restrict__ off, uint64_t nb,
                                                 const uint32_t *__restrict__ pos, uint32_t *__restrict__ keys) {
    for (uint64_t b = (uint64_t)blockIdx.x * 256 + threadIdx.x; b < nb; b += (uint64_t)gridDim.x * 256) {
        const uint32_t end = off[b + 1];
        for (uint64_t g = (uint64_t)off[b] + SWM_PER_FETCH - 1; g + 1 < end; g += SWM_PER_FETCH)
            keys[g / SWM_PER_FETCH] = pos[g];
    }
}

// ----------------------------------------------------------- host helpers

static int sm_count(int device) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
    return n > 0 ? n : 1;
}

static unsigned grid_for(uint64_t work, unsigned threads, int device, int per_sm = 8) {
    uint64_t g = (work + threads - 1) / threads;
    uint64_t cap = (uint64_t)sm_count(device) * per_sm;
    if (g > cap) g = cap;
    return (unsigned)(g ? g : 1);
}

static void index_release(swm_index *ix) {
    if (!ix) return;
    if (ix->chain_ev) cudaEventDestroy(ix->chain_ev);
    cudaFree(ix->d_ctab_off);
    cudaFree(ix->d_ctab_pos);
    cudaFree(ix->d_keys32);
    if (ix->arena) { // a built index: its arrays are parts of one allocation
        cudaFree(ix->arena);
    } else {
        cudaFree(ix->d_count);
        cudaFree(ix->d_off);
        cudaFree(ix->d_pos);
        cudaFree(ix->d_ls);
        cudaFree(ix->d_b2);
        cudaFree(ix->d_b3);
    }
    free(ix);
}

template <typename T>
static int dalloc(T **p, uint64_t count) {
    *p = nullptr;
    cudaError_t e = cudaMalloc((void **)p, (count ? count : 1) * sizeof(T));
    if (e != cudaSuccess) {
        swm_set_error("cudaMalloc(%llu bytes): %s", (unsigned long long)(count * sizeof(T)), cudaGetErrorString(e));
        *p = nullptr;
        return SWM_ERR_OOM;
    }
    return SWM_OK;
}

// Sizes of the parts of one device allocation, each part 256-byte aligned.
struct Parts {
    uint64_t bytes = 0;
    uint64_t add(uint64_t b) {
        const uint64_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    }
};

static int build_on_device(const uint8_t *d_seq, uint64_t n, uint32_t k, int device, swm_index **out) {
    if (k < 1 || k > 14 || n >= 0xffffffffull) {
        swm_set_error("swm_index_build: k must be in [1, 14] and n < 2^32 (k=%u n=%llu)", k, (unsigned long long)n);
        return SWM_ERR_ARG;
    }
    SWM_CUDA(cudaSetDevice(device));
    swm_index *ix = (swm_index *)calloc(1, sizeof(swm_index));
    if (!ix) return SWM_ERR_OOM;
    ix->device = device;
    ix->k = k;
    ix->n = n;
    const uint64_t W = (n + 31) / 32;
    const uint64_t nb = 1ull << (2 * k);
    ix->n_words2 = 2 * W;
    ix->n_words3 = W;
    ix->ref_length = ix->n_words2 * 4 * 16;
    cudaStream_t st = 0;
    uint8_t *d_tmp = nullptr;
#define CUC(x)                                                                                   \
    do {                                                                                         \
        cudaError_t e_ = (x);                                                                    \
        if (e_ != cudaSuccess) {                                                                 \
            swm_set_error("%s:%d %s: %s", __FILE__, __LINE__, #x, cudaGetErrorString(e_));       \
            cudaFree(d_tmp);                                                                     \
            index_release(ix);                                                                   \
            return SWM_ERR_CUDA;                                                                 \
        }                                                                                        \
    } while (0)
    // One allocation for the index and one for the scratch: an allocation and
    // its release cost 80 us and more (measured), which for a small genome is
    // most of a build. There are at most T = one per four bases entries, so
    // their arrays are sized before the count is known.
    const uint64_t T = (n >= k) ? (n - k) / SWM_SEED_STEP + 1 : 0;
    const uint64_t tiles = (T + RADIX_TILE - 1) / RADIX_TILE;
    const uint64_t resident = (uint64_t)sm_count(device) * RADIX_BLOCKS_PER_SM;
    const unsigned chunks = (unsigned)(tiles < resident ? tiles : resident);
    const uint64_t chunk = chunks ? (tiles + chunks - 1) / chunks * RADIX_TILE : 0;
    const uint32_t passes = (2 * k + 7) / 8;
    uint32_t digit_at[RADIX_MAX_PASSES], digit_bits[RADIX_MAX_PASSES]; // as even as 2k bits allow
    for (uint32_t q = 0, at = 0; q < passes; q++) {
        digit_at[q] = at;
        digit_bits[q] = (2 * k - at + passes - q - 1) / (passes - q);
        at += digit_bits[q];
    }
    Parts ip, tp;
    const uint64_t o_b2 = ip.add((ix->n_words2 + SWM_PAD_WORDS) * 4), o_b3 = ip.add((ix->n_words3 + SWM_PAD_WORDS) * 4);
    const uint64_t o_count = ip.add(nb * 4), o_off = ip.add((nb + 1) * 4);
    const uint64_t o_pos = ip.add((T + 8) * 4), o_ls = ip.add((T + 8) * 2);
    const uint64_t nhist = (uint64_t)RADIX_BINS * chunks;
    const uint64_t o_scan = tp.add(swm_scan_tmp_words(nb > nhist ? nb : nhist) * 4);
    const uint64_t o_hist = tp.add(nhist * 4), o_first = tp.add((nhist + 1) * 4);
    // keys between the passes, two buffers in turn
    const uint64_t o_a = tp.add(passes > 1 ? T * 8 + 16 : 0), o_b = tp.add(passes > 2 ? T * 8 + 16 : 0);
    if (cudaMalloc(&ix->arena, ip.bytes) != cudaSuccess || cudaMalloc(&d_tmp, tp.bytes) != cudaSuccess) {
        cudaGetLastError();
        swm_set_error("cudaMalloc(index %llu + scratch %llu bytes) failed", (unsigned long long)ip.bytes,
                      (unsigned long long)tp.bytes);
        index_release(ix);
        return SWM_ERR_OOM;
    }
    uint8_t *base = (uint8_t *)ix->arena;
    ix->d_b2 = (uint32_t *)(base + o_b2);
    ix->d_b3 = (uint32_t *)(base + o_b3);
    ix->d_count = (uint32_t *)(base + o_count);
    ix->d_off = (uint32_t *)(base + o_off);
    ix->d_pos = (uint32_t *)(base + o_pos);
    ix->d_ls = (uint16_t *)(base + o_ls);
    uint32_t *d_scan = (uint32_t *)(d_tmp + o_scan), *d_hist = (uint32_t *)(d_tmp + o_hist);
    uint32_t *d_first = (uint32_t *)(d_tmp + o_first);
    unsigned long long *d_key[2] = {(unsigned long long *)(d_tmp + o_a), (unsigned long long *)(d_tmp + o_b)};
    auto scan = [&](const uint32_t *in, uint32_t *o, uint64_t count) {
        return swm_exclusive_scan(in, o, nullptr, count, count, d_scan, nullptr, st) == SWM_OK;
    };
#define SCAN(in, o, count)             \
    do {                               \
        if (!scan(in, o, count)) {     \
            cudaFree(d_tmp);           \
            index_release(ix);         \
            return SWM_ERR_CUDA;       \
        }                              \
    } while (0)
    CUC(cudaMemsetAsync(ix->d_b2 + ix->n_words2, 0, SWM_PAD_WORDS * 4, st));
    CUC(cudaMemsetAsync(ix->d_b3 + ix->n_words3, 0, SWM_PAD_WORDS * 4, st));
    CUC(cudaMemsetAsync(ix->d_count, 0, nb * 4, st));
    const uint2 *b2p = (const uint2 *)ix->d_b2;
    if (W) kb_encode<<<grid_for(W, 256, device, 16), 256, 0, st>>>(d_seq, n, ix->d_b2, ix->d_b3);
    if (T) kb_count<<<chunks, 512, 0, st>>>(b2p, ix->d_b3, T, chunk, k, digit_bits[0], ix->d_count, d_hist);
    CUC(cudaGetLastError());
    SCAN(ix->d_count, ix->d_off, nb);
    const uint32_t *d_n = ix->d_off + nb; // entries
    for (uint32_t q = 0; T && q < passes; q++) {
        const bool first = q == 0, last = q + 1 == passes;
        const uint32_t shift = first ? 0 : digit_at[q] - digit_bits[0];
        if (!first) kb_hist<<<chunks, 512, 0, st>>>(d_key[(q + 1) & 1], d_n, shift, digit_bits[q], d_hist);
        SCAN(d_hist, d_first, nhist);
        auto f = first ? (last ? kb_radix<true, true> : kb_radix<true, false>)
                       : (last ? kb_radix<false, true> : kb_radix<false, false>);
        f<<<chunks, RADIX_THREADS, 0, st>>>(b2p, ix->d_b3, T, chunk, k, d_key[(q + 1) & 1], d_n, shift, digit_bits[q],
                                            d_first, d_key[q & 1], ix->d_pos, ix->d_ls);
        CUC(cudaGetLastError());
    }
    uint32_t S = 0;
    CUC(cudaMemcpyAsync(&S, d_n, 4, cudaMemcpyDeviceToHost, st));
    CUC(cudaStreamSynchronize(st));
    ix->n_seeds = S;
    CUC(cudaMemsetAsync(ix->d_pos + S, 0, 8 * 4, st));
    CUC(cudaMemsetAsync(ix->d_ls + S, 0, 8 * 2, st));
    CUC(cudaStreamSynchronize(st));
    cudaFree(d_tmp);
    *out = ix;
    return SWM_OK;
#undef SCAN
#undef CUC
}

extern "C" int swm_index_build_device(const uint8_t *d_seq, uint64_t n, uint32_t k, int device, swm_index **out) {
    if (!out || (!d_seq && n)) return SWM_ERR_ARG;
    return build_on_device(d_seq, n, k, device, out);
}

extern "C" int swm_index_build(const uint8_t *seq, uint64_t n, uint32_t k, int device, swm_index **out) {
    if (!out || (!seq && n)) return SWM_ERR_ARG;
    SWM_CUDA(cudaSetDevice(device));
    uint8_t *d_seq = nullptr;
    if (n) {
        cudaError_t e = cudaMalloc(&d_seq, n);
        if (e != cudaSuccess) {
            swm_set_error("cudaMalloc(sequence %llu): %s", (unsigned long long)n, cudaGetErrorString(e));
            return SWM_ERR_OOM;
        }
        e = cudaMemcpy(d_seq, seq, n, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(d_seq);
            swm_set_error("H2D sequence: %s", cudaGetErrorString(e));
            return SWM_ERR_CUDA;
        }
    }
    int rc = build_on_device(d_seq, n, k, device, out);
    cudaFree(d_seq);
    return rc;
}

extern "C" int swm_index_get_info(const swm_index *ix, swm_index_info *info) {
    if (!ix || !info) return SWM_ERR_ARG;
    info->k = ix->k;
    info->n = ix->n;
    info->n_seeds = ix->n_seeds;
    info->n_words2 = ix->n_words2;
    info->n_words3 = ix->n_words3;
    info->ref_length = ix->ref_length;
    info->device = ix->device;
    return SWM_OK;
}

extern "C" int swm_index_download(const swm_index *ix, uint32_t *hash_count, uint32_t *hash_offset_end,
                                  uint32_t *positions, uint16_t *pos_lseeds, uint32_t *base_2bits,
                                  uint32_t *base_3bits) {
    if (!ix) return SWM_ERR_ARG;
    SWM_CUDA(cudaSetDevice(ix->device));
    const uint64_t nb = 1ull << (2 * ix->k);
    if (hash_count) SWM_CUDA(cudaMemcpy(hash_count, ix->d_count, nb * 4, cudaMemcpyDeviceToHost));
    if (hash_offset_end) {
        // the reference's file holds the scatter cursors: start[i + 1] for
        // bucket i, and the total once more at [4^k] (serial_index.c:337-352)
        SWM_CUDA(cudaMemcpy(hash_offset_end, ix->d_off + 1, nb * 4, cudaMemcpyDeviceToHost));
        hash_offset_end[nb] = (uint32_t)ix->n_seeds;
    }
    if (positions && ix->n_seeds)
        SWM_CUDA(cudaMemcpy(positions, ix->d_pos, ix->n_seeds * 4, cudaMemcpyDeviceToHost));
    if (pos_lseeds && ix->n_seeds)
        SWM_CUDA(cudaMemcpy(pos_lseeds, ix->d_ls, ix->n_seeds * 2, cudaMemcpyDeviceToHost));
    if (base_2bits && ix->n_words2)
        SWM_CUDA(cudaMemcpy(base_2bits, ix->d_b2, ix->n_words2 * 4, cudaMemcpyDeviceToHost));
    if (base_3bits && ix->n_words3)
        SWM_CUDA(cudaMemcpy(base_3bits, ix->d_b3, ix->n_words3 * 4, cudaMemcpyDeviceToHost));
    return SWM_OK;
}

extern "C" int swm_index_save(const swm_index *ix, const char *prefix, const char *ref_info, size_t ref_info_len) {
    if (!ix || !prefix) return SWM_ERR_ARG;
    const uint64_t nb = 1ull << (2 * ix->k);
    std::vector<uint32_t> cnt(nb), off(nb + 1), pos(ix->n_seeds), b2(ix->n_words2), b3(ix->n_words3);
    std::vector<uint16_t> ls(ix->n_seeds);
    int rc = swm_index_download(ix, cnt.data(), off.data(), pos.data(), ls.data(), b2.data(), b3.data());
    if (rc) return rc;
    if (swmf_write(prefix, ".ref_info", ref_info ? ref_info : "", ref_info ? ref_info_len : 0) ||
        swmf_write(prefix, ".hash_count", cnt.data(), nb * 4) ||
        swmf_write(prefix, ".hash_offset", off.data(), (nb + 1) * 4) ||
        swmf_write(prefix, ".positions", pos.data(), ix->n_seeds * 4) ||
        swmf_write(prefix, ".pos_lseeds", ls.data(), ix->n_seeds * 2) ||
        swmf_write(prefix, ".base_2bits", b2.data(), ix->n_words2 * 4) ||
        swmf_write(prefix, ".base_3bits", b3.data(), ix->n_words3 * 4)) {
        swm_set_error("cannot write index files under %s", prefix);
        return SWM_ERR_IO;
    }
    return SWM_OK;
}

extern "C" int swm_index_build_fasta(const char *fasta_path, const char *prefix, uint32_t k, int device) {
    if (!fasta_path || !prefix) return SWM_ERR_ARG;
    uint8_t *seq = nullptr;
    uint64_t n = 0;
    char *info = nullptr;
    size_t info_len = 0;
    int rc = swmf_read_fasta(fasta_path, &seq, &n, &info, &info_len);
    if (rc) {
        swm_set_error("cannot read FASTA %s", fasta_path);
        return rc == -3 ? SWM_ERR_OOM : SWM_ERR_IO;
    }
    swm_index *ix = nullptr;
    rc = swm_index_build(seq, n, k, device, &ix);
    free(seq);
    if (rc == SWM_OK) {
        rc = swm_index_save(ix, prefix, info, info_len);
        swm_index_free(ix);
    }
    free(info);
    return rc;
}

// ------------------------------------------------------------ index load
//
// load_ref_info (mapper_mpe.c:198-314) freads each file whole into malloc'ed
// memory before the mapper uses it. Here each file streams into device
// memory: one host thread per file reads 32 MiB chunks with pread into two
// page-locked buffers in turn while the previous chunk's copy runs on the
// thread's own stream, so disk (or page cache) reads overlap the H2D copies
// and the five files load concurrently.

#define LOAD_CHUNK (32ull << 20)

static std::string index_path(const char *prefix, const char *ext) { return std::string(prefix) + ext; }

// Size of a regular file, or -1 when it cannot be stat'ed.
static int64_t file_bytes(const std::string &path) {
    struct stat sb;
    if (stat(path.c_str(), &sb) != 0 || !S_ISREG(sb.st_mode)) return -1;
    return (int64_t)sb.st_size;
}

struct FileLoad {
    std::string path;
    uint64_t bytes;
    void *d_dst;
    bool sum_words; // add up the file's u32 words (the bucket counts)
    uint64_t sum;
    int rc;
    char err[256];
};

static void load_file(FileLoad *L, int device) {
    L->rc = SWM_OK;
    L->sum = 0;
    if (cudaSetDevice(device) != cudaSuccess) {
        snprintf(L->err, sizeof L->err, "cudaSetDevice(%d) failed", device);
        L->rc = SWM_ERR_CUDA;
        return;
    }
    const int fd = open(L->path.c_str(), O_RDONLY);
    if (fd < 0) {
        snprintf(L->err, sizeof L->err, "cannot open %s", L->path.c_str());
        L->rc = SWM_ERR_IO;
        return;
    }
#ifdef POSIX_FADV_SEQUENTIAL
    posix_fadvise(fd, 0, 0, POSIX_FADV_SEQUENTIAL);
#endif
    cudaStream_t st = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    uint8_t *buf[2] = {nullptr, nullptr};
    const uint64_t chunk = L->bytes < LOAD_CHUNK ? (L->bytes ? L->bytes : 1) : LOAD_CHUNK;
    bool ok = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess;
    for (int i = 0; i < 2 && ok; i++)
        ok = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming) == cudaSuccess &&
             cudaHostAlloc((void **)&buf[i], chunk, 0) == cudaSuccess;
    if (!ok) {
        snprintf(L->err, sizeof L->err, "staging buffers for %s", L->path.c_str());
        L->rc = SWM_ERR_OOM;
    }
    bool used[2] = {false, false};
    for (uint64_t off = 0, i = 0; L->rc == SWM_OK && off < L->bytes; i ^= 1) {
        const uint64_t len = L->bytes - off < chunk ? L->bytes - off : chunk;
        if (used[i] && cudaEventSynchronize(ev[i]) != cudaSuccess) { // buffer i's last copy is done
            snprintf(L->err, sizeof L->err, "H2D of %s failed", L->path.c_str());
            L->rc = SWM_ERR_CUDA;
            break;
        }
        uint64_t got = 0;
        while (got < len) {
            const ssize_t r = pread(fd, buf[i] + got, len - got, (off_t)(off + got));
            if (r < 0 && errno == EINTR) continue;
            if (r <= 0) break;
            got += (uint64_t)r;
        }
        if (got != len) {
            snprintf(L->err, sizeof L->err, "%s is shorter than its %llu bytes", L->path.c_str(),
                     (unsigned long long)L->bytes);
            L->rc = SWM_ERR_IO;
            break;
        }
        if (L->sum_words) {
            const uint32_t *w = (const uint32_t *)buf[i];
            for (uint64_t j = 0; j < len / 4; j++) L->sum += w[j];
        }
        if (cudaMemcpyAsync((uint8_t *)L->d_dst + off, buf[i], len, cudaMemcpyHostToDevice, st) != cudaSuccess ||
            cudaEventRecord(ev[i], st) != cudaSuccess) {
            snprintf(L->err, sizeof L->err, "H2D of %s failed", L->path.c_str());
            L->rc = SWM_ERR_CUDA;
            break;
        }
        used[i] = true;
        off += len;
    }
    if (st && cudaStreamSynchronize(st) != cudaSuccess && L->rc == SWM_OK) {
        snprintf(L->err, sizeof L->err, "H2D of %s failed", L->path.c_str());
        L->rc = SWM_ERR_CUDA;
    }
    for (int i = 0; i < 2; i++) {
        if (buf[i]) cudaFreeHost(buf[i]);
        if (ev[i]) cudaEventDestroy(ev[i]);
    }
    if (st) cudaStreamDestroy(st);
    close(fd);
}

extern "C" int swm_index_open(const char *prefix, uint32_t k, int device, swm_index **out) {
    if (!prefix || !out || k < 1 || k > 14) {
        swm_set_error("swm_index_open: null argument or k outside [1, 14]");
        return SWM_ERR_ARG;
    }
    // every file present and the sizes consistent before any device work
    static const char *exts[5] = {".hash_count", ".positions", ".pos_lseeds", ".base_2bits", ".base_3bits"};
    int64_t sz[5];
    for (int f = 0; f < 5; f++) {
        sz[f] = file_bytes(index_path(prefix, exts[f]));
        if (sz[f] < 0) {
            swm_set_error("index file %s is missing", index_path(prefix, exts[f]).c_str());
            return SWM_ERR_IO;
        }
    }
    const uint64_t nb = 1ull << (2 * k);
    const uint64_t S = (uint64_t)sz[1] / 4;
    if ((uint64_t)sz[0] != nb * 4 || sz[1] % 4 || (uint64_t)sz[2] != S * 2 || sz[3] % 8 || sz[3] != 2 * sz[4] ||
        S >= 0xffffffffull) {
        swm_set_error("index files under %s have inconsistent sizes for k=%u (hash_count %lld, positions %lld, "
                      "pos_lseeds %lld, base_2bits %lld, base_3bits %lld bytes)",
                      prefix, k, (long long)sz[0], (long long)sz[1], (long long)sz[2], (long long)sz[3],
                      (long long)sz[4]);
        return SWM_ERR_IO;
    }
    SWM_CUDA(cudaSetDevice(device));
    swm_index *ix = (swm_index *)calloc(1, sizeof(swm_index));
    if (!ix) return SWM_ERR_OOM;
    ix->device = device;
    ix->k = k;
    ix->n_seeds = S;
    ix->n_words2 = (uint64_t)sz[3] / 4;
    ix->n_words3 = (uint64_t)sz[4] / 4;
    ix->ref_length = (uint64_t)sz[3] * 16; // mapper_mpe.c:288
    ix->n = 32 * ix->n_words3;
    void *info = nullptr;
    size_t ninfo = 0;
    if (swmf_read(prefix, ".ref_info", &info, &ninfo) == 0) {
        const uint64_t t = swmf_ref_info_total((const char *)info, ninfo);
        if (t) ix->n = t;
        free(info);
    }
    uint32_t *d_tmp = nullptr;
    int rc = SWM_OK;
    if (dalloc(&ix->d_count, nb) || dalloc(&ix->d_off, nb + 1) || dalloc(&ix->d_pos, S + 8) ||
        dalloc(&ix->d_ls, S + 8) || dalloc(&ix->d_b2, ix->n_words2 + SWM_PAD_WORDS) ||
        dalloc(&ix->d_b3, ix->n_words3 + SWM_PAD_WORDS) || dalloc(&d_tmp, swm_scan_tmp_words(nb))) {
        rc = SWM_ERR_OOM;
    }
    if (rc == SWM_OK) {
        FileLoad loads[5];
        void *dst[5] = {ix->d_count, ix->d_pos, ix->d_ls, ix->d_b2, ix->d_b3};
        for (int f = 0; f < 5; f++) {
            loads[f].path = index_path(prefix, exts[f]);
            loads[f].bytes = (uint64_t)sz[f];
            loads[f].d_dst = dst[f];
            loads[f].sum_words = f == 0;
            loads[f].err[0] = 0;
        }
        std::vector<std::thread> th;
        for (int f = 1; f < 5; f++) th.emplace_back(load_file, &loads[f], device);
        load_file(&loads[0], device);
        for (auto &t : th) t.join();
        for (int f = 0; f < 5 && rc == SWM_OK; f++)
            if (loads[f].rc != SWM_OK) {
                swm_set_error("%s", loads[f].err);
                rc = loads[f].rc;
            }
        if (rc == SWM_OK && loads[0].sum != S) {
            swm_set_error("index files under %s are inconsistent: hash_count adds up to %llu, positions hold %llu",
                          prefix, (unsigned long long)loads[0].sum, (unsigned long long)S);
            rc = SWM_ERR_IO;
        }
    }
    if (rc == SWM_OK) {
        if (cudaMemset(ix->d_pos + S, 0, 32) != cudaSuccess || cudaMemset(ix->d_ls + S, 0, 16) != cudaSuccess ||
            cudaMemset(ix->d_b2 + ix->n_words2, 0, SWM_PAD_WORDS * 4) != cudaSuccess ||
            cudaMemset(ix->d_b3 + ix->n_words3, 0, SWM_PAD_WORDS * 4) != cudaSuccess) {
            swm_set_error("clearing the index padding under %s failed", prefix);
            rc = SWM_ERR_CUDA;
        }
    }
    if (rc == SWM_OK) {
        // hash_offset rebuilt from the counts (mapper_mpe.c:250-255)
        rc = swm_exclusive_scan(ix->d_count, ix->d_off, nullptr, nb, nb, d_tmp, nullptr, 0);
        if (rc == SWM_OK && cudaDeviceSynchronize() != cudaSuccess) {
            swm_set_error("rebuilding hash_offset under %s failed", prefix);
            rc = SWM_ERR_CUDA;
        }
    }
    cudaFree(d_tmp);
    if (rc != SWM_OK) {
        index_release(ix);
        return rc;
    }
    *out = ix;
    return SWM_OK;
}

extern "C" void swm_index_free(swm_index *ix) {
    if (!ix) return;
    cudaSetDevice(ix->device);
    index_release(ix);
}

static std::mutex g_ctab_mu;

// Device bytes of the candidate table of ix.
static uint64_t ctab_bytes(const swm_index *ix) { return (SWM_CTAB_KEYS + 1) * 4 + (4 * ix->n_seeds + 8) * 4; }

// Build the candidate table when it is missing, k is 12, the caller has not
// dropped it, and the device holds it with a margin (8 GiB) to spare. Not
// building it is not an error: the mapper then filters the buckets entry by
// entry. Returns SWM_OK in both cases; a CUDA error while building is returned.
int swm_ctab_build(swm_index *ix, int forced) {
    std::lock_guard<std::mutex> lk(g_ctab_mu);
    if (ix->d_ctab_off || ix->ctab_off || ix->k != 12 || 4 * ix->n_seeds + 8 >= 0xffffffffull) return SWM_OK;
    // Built on its own only for genomes whose buckets average SWM_CTAB_MIN_MEAN
    // entries or more: its lookup is a random read of a 17 GiB array per
    // selected long seed, which costs more than filtering buckets of a few entries
    // (a 100 Mbp genome averages 1.5 per bucket, a 3.1 Gbp one 44).
    if (!forced && ix->n_seeds < (uint64_t)SWM_CTAB_MIN_MEAN << (2 * ix->k)) return SWM_OK;
    SWM_CUDA(cudaSetDevice(ix->device));
    size_t fr = 0, total = 0;
    if (cudaMemGetInfo(&fr, &total) != cudaSuccess || fr < ctab_bytes(ix) + (8ull << 30)) {
        cudaGetLastError();
        return SWM_OK;
    }
    uint32_t *d_o = nullptr, *d_p = nullptr;
    if (cudaMalloc(&d_o, (SWM_CTAB_KEYS + 1) * 4) != cudaSuccess ||
        cudaMalloc(&d_p, (4 * ix->n_seeds + 8) * 4) != cudaSuccess) {
        cudaFree(d_o);
        cudaGetLastError();
        return SWM_OK;
    }
    const uint32_t last = (uint32_t)(4 * ix->n_seeds);
    uint32_t *d_t = nullptr; // the partitions' sums and starts
    cudaError_t e = cudaMalloc(&d_t, (2ull * CTAB_CORES + 64 + swm_scan_tmp_words(CTAB_CORES)) * 4);
    if (e == cudaSuccess) e = cudaMemcpy(d_o + SWM_CTAB_KEYS, &last, 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(d_p + 4 * ix->n_seeds, 0, 32);
    if (e == cudaSuccess) {
        uint32_t *d_sums = d_t, *d_base = d_t + CTAB_CORES, *d_scan = d_base + CTAB_CORES + 64;
        const size_t smem = (CTAB_KEYS_CORE + 2 * CTAB_BUCKETS_CORE) * 4;
        kb_ctab_sums<<<CTAB_CORES / 8, 256>>>(ix->d_count, d_sums);
        if (swm_exclusive_scan(d_sums, d_base, nullptr, CTAB_CORES, CTAB_CORES, d_scan, nullptr, 0) == SWM_OK &&
            cudaFuncSetAttribute(kb_ctab, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess)
            kb_ctab<<<sm_count(ix->device) * 3, CTAB_THREADS, smem>>>(ix->d_off, ix->d_pos, ix->d_ls, d_base, d_o, d_p);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    cudaFree(d_t);
    if (e != cudaSuccess) {
        cudaFree(d_o);
        cudaFree(d_p);
        swm_set_error("building the candidate table: %s", cudaGetErrorString(e));
        return SWM_ERR_CUDA;
    }
    ix->d_ctab_off = d_o;
    ix->d_ctab_pos = d_p;
    ix->ctab_gen++;
    return SWM_OK;
}

int swm_keys32_build(swm_index *ix) {
    std::lock_guard<std::mutex> lk(g_ctab_mu);
    if (ix->d_keys32 || ix->n_seeds < (uint64_t)SWM_CTAB_MIN_MEAN << (2 * ix->k)) return SWM_OK;
    SWM_CUDA(cudaSetDevice(ix->device));
    uint32_t *d = nullptr;
    if (cudaMalloc(&d, (ix->n_seeds / SWM_PER_FETCH + 1) * 4) != cudaSuccess) {
        cudaGetLastError();
        return SWM_OK;
    }
    const uint64_t nb = 1ull << (2 * ix->k);
    kb_keys32<<<grid_for(nb, 256, ix->device, 8), 256>>>(ix->d_off, nb, ix->d_pos, d);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        cudaFree(d);
        swm_set_error("building the refill keys: %s", cudaGetErrorString(e));
        return SWM_ERR_CUDA;
    }
    ix->d_keys32 = d;
    return SWM_OK;
}

extern "C" int swm_index_candidate_table(swm_index *ix, int enable, uint64_t *bytes) {
    if (!ix) return SWM_ERR_ARG;
    if (enable < 0) { // query only
        std::lock_guard<std::mutex> lk(g_ctab_mu);
        if (bytes) *bytes = ix->d_ctab_off ? ctab_bytes(ix) : 0;
        return SWM_OK;
    }
    if (enable) {
        {
            std::lock_guard<std::mutex> lk(g_ctab_mu);
            ix->ctab_off = 0;
        }
        const int rc = swm_ctab_build(ix, 1);
        if (rc) return rc;
    } else {
        std::lock_guard<std::mutex> lk(g_ctab_mu);
        ix->ctab_off = 1;
        if (ix->d_ctab_off) {
            SWM_CUDA(cudaSetDevice(ix->device));
            cudaDeviceSynchronize(); // no block may still read the table
            cudaFree(ix->d_ctab_off);
            cudaFree(ix->d_ctab_pos);
            ix->d_ctab_off = ix->d_ctab_pos = nullptr;
            ix->ctab_gen++;
        }
    }
    if (bytes) *bytes = ix->d_ctab_off ? ctab_bytes(ix) : 0;
    return SWM_OK;
}

// ------------------------------------------------ allocation-free offsets

// Scratch of swm_hash_offset_noalloc: the scan's block partial sums, one word
// per 2048 counts, so 32768 words cover 4^13 buckets (k <= 13). Every device
// that loads this library holds these 128 KB until the process exits.
#define NOALLOC_PARTIALS 32768
static __device__ __align__(256) uint32_t g_noalloc_partials[NOALLOC_PARTIALS + 64];

#define NOALLOC_MAX_DEVICES 64
static std::mutex g_noalloc_mu;
static uint32_t *g_noalloc_addr[NOALLOC_MAX_DEVICES]; // device address of the array, per device

// For callers that must not allocate device memory: the caller owns both
// arrays, and the scan's partial sums go to the static array above instead of
// a cudaMalloc'ed buffer. Its first call on a device looks up the array's
// device address (cudaGetSymbolAddress) with that device current; make that
// first call before any stream capture. The address is cached for the life of
// the process: a cudaDeviceReset of the primary context would leave it stale,
// so resetting a device the library uses is not supported.
extern "C" int swm_hash_offset_noalloc(const uint32_t *d_hash_count, uint32_t *d_hash_offset, uint32_t k,
                                       void *stream) {
    if (!d_hash_count || !d_hash_offset || k < 1 || k > 16) {
        swm_set_error("swm_hash_offset_noalloc: null array or k out of range (k=%u)", k);
        return SWM_ERR_ARG;
    }
    const uint64_t n = 1ull << (2 * k);
    const uint64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (nb > NOALLOC_PARTIALS) {
        swm_set_error("swm_hash_offset_noalloc: k=%u needs %llu partial sums, the static scratch holds %d (k <= 13)",
                      k, (unsigned long long)nb, NOALLOC_PARTIALS);
        return SWM_ERR_ARG;
    }
    int dev = 0;
    SWM_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
        swm_set_error("swm_hash_offset_noalloc: device %d beyond the %d supported", dev, NOALLOC_MAX_DEVICES);
        return SWM_ERR_ARG;
    }
    uint32_t *scratch;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_addr[dev]) {
            void *addr = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&addr, g_noalloc_partials);
            if (e != cudaSuccess || !addr) {
                swm_set_error("swm_hash_offset_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
                return SWM_ERR_CUDA;
            }
            g_noalloc_addr[dev] = (uint32_t *)addr;
        }
        scratch = g_noalloc_addr[dev];
    }
    // every partial the scan reads is written earlier in the same call, so
    // nothing in the scratch has to be cleared between calls
    return swm_exclusive_scan(d_hash_count, d_hash_offset, nullptr, n, n, scratch, nullptr, (cudaStream_t)stream);
}
