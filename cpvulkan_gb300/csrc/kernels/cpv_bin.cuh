/*
 * cpv_bin.cuh — order-preserving sort-middle binning and the other generic
 * device kernels (scan, fills).
 *
 * The per-draw binning builds, for every bin (a square of screen tiles, at
 * most CPV_MAX_BINS on the target), the list of primitive ids that touch it,
 * in API order — the per-pixel order the reference's serial loop
 * (CPVulkan/CommandBuffer.Draw.cpp:1526-1593) produces. The raster CTA of a
 * tile filters its bin's list by the entries' tile rectangles, in order.
 * Primitives are split into rows of row_prims consecutive ones:
 *
 *   1. cpv_setup_rects (the pipeline's module) writes every primitive's tile
 *      rectangle and each row's count of primitives per bin;
 *   2. cpv_bin_scan turns the counts, column by column, into the position of
 *      each (row, bin)'s first entry and stores every bin's list range;
 *   3. cpv_bin_write: one CTA per row writes the ids and the rectangles
 *      within the bin at those positions, in primitive order.
 *
 * Every launch has a shape the host knows and no value is carried from one
 * draw to the next, so the sequence needs no memset and can be captured in a
 * CUDA graph. The list has a fixed capacity; a draw that would exceed it
 * writes none and the raster filters the rectangles of all primitives
 * (slower, same result).
 *
 * Bins instead of tiles: a (tile x span) count matrix with one warp per span
 * of 256 primitives is bound by its serial chain (a warp places 32
 * (primitive, tile) pairs per dependent global step) for large primitives
 * and by the matrix's size on large targets. Binning + raster on GB300, per
 * tile then per bin: 300 triangles at 1280x720, 4800 + 526 us then 8 + 527
 * (filtered); 12k quad triangles at 1280x720, 300 + 572 then 25 + 577; 400k at
 * 1920x1080, 523 + 2385 then 68 + 2304; 500k small ones at 2048x2048, 173 + 315
 * then 47 + 263. A bin's list is several times shorter than its tiles'
 * lists together, and the filter reads 4 bytes per entry from L2.
 */
#ifndef CPV_BIN_CUH
#define CPV_BIN_CUH

#include "cpv_device.cuh"

/* 2. counts[row][bin] → the list position of the row's first entry in the
 * bin; range[bin] = the bin's list. One CTA of 1024 threads per 8 bins: 128
 * groups of rows are summed, scanned over the groups and walked again. A
 * bin's list starts where an atomic on *total puts it (the lists' order in
 * memory does not matter); *total (zeroed by cpv_setup_rects) ends as the
 * draw's pair count. */
#define CPV_BIN_SCAN_THREADS 1024
#define CPV_BIN_SCAN_BINS 8
extern "C" __global__ void __launch_bounds__(CPV_BIN_SCAN_THREADS) cpv_bin_scan(uint32_t* __restrict__ counts, uint32_t rows, uint32_t bins,
                                                                               uint2* __restrict__ range, unsigned long long* __restrict__ total) {
    __shared__ uint32_t warp_sums[CPV_BIN_SCAN_THREADS / 32][CPV_BIN_SCAN_BINS];
    __shared__ uint32_t list_base[CPV_BIN_SCAN_BINS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t b = threadIdx.x % CPV_BIN_SCAN_BINS, group = threadIdx.x / CPV_BIN_SCAN_BINS;
    const uint32_t bin = blockIdx.x * CPV_BIN_SCAN_BINS + b;
    const uint32_t groups = CPV_BIN_SCAN_THREADS / CPV_BIN_SCAN_BINS;
    const uint32_t per = (rows + groups - 1u) / groups;
    const uint32_t r0 = per * group < rows ? per * group : rows;
    const uint32_t r1 = bin < bins ? (r0 + per < rows ? r0 + per : rows) : r0;
    uint32_t* column = counts + bin;
    uint32_t sum = 0u;
#pragma unroll 8
    for (uint32_t r = r0; r < r1; r++) sum += column[static_cast<uint64_t>(r) * bins];
    uint32_t incl = sum;
#pragma unroll
    for (uint32_t o = CPV_BIN_SCAN_BINS; o < 32u; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane >= 32u - CPV_BIN_SCAN_BINS) warp_sums[warp][b] = incl;
    __syncthreads();
    if (warp < CPV_BIN_SCAN_BINS) {  /* warp k scans bin k over the 32 warps */
        const uint32_t v = warp_sums[lane][warp];
        uint32_t s = v;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= o) s += t;
        }
        warp_sums[lane][warp] = s - v;
        const uint32_t k = blockIdx.x * CPV_BIN_SCAN_BINS + warp;
        if (lane == 31u && k < bins) {
            const uint32_t base = s ? static_cast<uint32_t>(atomicAdd(total, static_cast<unsigned long long>(s))) : 0u;
            list_base[warp] = base;
            range[k] = make_uint2(base, base + s);
        }
    }
    __syncthreads();
    if (r1 <= r0) return;
    uint32_t run = list_base[b] + warp_sums[warp][b] + incl - sum;
#pragma unroll 8
    for (uint32_t r = r0; r < r1; r++) {
        const uint32_t c = column[static_cast<uint64_t>(r) * bins];
        column[static_cast<uint64_t>(r) * bins] = run;
        run += c;
    }
}

/* 3. One CTA per row, 256 primitives at a time: each warp counts its 32
 * primitives per bin, the counts are scanned over the CTA's 8 warps onto the
 * row's running positions, and each warp then places its (primitive, bin)
 * pairs 32 at a time in primitive order (a match-any rank within the step,
 * the warp's own position per bin between steps, all in shared memory).
 * Dynamic shared memory: 9 words per bin. */
extern "C" __global__ void __launch_bounds__(256) cpv_bin_write(const uint2* __restrict__ rects, uint64_t prims, uint32_t row_prims, uint32_t shift,
                                                                uint32_t bins_x, uint32_t bins, const uint32_t* __restrict__ offsets,
                                                                uint32_t* __restrict__ list, uint32_t* __restrict__ list_rects, uint32_t capacity,
                                                                const unsigned long long* __restrict__ total) {
    extern __shared__ uint32_t cpv_bin_smem[];
    if (*total > capacity) return;
    uint32_t* next = cpv_bin_smem;  /* [bin]: the row's next position */
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t* mine = cpv_bin_smem + (1u + warp) * bins;  /* [bin]: this warp's count, then its next position */
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint64_t begin = static_cast<uint64_t>(blockIdx.x) * row_prims;
    const uint64_t end = begin + row_prims < prims ? begin + row_prims : prims;
    for (uint32_t i = threadIdx.x; i < bins; i += 256u) next[i] = offsets[static_cast<uint64_t>(blockIdx.x) * bins + i];
    for (uint64_t base = begin; base < end; base += 256u) {
        for (uint32_t i = lane; i < bins; i += 32u) mine[i] = 0u;
        __syncwarp();
        const uint64_t g = base + threadIdx.x;
        uint2 r = make_uint2(0u, 0u);
        if (g < end) r = rects[g];
        const uint32_t x0 = r.x & 0xFFFFu, y0 = r.x >> 16, x1 = r.y & 0xFFFFu, y1 = r.y >> 16;
        const bool any = x1 > x0 && y1 > y0;
        const uint32_t bx0 = x0 >> shift, by0 = y0 >> shift;
        const uint32_t bw = any ? ((x1 - 1u) >> shift) + 1u - bx0 : 0u, bh = any ? ((y1 - 1u) >> shift) + 1u - by0 : 0u;
        for (uint32_t y = 0; y < bh; y++)
            for (uint32_t x = 0; x < bw; x++) atomicAdd(&mine[(by0 + y) * bins_x + bx0 + x], 1u);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < bins; i += 256u) {
            uint32_t run = next[i];
#pragma unroll
            for (uint32_t w = 0; w < 8u; w++) {
                uint32_t* c = &cpv_bin_smem[(1u + w) * bins + i];
                const uint32_t n = *c;
                *c = run;
                run += n;
            }
            next[i] = run;
        }
        __syncthreads();
        /* inclusive warp scan of the pair counts */
        const uint32_t n = bw * bh;
        uint32_t incl = n;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += v;
        }
        const uint32_t pairs = __shfl_sync(0xFFFFFFFFu, incl, 31);
        const uint32_t excl = incl - n;
        for (uint32_t p0 = 0; p0 < pairs; p0 += 32u) {
            const uint32_t p = p0 + lane;
            const bool valid = p < pairs;
            /* owner lane: the last lane whose exclusive start is <= p (lanes
             * without pairs share the next lane's start and are skipped) */
            uint32_t owner = 0;
#pragma unroll
            for (uint32_t step = 16u; step >= 1u; step >>= 1) {
                const uint32_t cand = owner + step;
                if (__shfl_sync(0xFFFFFFFFu, excl, cand) <= p) owner = cand;
            }
            const uint32_t local = p - __shfl_sync(0xFFFFFFFFu, excl, owner);
            const uint32_t o_x = __shfl_sync(0xFFFFFFFFu, r.x, owner), o_y = __shfl_sync(0xFFFFFFFFu, r.y, owner);
            const uint32_t o_w = __shfl_sync(0xFFFFFFFFu, bw, owner);
            uint32_t bin = 0xFFFFFFFFu, bx = 0u, by = 0u;
            if (valid) {
                const uint32_t row = local / o_w;
                bx = ((o_x & 0xFFFFu) >> shift) + local - row * o_w;
                by = (o_x >> (16u + shift)) + row;
                bin = by * bins_x + bx;
            }
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, valid ? bin : (0x80000000u | lane));
            const uint32_t rank = __popc(peers & lt_mask);
            uint32_t first = 0u;
            if (valid) first = mine[bin];
            __syncwarp();
            if (valid) {
                if (rank == 0u) mine[bin] = first + __popc(peers);
                const uint32_t pos = first + rank;
                if (pos < capacity) {  /* always, unless the pair total wrapped */
                    /* the rectangle within the bin, in tiles */
                    const uint32_t side = 1u << shift, tx = bx << shift, ty = by << shift;
                    const uint32_t rx0 = o_x & 0xFFFFu, ry0 = o_x >> 16, rx1 = o_y & 0xFFFFu, ry1 = o_y >> 16;
                    const uint32_t lx0 = rx0 > tx ? rx0 - tx : 0u, ly0 = ry0 > ty ? ry0 - ty : 0u;
                    const uint32_t lx1 = rx1 - tx < side ? rx1 - tx : side, ly1 = ry1 - ty < side ? ry1 - ty : side;
                    list[pos] = static_cast<uint32_t>(base + (threadIdx.x & ~31u) + owner);
                    list_rects[pos] = lx0 | (ly0 << 8) | (lx1 << 16) | (ly1 << 24);
                }
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

/* ---- exclusive scan of u32 (three-level, 2048 elements per block) ---- */

#define CPV_SCAN_THREADS 256
#define CPV_SCAN_ITEMS 8
#define CPV_SCAN_BLOCK (CPV_SCAN_THREADS * CPV_SCAN_ITEMS)

__device__ __forceinline__ uint32_t cpv_block_exclusive_scan(uint32_t v, uint32_t& block_total) {
    __shared__ uint32_t warp_sums[CPV_SCAN_THREADS / 32];
    __shared__ uint32_t total_sh;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= static_cast<uint32_t>(o)) incl += t;
    }
    if (lane == 31u) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0u) {
        const uint32_t s = lane < CPV_SCAN_THREADS / 32 ? warp_sums[lane] : 0u;
        uint32_t si = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, si, o);
            if (lane >= static_cast<uint32_t>(o)) si += t;
        }
        if (lane < CPV_SCAN_THREADS / 32) warp_sums[lane] = si - s;
        if (lane == CPV_SCAN_THREADS / 32 - 1) total_sh = si;
    }
    __syncthreads();
    const uint32_t r = warp_sums[warp] + incl - v;
    block_total = total_sh;
    __syncthreads();
    return r;
}

/* Level scan: out[i] = exclusive prefix within the block; block_sums[b] = block total. */
extern "C" __global__ void __launch_bounds__(CPV_SCAN_THREADS) cpv_scan_blocks(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                                              uint64_t n, uint32_t* __restrict__ block_sums) {
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * CPV_SCAN_BLOCK + static_cast<uint64_t>(threadIdx.x) * CPV_SCAN_ITEMS;
    uint32_t v[CPV_SCAN_ITEMS];
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < CPV_SCAN_ITEMS; i++) {
        v[i] = (base + i < n) ? in[base + i] : 0u;
        sum += v[i];
    }
    uint32_t total = 0;
    uint32_t run = cpv_block_exclusive_scan(sum, total);
#pragma unroll
    for (int i = 0; i < CPV_SCAN_ITEMS; i++) {
        if (base + i < n) out[base + i] = run;
        run += v[i];
    }
    if (threadIdx.x == 0 && block_sums) block_sums[blockIdx.x] = total;
}

/* out[i] += add[block(i)]; optionally writes the grand total. */
extern "C" __global__ void __launch_bounds__(CPV_SCAN_THREADS) cpv_scan_add(uint32_t* __restrict__ out, uint64_t n, const uint32_t* __restrict__ add) {
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * CPV_SCAN_BLOCK;
    const uint32_t a = add[blockIdx.x];
    for (uint32_t i = threadIdx.x; i < CPV_SCAN_BLOCK; i += CPV_SCAN_THREADS) {
        if (base + i < n) out[base + i] += a;
    }
}

/* total = last exclusive prefix + last input. */
extern "C" __global__ void cpv_scan_total(const uint32_t* __restrict__ in, const uint32_t* __restrict__ out, uint64_t n, uint32_t* __restrict__ total) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *total = n ? out[n - 1] + in[n - 1] : 0u;
}

/* ---- batched binning: pairs, stable radix sort by tile, tile ranges ----
 *
 * The batched path bins every draw of a render pass at once. Set-up writes
 * one tile rectangle per primitive and the pair count of each 256-primitive
 * block; after an exclusive scan of the block counts, cpv_batch_emit writes
 * the (tile, primitive) pairs in primitive order; a stable LSD radix sort by
 * tile (8-bit digits, one or two passes) groups them by tile while keeping
 * primitive (API) order inside each tile; cpv_tile_ranges records where each
 * tile's run starts and ends. Sizes that depend on the data (the pair count)
 * are read on the device, so the sequence has fixed launch shapes and can be
 * captured in a CUDA graph. Pairs beyond the capacity are not written; the
 * raster then scans the rectangles instead (same image). */

#define CPV_RADIX_THREADS 256
#define CPV_RADIX_DIGITS 256

__device__ __forceinline__ uint32_t cpv_pairs_in_bounds(const uint32_t* pair_total, uint32_t capacity) {
    const uint32_t p = *pair_total;
    return p <= capacity ? p : 0u;
}

/* Block-wide exclusive sum over 256 threads. */
__device__ __forceinline__ uint32_t cpv_block256_exclusive(uint32_t v, uint32_t* warp_sums /* [8] */) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= static_cast<uint32_t>(o)) incl += t;
    }
    if (lane == 31u) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t base = 0;
    for (uint32_t k = 0; k < warp; k++) base += warp_sums[k];
    return base + incl - v;
}

/* One block per 256-primitive set-up block: the block's pairs at
 * block_offsets[block] + (pairs of the block's earlier primitives). A block
 * without pairs has no rectangles written this frame and emits nothing. */
extern "C" __global__ void __launch_bounds__(256) cpv_batch_emit(const uint2* __restrict__ rects, const uint32_t* __restrict__ block_pairs,
                                                                 const uint32_t* __restrict__ block_offsets, uint32_t tiles_x,
                                                                 uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t capacity,
                                                                 const uint32_t* __restrict__ pair_total) {
    __shared__ uint32_t warp_sums[8];
    if (block_pairs[blockIdx.x] == 0u) return;
    const uint64_t g = static_cast<uint64_t>(blockIdx.x) * 256u + threadIdx.x;
    const uint2 r = rects[g];
    const uint32_t x0 = r.x & 0xFFFFu, y0 = r.x >> 16, x1 = r.y & 0xFFFFu, y1 = r.y >> 16;
    const uint32_t w = x1 - x0;
    const uint32_t n = w * (y1 - y0);
    const uint32_t excl = cpv_block256_exclusive(n, warp_sums);
    if (*pair_total > capacity) return;
    const uint32_t base = block_offsets[blockIdx.x] + excl;
    for (uint32_t k = 0; k < n; k++) {
        const uint64_t pos = static_cast<uint64_t>(base) + k;
        if (pos >= capacity) break;  /* only reachable if the pair total wrapped 32 bits */
        const uint32_t ty = y0 + k / w, tx = x0 + k % w;
        keys[pos] = ty * tiles_x + tx;
        vals[pos] = static_cast<uint32_t>(g);
    }
}

/* Vertex-stage sizing: one CTA per draw d with want[d] set finds the
 * smallest and largest index value the draw reads inside its bound index
 * buffer (indices outside the buffer read as 0 and are not counted; the
 * set-up shades any vertex outside the found range itself). Writes
 * range[d] = (min, max), or (0xFFFFFFFF, 0) when there is none. */
extern "C" __global__ void __launch_bounds__(256) cpv_index_range(const CpvDrawParams* __restrict__ draws, const uint8_t* __restrict__ want,
                                                                  uint2* __restrict__ range) {
    __shared__ uint32_t smin[8], smax[8];
    const uint32_t d = blockIdx.x;
    uint32_t lo = 0xFFFFFFFFu, hi = 0u;
    if (want[d]) {
        const CpvDrawParams& P = draws[d];
        const uint32_t size = P.index_size;
        for (uint32_t i = threadIdx.x; i < P.count; i += 256u) {
            const uint64_t off = (static_cast<uint64_t>(P.first) + i) * size;
            if (size == 0u || off + size > P.ib_bytes) continue;
            const uint32_t v = size == 2u ? static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(P.ib + off)))
                                          : __ldg(reinterpret_cast<const uint32_t*>(P.ib + off));
            lo = v < lo ? v : lo;
            hi = v > hi ? v : hi;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint32_t a = __shfl_xor_sync(0xFFFFFFFFu, lo, o), b = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
    }
    if ((threadIdx.x & 31u) == 0u) {
        smin[threadIdx.x >> 5] = lo;
        smax[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) {
            lo = smin[w] < lo ? smin[w] : lo;
            hi = smax[w] > hi ? smax[w] : hi;
        }
        range[d] = make_uint2(lo, hi);
    }
}

/* Contiguous item range of CTA c of `ctas` over n items. */
__device__ __forceinline__ void cpv_cta_range(uint32_t n, uint32_t c, uint32_t ctas, uint32_t& begin, uint32_t& end) {
    const uint32_t per = (n + ctas - 1u) / ctas;
    const uint64_t b = static_cast<uint64_t>(per) * c, e = b + per;
    begin = static_cast<uint32_t>(b < n ? b : n);
    end = static_cast<uint32_t>(e < n ? e : n);
}

/* hist[digit * gridDim.x + cta] = items of the CTA's range with that digit. */
extern "C" __global__ void __launch_bounds__(CPV_RADIX_THREADS) cpv_radix_hist(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ pair_total,
                                                                               uint32_t capacity, uint32_t shift, uint32_t* __restrict__ hist) {
    __shared__ uint32_t counts[CPV_RADIX_DIGITS];
    counts[threadIdx.x] = 0u;
    __syncthreads();
    uint32_t begin, end;
    cpv_cta_range(cpv_pairs_in_bounds(pair_total, capacity), blockIdx.x, gridDim.x, begin, end);
    for (uint32_t i = begin + threadIdx.x; i < end; i += CPV_RADIX_THREADS) atomicAdd(&counts[(keys[i] >> shift) & 0xFFu], 1u);
    __syncthreads();
    hist[threadIdx.x * gridDim.x + blockIdx.x] = counts[threadIdx.x];
}

/* Stable scatter: offsets = exclusive scan of hist (digit-major). Each CTA
 * walks its range in order, 256 items at a time; an item's position is its
 * digit's running offset plus the number of earlier items of the sub-chunk
 * with the same digit (earlier warps, then earlier lanes). */
extern "C" __global__ void __launch_bounds__(CPV_RADIX_THREADS) cpv_radix_scatter(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                                                                                  uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                                                                  const uint32_t* __restrict__ pair_total, uint32_t capacity, uint32_t shift,
                                                                                  const uint32_t* __restrict__ offsets) {
    __shared__ uint32_t running[CPV_RADIX_DIGITS];
    __shared__ uint32_t warp_count[CPV_RADIX_THREADS / 32][CPV_RADIX_DIGITS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    running[threadIdx.x] = offsets[threadIdx.x * gridDim.x + blockIdx.x];
    uint32_t begin, end;
    cpv_cta_range(cpv_pairs_in_bounds(pair_total, capacity), blockIdx.x, gridDim.x, begin, end);
    for (uint32_t base = begin; base < end; base += CPV_RADIX_THREADS) {
#pragma unroll
        for (uint32_t w = 0; w < CPV_RADIX_THREADS / 32; w++) warp_count[w][threadIdx.x] = 0u;
        __syncthreads();
        const uint32_t i = base + threadIdx.x;
        const bool valid = i < end;
        uint32_t key = 0, val = 0, digit = CPV_RADIX_DIGITS + lane;  /* invalid lanes never match a digit */
        if (valid) {
            key = keys_in[i];
            val = vals_in[i];
            digit = (key >> shift) & 0xFFu;
        }
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank == 0u) warp_count[warp][digit] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t pos = running[digit] + rank;
            for (uint32_t w = 0; w < warp; w++) pos += warp_count[w][digit];
            keys_out[pos] = key;
            vals_out[pos] = val;
        }
        __syncthreads();
        uint32_t add = 0;
#pragma unroll
        for (uint32_t w = 0; w < CPV_RADIX_THREADS / 32; w++) add += warp_count[w][threadIdx.x];
        running[threadIdx.x] += add;
        __syncthreads();
    }
}

/* tile_begin / tile_end (zeroed beforehand) from the sorted keys. */
extern "C" __global__ void __launch_bounds__(256) cpv_tile_ranges(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ pair_total,
                                                                  uint32_t capacity, uint32_t* __restrict__ tile_begin, uint32_t* __restrict__ tile_end) {
    const uint32_t n = cpv_pairs_in_bounds(pair_total, capacity);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = keys[i];
        if (i == 0u || keys[i - 1u] != k) tile_begin[k] = i;
        if (i + 1u == n || keys[i + 1u] != k) tile_end[k] = i + 1u;
    }
}

/* ---- vkCmdBlitImage (CPVulkan/CommandBuffer.cpp:32-240), colour aspect ----
 *
 * One thread per destination texel of a region (2D; the reference's third
 * axis has depth 1 and contributes an exact lerp by 0). Its source position
 * is the reference's: u = (dstX + 0.5 - dst0.x) * ((src1.x - src0.x) / (dst1.x
 * - dst0.x)) + src0.x in binary32, normalised by the source level's width,
 * and the source level is sampled as SampleImage samples it for a blit
 * (level 0 of a one-level image, the blit's filter, CLAMP_TO_EDGE). The
 * result is written through the UNORM8 encoder. `src` describes the source
 * level as level 0. */
struct CpvBlitRegion {
    int32_t src[4]; /* x0, y0, x1, y1 */
    int32_t dst[4];
};

extern "C" __global__ void __launch_bounds__(256) cpv_blit(CpvTexture src, uint8_t* __restrict__ dst, uint32_t dst_w, uint32_t dst_h,
                                                           uint32_t dst_format, CpvBlitRegion r, uint32_t filter) {
    const int32_t dw = abs(r.dst[2] - r.dst[0]), dh = abs(r.dst[3] - r.dst[1]);
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (dw == 0 || dh == 0 || i >= static_cast<uint64_t>(dw) * dh) return;
    const int32_t x = static_cast<int32_t>(i % static_cast<uint64_t>(dw)), y = static_cast<int32_t>(i / static_cast<uint64_t>(dw));
    const int32_t dst_x = r.dst[2] < r.dst[0] ? x + r.dst[2] : x + r.dst[0];
    const int32_t dst_y = r.dst[3] < r.dst[1] ? y + r.dst[3] : y + r.dst[1];
    if (dst_x < 0 || dst_y < 0 || dst_x >= static_cast<int32_t>(dst_w) || dst_y >= static_cast<int32_t>(dst_h)) return;
    const float sx = __fdiv_rn(static_cast<float>(r.src[2] - r.src[0]), static_cast<float>(r.dst[2] - r.dst[0]));
    const float sy = __fdiv_rn(static_cast<float>(r.src[3] - r.src[1]), static_cast<float>(r.dst[3] - r.dst[1]));
    const float u = __fadd_rn(__fmul_rn(__fsub_rn(__fadd_rn(static_cast<float>(dst_x), 0.5f), static_cast<float>(r.dst[0])), sx),
                              static_cast<float>(r.src[0]));
    const float v = __fadd_rn(__fmul_rn(__fsub_rn(__fadd_rn(static_cast<float>(dst_y), 0.5f), static_cast<float>(r.dst[1])), sy),
                              static_cast<float>(r.src[1]));
    float value[4];
    cpv_sample_level(src, 0u, __fdiv_rn(u, __uint2float_rn(src.level_w[0])), __fdiv_rn(v, __uint2float_rn(src.level_h[0])), filter, value);
    uint32_t packed = 0u;
    const bool bgra = dst_format == CPV_FMT_B8G8R8A8_UNORM;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int byte = (bgra && c < 3) ? 2 - c : c;
        packed |= cpv_encode_unorm(value[c], 255.0f) << (8 * byte);
    }
    reinterpret_cast<uint32_t*>(dst)[static_cast<uint64_t>(dst_y) * dst_w + dst_x] = packed;
}

/* ---- fills ---- */

extern "C" __global__ void __launch_bounds__(256) cpv_fill_u32(uint32_t* __restrict__ dst, uint64_t count, uint32_t value) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        dst[i] = value;
}

extern "C" __global__ void __launch_bounds__(256) cpv_fill_u16(uint16_t* __restrict__ dst, uint64_t count, uint32_t value) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        dst[i] = static_cast<uint16_t>(value);
}

extern "C" __global__ void __launch_bounds__(256) cpv_fill_u64(uint2* __restrict__ dst, uint64_t count, uint32_t lo, uint32_t hi) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        dst[i] = make_uint2(lo, hi);
}

extern "C" __global__ void __launch_bounds__(256) cpv_fill_u128(uint4* __restrict__ dst, uint64_t count, uint4 value) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        dst[i] = value;
}

/* Fill of a w x h texel rectangle whose rows start `pitch` bytes apart with
 * the texel v (words x, y, z, w): a 2-byte texel takes the low half of v.x;
 * 4- and 8-byte texels take v.x in their first word when write_lo, an
 * 8-byte texel v.y in its second word when write_hi (a D32 + stencil
 * texel's stencil, or an 8-byte colour texel's upper half), a 16-byte
 * texel all four words. */
extern "C" __global__ void __launch_bounds__(256) cpv_fill_rect(uint8_t* __restrict__ base, uint64_t pitch, uint32_t w, uint32_t h, uint32_t texel_bytes,
                                                                uint4 v, uint32_t write_lo, uint32_t write_hi) {
    const uint32_t lo = v.x, hi = v.y;
    /* rows over blockIdx.y, texels of a row over x */
    for (uint32_t y = blockIdx.y; y < h; y += gridDim.y) {
        uint8_t* row = base + static_cast<uint64_t>(y) * pitch;
        for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < w; x += gridDim.x * blockDim.x) {
            uint8_t* p = row + static_cast<uint64_t>(x) * texel_bytes;
            if (texel_bytes == 1) {
                *p = static_cast<uint8_t>(lo);
            } else if (texel_bytes == 2) {
                *reinterpret_cast<uint16_t*>(p) = static_cast<uint16_t>(lo);
            } else if (texel_bytes == 16) {
                *reinterpret_cast<uint4*>(p) = v;
            } else {
                if (write_lo) *reinterpret_cast<uint32_t*>(p) = lo;
                if (texel_bytes == 8 && write_hi) *reinterpret_cast<uint32_t*>(p + 4) = hi;
            }
        }
    }
}

/* ---- host → HBM copy read by the SMs ----
 * Copies `words` 16-byte words from pinned host memory (device-accessible)
 * to HBM with every SM issuing loads across the chip-to-chip link. Both
 * pointers are 16-byte aligned; the caller copies any tail. */
extern "C" __global__ void __launch_bounds__(256) cpv_copy_words(uint4* __restrict__ dst, const uint4* __restrict__ src, uint64_t words) {
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    /* four independent loads in flight per thread */
    for (; i + 3 * stride < words; i += 4 * stride) {
        const uint4 a = src[i], b = src[i + stride], c = src[i + 2 * stride], d = src[i + 3 * stride];
        dst[i] = a;
        dst[i + stride] = b;
        dst[i + 2 * stride] = c;
        dst[i + 3 * stride] = d;
    }
    for (; i < words; i += stride) dst[i] = src[i];
}

#endif /* CPV_BIN_CUH */
