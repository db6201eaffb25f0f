/*
 * cpv_bin.cuh — order-preserving sort-middle binning and the other generic
 * device kernels (the batched sort, blits, fills, copies).
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
 * CUDA graph. The list has a capacity; a draw that would exceed it
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

/* The words of a batch: its pairs, the raster's tile counter, the sort's
 * chunks a CTA and its CTAs that have any, the two digits' totals. */
#define CPV_WORD_PAIRS 0
#define CPV_WORD_TILE 2
#define CPV_WORD_CHUNKS 3
#define CPV_WORD_DIGITS 4
#define CPV_WORD_ROWS 8

/* 2. counts[row][bin] → the list position of the row's first entry in the
 * bin; range[bin] = the bin's list. One CTA of 1024 threads per 8 bins: 128
 * groups of rows are summed, scanned over the groups and walked again. A
 * bin's list starts where an atomic on *total puts it (the lists' order in
 * memory does not matter); *total (zeroed by cpv_setup_rects) ends as the
 * draw's pair count. With `words` the columns are a sort digit's counts and
 * the rows are those of CPV_WORD_ROWS. */
#define CPV_BIN_SCAN_THREADS 1024
#define CPV_BIN_SCAN_BINS 8
extern "C" __global__ void __launch_bounds__(CPV_BIN_SCAN_THREADS) cpv_bin_scan(uint32_t* __restrict__ counts, uint32_t rows, uint32_t bins,
                                                                               uint2* __restrict__ range, unsigned long long* __restrict__ total,
                                                                               const uint32_t* __restrict__ words) {
    __shared__ uint32_t warp_sums[CPV_BIN_SCAN_THREADS / 32][CPV_BIN_SCAN_BINS];
    __shared__ uint32_t list_base[CPV_BIN_SCAN_BINS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t b = threadIdx.x % CPV_BIN_SCAN_BINS, group = threadIdx.x / CPV_BIN_SCAN_BINS;
    const uint32_t bin = blockIdx.x * CPV_BIN_SCAN_BINS + b;
    const uint32_t groups = CPV_BIN_SCAN_THREADS / CPV_BIN_SCAN_BINS;
    if (words) rows = words[CPV_WORD_ROWS];
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
 * A draw over the capacity leaves its pairs in *need (host memory; may be
 * null), for the host to grow the lists. Dynamic shared memory: 9 words per
 * bin. */
extern "C" __global__ void __launch_bounds__(256) cpv_bin_write(const uint2* __restrict__ rects, uint64_t prims, uint32_t row_prims, uint32_t shift,
                                                                uint32_t bins_x, uint32_t bins, const uint32_t* __restrict__ offsets,
                                                                uint32_t* __restrict__ list, uint32_t* __restrict__ list_rects, uint32_t capacity,
                                                                const unsigned long long* __restrict__ total, unsigned long long* need) {
    extern __shared__ uint32_t cpv_bin_smem[];
    if (*total > capacity) {
        if (need && blockIdx.x == 0u && threadIdx.x == 0u && *need < *total) *need = *total;
        return;
    }
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

/* ---- batched binning: pairs, stable radix sort by tile, tile ranges ----
 *
 * The batched path bins every draw of a render pass at once. Set-up writes
 * one tile rectangle per primitive and the pair count of each 256-primitive
 * block; cpv_batch_scan makes the counts positions within chunks of
 * CPV_SCAN_BLOCK blocks; cpv_batch_emit writes the (tile, primitive) pairs
 * in primitive order; a stable radix sort by tile (one digit of at most
 * CPV_RADIX_DIGITS, or two) groups them by tile while keeping primitive
 * (API) order inside each tile. Each digit takes three launches:
 * cpv_radix_hist, cpv_bin_scan over its counts, cpv_radix_scatter. The
 * groups of one digit may lie in any order (cpv_bin_scan places them by an
 * atomic): a tile's pairs stay together and in order all the same. With one
 * digit the scan's ranges are the tiles'; with two, cpv_tile_ranges records
 * where each tile's run starts and ends. Sizes that depend on the data (the
 * pair count) are read on the device, so the sequence has fixed launch
 * shapes, needs no memset and can be captured in a CUDA graph. Pairs beyond
 * the capacity are not written; the raster then scans the rectangles instead
 * (same image). */

#define CPV_SCAN_THREADS 256
#define CPV_SCAN_ITEMS 8
#define CPV_SCAN_BLOCK (CPV_SCAN_THREADS * CPV_SCAN_ITEMS)
#define CPV_RADIX_THREADS 256
#define CPV_RADIX_DIGITS 1024
#define CPV_RADIX_ITEMS 8
#define CPV_RADIX_CHUNK (CPV_RADIX_THREADS * CPV_RADIX_ITEMS)

__device__ __forceinline__ uint32_t cpv_pairs_in_bounds(const uint32_t* words, uint32_t capacity) {
    const uint32_t p = words[CPV_WORD_PAIRS];
    return p <= capacity ? p : 0u;
}

/* Exclusive sum over the warp; `total` is the warp's sum. */
__device__ __forceinline__ uint32_t cpv_warp_exclusive(uint32_t v, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t incl = v;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += t;
    }
    total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    return incl - v;
}

/* Block-wide exclusive sum over 256 threads; `total` is the block's sum. */
__device__ __forceinline__ uint32_t cpv_block256_exclusive(uint32_t v, uint32_t* warp_sums /* [8] */, uint32_t& total) {
    const uint32_t warp = threadIdx.x >> 5;
    uint32_t mine;
    const uint32_t excl = cpv_warp_exclusive(v, mine);
    if ((threadIdx.x & 31u) == 0u) warp_sums[warp] = mine;
    __syncthreads();
    uint32_t base = 0;
    total = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8u; k++) {
        const uint32_t s = warp_sums[k];
        base += k < warp ? s : 0u;
        total += s;
    }
    return base + excl;
}

/* out[i] = exclusive prefix of in within its chunk; chunk_sums[b] = chunk total. */
extern "C" __global__ void __launch_bounds__(CPV_SCAN_THREADS) cpv_batch_scan(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t n,
                                                                              uint32_t* __restrict__ chunk_sums) {
    __shared__ uint32_t warp_sums[8];
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * CPV_SCAN_BLOCK + static_cast<uint64_t>(threadIdx.x) * CPV_SCAN_ITEMS;
    uint32_t v[CPV_SCAN_ITEMS];
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < CPV_SCAN_ITEMS; i++) {
        v[i] = (base + i < n) ? in[base + i] : 0u;
        sum += v[i];
    }
    uint32_t total;
    uint32_t run = cpv_block256_exclusive(sum, warp_sums, total);
#pragma unroll
    for (int i = 0; i < CPV_SCAN_ITEMS; i++) {
        if (base + i < n) out[base + i] = run;
        run += v[i];
    }
    if (threadIdx.x == 0) chunk_sums[blockIdx.x] = total;
}

/* One warp per set-up block, eight blocks (of one chunk) a CTA: the block's
 * pairs at the position of its chunk (summed here from the chunks' totals)
 * + block_offsets[block] + the pairs of its earlier primitives. A block
 * without pairs has no rectangles written this frame and emits nothing. A
 * lane writes its primitive's pairs; those of one with many are written by
 * the warp. Two dependent loads, then stores of 6 bytes a pair: latency-bound
 * (99 M primitives, 30 M pairs: 260 us; a CTA per block, a block-wide scan
 * and a division a pair took 500, every register of one fewer CTA an SM 272).
 * CTA 0 stores the pair total, clears the words of the kernels that follow
 * and shares the pairs out among the sort's CTAs: whole chunks, as few each as
 * cover them, for the `sort_ctas` that are launched (four an SM); those
 * without any leave at once. One digit's scatter with the pairs split evenly
 * over all 608 CTAs, then in whole chunks: 14.6 us then 8.5 for 316k pairs and
 * 1024 digits (155 CTAs; 12.2 at 78 of two chunks), 15.9 then 12.4 for 1.7 M
 * pairs and 128 digits. By the pairs of each frame, since those of the plan's
 * build may be none: geometry moves under a recorded command buffer. */
#define CPV_EMIT_LANE_PAIRS 16u
extern "C" __global__ void __launch_bounds__(256, 6) cpv_batch_emit(const uint2* __restrict__ rects, const uint32_t* __restrict__ block_pairs,
                                                                 const uint32_t* __restrict__ block_offsets, const uint32_t* __restrict__ chunk_sums,
                                                                 uint32_t blocks, uint32_t tiles_x, uint16_t* __restrict__ keys,
                                                                 uint32_t* __restrict__ vals, uint32_t capacity, uint32_t* __restrict__ words,
                                                                 uint32_t sort_ctas) {
    __shared__ uint32_t sums[2][8];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t block = blockIdx.x * 8u + warp;
    const bool any = block < blocks;
    const uint32_t block_n = any ? block_pairs[block] : 0u, block_pos = any ? block_offsets[block] : 0u;
    const uint32_t chunk = blockIdx.x * 8u / CPV_SCAN_BLOCK, chunks = (blocks + CPV_SCAN_BLOCK - 1u) / CPV_SCAN_BLOCK;
    uint32_t before = 0u, total = 0u;
    for (uint32_t i = threadIdx.x; i < chunks; i += 256u) {
        const uint32_t s = chunk_sums[i];
        total += s;
        before += i < chunk ? s : 0u;
    }
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    total = __reduce_add_sync(0xFFFFFFFFu, total);
    if (lane == 0u) {
        sums[0][warp] = before;
        sums[1][warp] = total;
    }
    __syncthreads();
    before = total = 0u;
#pragma unroll
    for (int w = 0; w < 8; w++) {
        before += sums[0][w];
        total += sums[1][w];
    }
    if (blockIdx.x == 0u && threadIdx.x == 0u) {
        const uint32_t chunks_of_pairs = total <= capacity ? total / CPV_RADIX_CHUNK + (total % CPV_RADIX_CHUNK ? 1u : 0u) : 0u;
        const uint32_t per = (chunks_of_pairs + sort_ctas - 1u) / sort_ctas;
        words[CPV_WORD_PAIRS] = total;
        words[CPV_WORD_TILE] = 0u;
        words[CPV_WORD_CHUNKS] = per;
        words[CPV_WORD_ROWS] = per ? (chunks_of_pairs + per - 1u) / per : 0u;
        for (uint32_t i = 0; i < 4u; i++) words[CPV_WORD_DIGITS + i] = 0u;
    }
    if (total > capacity || block_n == 0u) return;
    uint2 r[8];
    const uint32_t g0 = block * 256u + lane;
#pragma unroll
    for (uint32_t j = 0; j < 8u; j++) r[j] = rects[g0 + 32u * j];
    uint32_t pos = before + block_pos;
#pragma unroll
    for (uint32_t j = 0; j < 8u; j++) {
        const uint32_t x0 = r[j].x & 0xFFFFu, y0 = r[j].x >> 16;
        const uint32_t w = (r[j].y & 0xFFFFu) - x0;
        const uint32_t n = w * ((r[j].y >> 16) - y0);
        /* positions by ballots for up to three pairs each, else by a scan */
        const uint32_t ones = __ballot_sync(0xFFFFFFFFu, (n & 1u) != 0u), more = __ballot_sync(0xFFFFFFFFu, n > 1u);
        if ((ones | more) == 0u) continue;
        const uint32_t earlier = (1u << lane) - 1u;
        uint32_t p = pos + __popc(ones & earlier), step = __popc(ones), many = 0u;
        if (more) {
            if (__any_sync(0xFFFFFFFFu, n > 3u)) {
                p = pos + cpv_warp_exclusive(n, step);
                many = __ballot_sync(0xFFFFFFFFu, n > CPV_EMIT_LANE_PAIRS);
            } else {
                const uint32_t twos = __ballot_sync(0xFFFFFFFFu, (n & 2u) != 0u);
                p += 2u * __popc(twos & earlier);
                step += 2u * __popc(twos);
            }
        }
        pos += step;
        uint32_t key = y0 * tiles_x + x0;
        while (many) {
            const uint32_t src = __ffs(static_cast<int>(many)) - 1u;
            many &= many - 1u;
            const uint32_t s_key = __shfl_sync(0xFFFFFFFFu, key, src), s_w = __shfl_sync(0xFFFFFFFFu, w, src), s_n = __shfl_sync(0xFFFFFFFFu, n, src);
            const uint32_t s_p = __shfl_sync(0xFFFFFFFFu, p, src), s_g = __shfl_sync(0xFFFFFFFFu, g0, src) + 32u * j;
            for (uint32_t k = lane; k < s_n; k += 32u) {
                const uint32_t row = k / s_w;
                if (s_p + k < capacity) {  /* always, unless the pair total wrapped 32 bits */
                    keys[s_p + k] = static_cast<uint16_t>(s_key + row * tiles_x + (k - row * s_w));
                    vals[s_p + k] = s_g;
                }
            }
        }
        if (n <= CPV_EMIT_LANE_PAIRS) {
            uint32_t x = 0u;
            for (uint32_t k = 0; k < n; k++, p++) {
                if (p < capacity) {
                    keys[p] = static_cast<uint16_t>(key);
                    vals[p] = g0 + 32u * j;
                }
                key++;
                if (++x == w) {
                    x = 0u;
                    key += tiles_x - w;
                }
            }
        }
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

/* The CTA's range of the pairs. */
__device__ __forceinline__ void cpv_cta_range(const uint32_t* words, uint32_t capacity, uint32_t& begin, uint32_t& end) {
    const uint32_t n = cpv_pairs_in_bounds(words, capacity);
    const uint64_t per = static_cast<uint64_t>(words[CPV_WORD_CHUNKS]) * CPV_RADIX_CHUNK;
    const uint64_t b = per * blockIdx.x, e = b + per;
    begin = static_cast<uint32_t>(b < n ? b : n);
    end = static_cast<uint32_t>(e < n ? e : n);
}

/* counts[cta * digits + digit] = items of the CTA's range with that digit.
 * With tile_range (the first of two digits) it is also cleared here, for
 * cpv_tile_ranges to fill. */
extern "C" __global__ void __launch_bounds__(CPV_RADIX_THREADS) cpv_radix_hist(const uint16_t* __restrict__ keys, const uint32_t* __restrict__ words,
                                                                               uint32_t capacity, uint32_t shift, uint32_t digits,
                                                                               uint32_t* __restrict__ counts, uint2* __restrict__ tile_range, uint32_t tiles) {
    __shared__ uint32_t count[CPV_RADIX_DIGITS];
    if (tile_range)
        for (uint32_t i = blockIdx.x * CPV_RADIX_THREADS + threadIdx.x; i < tiles; i += gridDim.x * CPV_RADIX_THREADS) tile_range[i] = make_uint2(0u, 0u);
    uint32_t begin, end;
    cpv_cta_range(words, capacity, begin, end);
    if (begin >= end) return;  /* not one of the rows */
    for (uint32_t d = threadIdx.x; d < digits; d += CPV_RADIX_THREADS) count[d] = 0u;
    __syncthreads();
    for (uint32_t i = begin + 8u * threadIdx.x; i < end; i += 8u * CPV_RADIX_THREADS) {
        /* the buffer is a multiple of 8 keys long */
        const uint4 v = *reinterpret_cast<const uint4*>(keys + i);
        const uint32_t word[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (uint32_t k = 0; k < 8u; k++)
            if (i + k < end) atomicAdd(&count[(((word[k >> 1] >> (16u * (k & 1u))) & 0xFFFFu) >> shift) & (digits - 1u)], 1u);
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < digits; d += CPV_RADIX_THREADS) counts[blockIdx.x * digits + d] = count[d];
}

/* Stable scatter to `offsets` (the counts made positions). Each CTA walks
 * its range in order, CPV_RADIX_CHUNK items at a time: every warp ranks its
 * 256 consecutive items by digit (a match-any rank within 32, the warp's own
 * count per digit between them), the counts are scanned over the warps and
 * the digits, and the chunk is put in digit order in shared memory first, so
 * that the writes to a digit's run are consecutive. keys_out may be null (the
 * last digit of a one-digit sort). Bound by the chunk's chain of shared
 * memory steps at four CTAs an SM (30 M pairs, 14400 tiles, both passes: 267 us;
 * 646 before, with 256 items a step written straight from the match and
 * 32-bit keys; ballots per bit instead of the match 328). */
extern "C" __global__ void __launch_bounds__(CPV_RADIX_THREADS) cpv_radix_scatter(const uint16_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                                                                                  uint16_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                                                                  const uint32_t* __restrict__ words, uint32_t capacity, uint32_t shift,
                                                                                  uint32_t digits, const uint32_t* __restrict__ offsets) {
    __shared__ uint32_t next[CPV_RADIX_DIGITS];   /* the digit's next position */
    __shared__ uint32_t place[CPV_RADIX_DIGITS];  /* that, less the digit's first position in the chunk */
    __shared__ uint16_t first[CPV_RADIX_DIGITS];  /* the digit's first position in the chunk */
    __shared__ uint16_t warp_count[CPV_RADIX_THREADS / 32][CPV_RADIX_DIGITS];
    __shared__ uint32_t chunk_val[CPV_RADIX_CHUNK];
    __shared__ uint16_t chunk_key[CPV_RADIX_CHUNK];
    __shared__ uint32_t warp_sums[8];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t per_thread = (digits + CPV_RADIX_THREADS - 1u) / CPV_RADIX_THREADS, d0 = threadIdx.x * per_thread;
    uint32_t begin, end;
    cpv_cta_range(words, capacity, begin, end);
    if (begin >= end) return;
    for (uint32_t d = threadIdx.x; d < digits; d += CPV_RADIX_THREADS) {
        next[d] = offsets[blockIdx.x * digits + d];
#pragma unroll
        for (uint32_t w = 0; w < CPV_RADIX_THREADS / 32u; w++) warp_count[w][d] = 0u;
    }
    __syncthreads();
    for (uint32_t base = begin; base < end; base += CPV_RADIX_CHUNK) {
        const uint32_t items = end - base < CPV_RADIX_CHUNK ? end - base : CPV_RADIX_CHUNK;
        uint32_t key[CPV_RADIX_ITEMS], val[CPV_RADIX_ITEMS], rank[CPV_RADIX_ITEMS];  /* rank: first the lanes of the same digit */
        const uint32_t i0 = warp * 32u * CPV_RADIX_ITEMS + lane;
#pragma unroll
        for (uint32_t j = 0; j < CPV_RADIX_ITEMS; j++) {
            const bool valid = i0 + 32u * j < items;
            key[j] = valid ? keys_in[base + i0 + 32u * j] : 0u;
            val[j] = valid ? vals_in[base + i0 + 32u * j] : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < CPV_RADIX_ITEMS; j++)
            rank[j] = __match_any_sync(0xFFFFFFFFu, i0 + 32u * j < items ? (key[j] >> shift) & (digits - 1u) : CPV_RADIX_DIGITS + lane);
#pragma unroll
        for (uint32_t j = 0; j < CPV_RADIX_ITEMS; j++) {
            const bool valid = i0 + 32u * j < items;
            const uint32_t digit = (key[j] >> shift) & (digits - 1u);
            const uint32_t peers = rank[j];
            const uint32_t earlier = __popc(peers & ((1u << lane) - 1u));
            const uint32_t seen = warp_count[warp][digit];
            rank[j] = seen + earlier;
            __syncwarp();
            if (valid && earlier == 0u) warp_count[warp][digit] = static_cast<uint16_t>(seen + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        uint32_t count[CPV_RADIX_DIGITS / CPV_RADIX_THREADS], sum = 0u;
#pragma unroll
        for (uint32_t m = 0; m < CPV_RADIX_DIGITS / CPV_RADIX_THREADS; m++) {
            uint32_t run = 0u;
            if (m < per_thread && d0 + m < digits) {
#pragma unroll
                for (uint32_t w = 0; w < CPV_RADIX_THREADS / 32u; w++) {
                    const uint32_t c = warp_count[w][d0 + m];
                    warp_count[w][d0 + m] = static_cast<uint16_t>(run);
                    run += c;
                }
            }
            count[m] = run;
            sum += run;
        }
        uint32_t total;
        uint32_t run = cpv_block256_exclusive(sum, warp_sums, total);
#pragma unroll
        for (uint32_t m = 0; m < CPV_RADIX_DIGITS / CPV_RADIX_THREADS; m++) {
            if (m < per_thread && d0 + m < digits) {
                const uint32_t at = next[d0 + m];
                first[d0 + m] = static_cast<uint16_t>(run);
                place[d0 + m] = at - run;
                next[d0 + m] = at + count[m];
                run += count[m];
            }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < CPV_RADIX_ITEMS; j++) {
            if (i0 + 32u * j < items) {
                const uint32_t digit = (key[j] >> shift) & (digits - 1u);
                const uint32_t p = first[digit] + warp_count[warp][digit] + rank[j];
                chunk_key[p] = static_cast<uint16_t>(key[j]);
                chunk_val[p] = val[j];
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < items; i += CPV_RADIX_THREADS) {
            const uint32_t k = chunk_key[i];
            const uint32_t p = place[(k >> shift) & (digits - 1u)] + i;
            if (keys_out) keys_out[p] = static_cast<uint16_t>(k);
            vals_out[p] = chunk_val[i];
        }
        for (uint32_t d = lane; d < digits; d += 32u) warp_count[warp][d] = 0u;
        __syncthreads();
    }
}

/* tile_range (zeroed beforehand) from the sorted keys, eight a thread. */
extern "C" __global__ void __launch_bounds__(256) cpv_tile_ranges(const uint16_t* __restrict__ keys, const uint32_t* __restrict__ words,
                                                                  uint32_t capacity, uint2* __restrict__ tile_range) {
    const uint32_t n = cpv_pairs_in_bounds(words, capacity);
    for (uint64_t at = 8ull * (blockIdx.x * 256u + threadIdx.x); at < n; at += 8ull * 256u * gridDim.x) {
        const uint32_t i = static_cast<uint32_t>(at);
        const uint4 v = *reinterpret_cast<const uint4*>(keys + i);
        const uint32_t word[4] = {v.x, v.y, v.z, v.w};
        uint32_t before = i ? keys[i - 1u] : 0x10000u;
#pragma unroll
        for (uint32_t k = 0; k < 8u; k++) {
            const uint32_t key = (word[k >> 1] >> (16u * (k & 1u))) & 0xFFFFu;
            if (i + k < n) {
                if (key != before) {
                    tile_range[key].x = i + k;
                    if (before < 0x10000u) tile_range[before].y = i + k;
                }
                if (i + k + 1u == n) tile_range[key].y = n;
            }
            before = key;
        }
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
