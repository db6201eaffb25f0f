/*
 * cpv_pipeline.cuh — the kernels of one graphics pipeline for the per-draw
 * path. Compiled by NVRTC at vkCreateGraphicsPipelines after cpv_device.cuh,
 * cpv_raster.cuh and the pipeline's stage functions (cpv_stage.cuh in
 * namespace cpv_p0).
 *
 * Kernels:
 *   cpv_setup_rects — one thread per primitive: runs the vertex shader for the
 *                     primitive's three vertices (positions only), the
 *                     reference's bounding box and cull test, and writes the
 *                     primitive's screen-tile rectangle and its row's
 *                     per-bin counts for the binning (cpv_bin.cuh).
 *   cpv_raster      — one CTA per screen tile: walks the tile's primitives in
 *                     API order (cpv_raster_tile), evaluates coverage per pixel
 *                     with the reference's float edge functions, interpolates,
 *                     runs the fragment shader and the per-fragment operations
 *                     against colour/depth/stencil held in registers, and
 *                     writes the tile back once.
 * Parameters are __grid_constant__: device functions read them in place
 * through references, without a per-thread copy.
 */
#ifndef CPV_PIPELINE_CUH
#define CPV_PIPELINE_CUH

/* One CTA per row of row_prims primitives. With bins (P.bin_counts) it also
 * counts the row's primitives per bin; the first CTA clears the draw's pair
 * total for the scan that follows. */
extern "C" __global__ void __launch_bounds__(256) cpv_setup_rects(const __grid_constant__ CpvDrawParams P) {
    __shared__ uint32_t hist[CPV_MAX_BINS];
    const bool lists = P.bin_counts != nullptr;
    if (lists) {
        for (uint32_t i = threadIdx.x; i < P.bins; i += 256u) hist[i] = 0u;
        if (blockIdx.x == 0u && threadIdx.x == 0u) *P.pair_total = 0ull;
    }
    __syncthreads();
    const uint64_t begin = static_cast<uint64_t>(blockIdx.x) * P.row_prims;
    const uint64_t end = begin + P.row_prims < P.total_prims ? begin + P.row_prims : P.total_prims;
    for (uint64_t g = begin + threadIdx.x; g < end; g += 256u) {
        CpvTri t;
        int4 box;
        cpv_p0::Stage::setup<false>(P, g, t, box);
        const uint2 r = cpv_tile_rect(t, box, P.viewport[2], P.viewport[3]);
        P.rects[g] = r;
        const uint32_t x0 = r.x & 0xFFFFu, y0 = r.x >> 16, x1 = r.y & 0xFFFFu, y1 = r.y >> 16;
        if (lists && x1 > x0 && y1 > y0) {
            const uint32_t s = P.bin_shift;
            for (uint32_t by = y0 >> s; by <= (y1 - 1u) >> s; by++)
                for (uint32_t bx = x0 >> s; bx <= (x1 - 1u) >> s; bx++) atomicAdd(&hist[by * P.bins_x + bx], 1u);
        }
    }
    if (lists) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < P.bins; i += 256u) P.bin_counts[static_cast<uint64_t>(blockIdx.x) * P.bins + i] = hist[i];
    }
}

/* Blend tables (pipelines that blend a per-primitive constant colour): one
 * thread per primitive shades it (vertex shader, flat inputs, fragment
 * shader), then the CTA fills the 4 × 256-byte table of each live primitive
 * of its 256, one destination byte per thread. Primitives whose tile
 * rectangle is empty are skipped (the raster never reads their tables). */
extern "C" __global__ void __launch_bounds__(256) cpv_blend_tables(const __grid_constant__ CpvDrawParams P) {
    __shared__ float colours[256][4];
    __shared__ uint32_t live[256];
    const uint64_t g = static_cast<uint64_t>(blockIdx.x) * 256u + threadIdx.x;
    uint32_t ok = 0u;
    if (cpv_p0::kBlendTable && g < P.total_prims) {
        bool drawn = true;
        if (P.rects) {
            const uint2 r = P.rects[g];
            drawn = r.x != r.y;  /* empty rectangles are all-zero */
        }
        if (drawn) {
            CpvTri t;
            int4 box;
            cpv_p0::Stage::setup<true>(P, g, t, box);
            ok = cpv_tri_live(t) ? 1u : 0u;
#pragma unroll
            for (int c = 0; c < 4; c++) colours[threadIdx.x][c] = t.var[0][c];
        }
    }
    live[threadIdx.x] = ok;
    __syncthreads();
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * 256u;
    for (uint32_t k = 0; k < 256u; k++) {
        if (!live[k]) continue;
        const float colour[4] = {colours[k][0], colours[k][1], colours[k][2], colours[k][3]};
        uint8_t bytes[4];
        cpv_p0::cpv_blend_table_column(colour, P.blend_constants, threadIdx.x, bytes);
        uint8_t* table = P.tables + (first + k) * 1024u;
#pragma unroll
        for (int c = 0; c < 4; c++) table[c * 256 + threadIdx.x] = bytes[c];
    }
}

/* Entries of a list that a CTA filters per step, and the ring of primitive
 * ids that passed: up to CPV_BATCH - 1 wait while a step adds its own. */
#define CPV_FILTER_STEP (2u * CPV_RT_THREADS)
#define CPV_RING_SIZE (CPV_BATCH + CPV_FILTER_STEP)

/* A tile's progress through its entries, in shared memory: between batches
 * it would only hold registers of the fragment loops. */
struct CpvTileList {
    uint32_t ring[CPV_RING_SIZE];  /* ids that passed the filter */
    uint32_t pos, end;             /* entries (or primitives) not yet looked at */
    uint32_t head, waiting, taken; /* ring state; taken: the size of the current batch */
    uint32_t by_list;              /* entries of the bin's list, else all primitives */
};

/* Primitives of one tile of a single draw, in API order: every primitive
 * (direct mode); the entries of the tile's bin list whose rectangle holds
 * the tile; or every primitive whose rectangle does (draws too small for
 * lists, or a list over its capacity). Rectangles are read coalesced, two
 * entries a thread and step, and compacted in order into a ring in shared
 * memory from which the set-up takes batches. */
struct CpvPlainSource {
    const CpvDrawParams& P;
    CpvTileList& L;
    float vw, vh;
    uint32_t fb_width, fb_height;

    __device__ __forceinline__ bool holds(uint32_t i, bool by_list, uint32_t tx, uint32_t ty) const {
        if (by_list) {
            const uint32_t r = P.bin_rects[i];
            return tx >= (r & 0xFFu) && ty >= ((r >> 8) & 0xFFu) && tx < ((r >> 16) & 0xFFu) && ty < (r >> 24);
        }
        if (!P.rects) return true;
        const uint2 r = P.rects[i];
        return tx >= (r.x & 0xFFFFu) && ty >= (r.x >> 16) && tx < (r.y & 0xFFFFu) && ty < (r.y >> 16);
    }
    static __device__ __forceinline__ uint32_t wrap(uint32_t i) { return i >= CPV_RING_SIZE ? i - CPV_RING_SIZE : i; }
    /* The next batch: its size, up to CPV_BATCH; 0 when the tile is done.
     * Every thread of the CTA calls it, none still reading the last batch's
     * ids; a barrier follows before the ids are read. */
    __device__ __forceinline__ uint32_t next(uint32_t* warp_sums) {
        uint32_t pos = L.pos, waiting = L.waiting - L.taken;
        const uint32_t end = L.end;
        if (waiting == 0u && pos >= end) return 0u;
        const uint32_t head = wrap(L.head + L.taken);
        const bool by_list = L.by_list != 0u;
        const uint32_t mask = by_list ? (1u << P.bin_shift) - 1u : 0xFFFFFFFFu;
        const uint32_t tx = (blockIdx.x % P.tiles_x) & mask, ty = (blockIdx.x / P.tiles_x) & mask;
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
        const uint32_t lt_mask = (1u << lane) - 1u;
        while (waiting < CPV_BATCH && pos < end) {
            const uint32_t left = end - pos;
            const uint32_t i0 = pos + threadIdx.x, i1 = i0 + CPV_RT_THREADS;
            const bool h0 = threadIdx.x < left && holds(i0, by_list, tx, ty);
            const bool h1 = threadIdx.x + CPV_RT_THREADS < left && holds(i1, by_list, tx, ty);
            const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, h0), b1 = __ballot_sync(0xFFFFFFFFu, h1);
            if (lane == 0u) warp_sums[warp] = __popc(b0) | (__popc(b1) << 16);
            __syncthreads();
            uint32_t before = 0u, all = 0u;
            for (uint32_t w = 0; w < CPV_RT_THREADS / 32; w++) {
                const uint32_t s = warp_sums[w];
                if (w < warp) before += s;
                all += s;
            }
            const uint32_t tail = head + waiting;
            if (h0) L.ring[wrap(tail + (before & 0xFFFFu) + __popc(b0 & lt_mask))] = by_list ? P.bin_list[i0] : i0;
            if (h1) L.ring[wrap(tail + (all & 0xFFFFu) + (before >> 16) + __popc(b1 & lt_mask))] = by_list ? P.bin_list[i1] : i1;
            waiting += (all & 0xFFFFu) + (all >> 16);
            pos = left > CPV_FILTER_STEP ? pos + CPV_FILTER_STEP : end;
            __syncthreads();
        }
        const uint32_t taken = waiting < CPV_BATCH ? waiting : CPV_BATCH;
        __syncthreads();  /* every thread has read L's words */
        if (threadIdx.x == 0u) {
            L.head = head;
            L.waiting = waiting;
            L.taken = taken;
            L.pos = pos;
        }
        return taken;
    }
    /* Sets up the i-th primitive of the current batch. */
    __device__ __forceinline__ void setup(uint32_t i, CpvTri& t, int4& box) const {
        cpv_p0::Stage::setup<true>(P, L.ring[wrap(L.head + i)], t, box);
    }
    __device__ __forceinline__ bool shade(const CpvTri& t, const float w[3], int32_t x, int32_t y, float* colour, float& mapped,
                                          const CpvPixel* early = nullptr) const {
        return cpv_p0::Stage::shade(P, t, w, x, y, colour, mapped, early);
    }
    __device__ __forceinline__ void rop(const CpvTri& t, const float* colour, float mapped, CpvPixel& s) const {
        cpv_p0::Stage::rop(P.blend_constants, cpv_tri_front(t), colour, mapped, s, cpv_p0::Stage::table(P, t));
    }
    /* A covered fragment of a table-only pipeline: the table lookup is the
     * whole of shade + rop (the colour is constant and nothing discards a
     * live primitive). */
    __device__ __forceinline__ bool table_only() const { return cpv_p0::kTableOnly && P.tables; }
    __device__ __forceinline__ uint32_t table_lookup(const CpvTri& t, uint32_t texel) const {
        return cpv_p0::cpv_table_lookup(P.tables, __float_as_uint(t.var[1][0]), texel);
    }
    __device__ __forceinline__ void load_linear(uint64_t pix, float d[4]) const { cpv_p0::cpv_load_linear(P.color, pix, P.clear, d); }
    __device__ __forceinline__ void store_linear(uint64_t pix, const float d[4]) const { cpv_p0::cpv_store_linear(P.color, pix, d); }
    __device__ __forceinline__ void load_pixel(uint64_t pix, CpvPixel& s) const { cpv_p0::Stage::load_pixel(P.color, P.depth, pix, s, P.color_extra, P.clear); }
    __device__ __forceinline__ void store_pixel(uint64_t pix, const CpvPixel& s) const {
        cpv_p0::Stage::store_pixel(P.color, P.depth, pix, s, P.color_extra, P.clear);
    }
    __device__ __forceinline__ void clear_pixel(uint64_t pix) const { cpv_p0::Stage::clear_pixel(P.color, P.depth, pix, P.clear); }
};

/* Raster kernel: one CTA per screen tile (blockIdx.x = tile id). Without
 * rectangles the tile walks every primitive of the draw (small draws), else
 * what its bin list (or all rectangles) holds for it. Dynamic shared memory:
 * CPV_RASTER_SMEM_BYTES. */
#if CPV_LINEAR_BLEND
/* the linear-blend loop runs best at five resident CTAs per SM (2.10 ms,
 * 2.19 at four, 2.13 at six) */
#ifndef CPV_LINEAR_MIN_BLOCKS
#define CPV_LINEAR_MIN_BLOCKS 5
#endif
#define CPV_PLAIN_BOUNDS __launch_bounds__(CPV_RT_THREADS, CPV_LINEAR_MIN_BLOCKS)
#elif defined(CPV_PLAIN_MIN_BLOCKS)
/* a register budget for CPV_PLAIN_MIN_BLOCKS resident CTAs per SM */
#define CPV_PLAIN_BOUNDS __launch_bounds__(CPV_RT_THREADS, CPV_PLAIN_MIN_BLOCKS)
#else
#define CPV_PLAIN_BOUNDS __launch_bounds__(CPV_RT_THREADS)
#endif
extern "C" __global__ void CPV_PLAIN_BOUNDS cpv_raster(const __grid_constant__ CpvDrawParams P) {
    extern __shared__ float4 cpv_dyn_smem[];
    __shared__ uint32_t warp_sums[CPV_RT_THREADS / 32];
    __shared__ CpvTileList list;
    const uint32_t tile = blockIdx.x;
    const uint32_t tx = tile % P.tiles_x, ty = tile / P.tiles_x;
    CpvPlainSource src{P, list, P.viewport[2], P.viewport[3], P.fb_width, P.fb_height};
    uint32_t first = static_cast<uint32_t>(P.total_prims);
    if (!P.rects && first <= CPV_BATCH) {
        /* every primitive in one batch: the ring is full and nothing follows */
        if (threadIdx.x < first) list.ring[threadIdx.x] = threadIdx.x;
        for (uint32_t i = CPV_RT_THREADS + threadIdx.x; i < first; i += CPV_RT_THREADS) list.ring[i] = i;
        if (threadIdx.x == 0u) {
            list.head = list.pos = list.end = 0u;
            list.waiting = list.taken = first;
        }
    } else {
        if (threadIdx.x == 0u) {
            list.head = list.waiting = list.taken = 0u;
            uint2 range = make_uint2(0u, first);
            const bool by_list = P.bin_counts && *P.pair_total <= P.list_capacity;
            if (by_list) range = P.bin_range[(ty >> P.bin_shift) * P.bins_x + (tx >> P.bin_shift)];
            list.by_list = by_list ? 1u : 0u;
            list.pos = range.x;
            list.end = range.y;
        }
        __syncthreads();
        first = src.next(warp_sums);
        if (first == 0u) {
            if (P.clear.mask) cpv_clear_tile(src, tx, ty);
            return;
        }
    }
    cpv_raster_tile(src, first, tx, ty, reinterpret_cast<CpvTri*>(cpv_dyn_smem), warp_sums);
}

#endif /* CPV_PIPELINE_CUH */

/* Launch shape of the raster kernel, read by the host at module load
 * (cudaLibraryGetGlobal): dynamic shared memory bytes and threads per CTA. */
extern "C" __device__ const uint32_t cpv_raster_smem_bytes = CPV_RASTER_SMEM_BYTES;
extern "C" __device__ const uint32_t cpv_raster_threads = CPV_RT_THREADS;
