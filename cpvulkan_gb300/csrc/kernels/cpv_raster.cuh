/*
 * cpv_raster.cuh — the pipeline-independent part of the tile rasteriser,
 * shared by the per-draw module (cpv_pipeline.cuh) and the batched module
 * (cpv_batch.cuh). Compiled by NVRTC after cpv_device.cuh; the module prefix
 * defines CPV_TILE_SHIFT, CPV_SCHEDULE, CPV_RT_WARPS, CPV_BATCH and
 * CPV_NV_MAX (the largest varying count over the module's pipelines).
 *
 * The per-pipeline part (primitive set-up, fragment shading and the
 * per-fragment operations, which depend on the pipeline's shaders and
 * fixed-function state) is cpv_stage.cuh, instantiated once per pipeline in
 * its own namespace. cpv_raster_tile() walks one screen tile's primitives
 * through a Source object that supplies the primitives in API order and
 * routes each to its pipeline's stage functions.
 */
#ifndef CPV_RASTER_CUH
#define CPV_RASTER_CUH

#ifndef CPV_TILE_SHIFT
#define CPV_TILE_SHIFT 4
#endif
#ifndef CPV_SCHEDULE
#define CPV_SCHEDULE 0 /* 0 immediate, 1 deferred, 2 sparse (see cpv_raster_tile) */
#endif
#define CPV_DEFERRED (CPV_SCHEDULE == 1)
#if CPV_DEFERRED && CPV_NUM_CA > 1
#error "the deferred schedule keeps one colour per recorded fragment: modules with several colour attachments use another"
#endif
#define CPV_SPARSE (CPV_SCHEDULE == 2)
#define CPV_WARP_LISTS (CPV_SCHEDULE == 0) /* immediate: each warp walks only the primitives reaching its rows */
#ifndef CPV_SLOT_DEPTH
#define CPV_SLOT_DEPTH 16 /* sparse: fragments a pixel takes per batch before its fallback */
#endif
#ifndef CPV_SMALL_PX
#define CPV_SMALL_PX 64 /* sparse: largest in-tile bounding box listed by the warp-spread tests (C4 raster 21.37 ms at 64, 21.65 at 32, 21.86 at 128) */
#endif
#ifndef CPV_DENSE
/* sparse: large primitives' pixels per tile pixel from which a batch runs the
 * immediate schedule: every pixel's thread walks the whole batch in order,
 * testing boxes (sparse modules have no per-warp lists), and shades what
 * covers it. A pixel whose list overflows walks the batch as well, but after
 * the listing, and its warp waits for it. 6k smooth quads at 1280x720 take 420
 * us without this rule, 273 at 2 to 8, 275 at 16, 289 at 24, 355 at 32; 300
 * half-float triangles 416, 322, 328, 340 and 386. By the boxes instead of the
 * triangles' areas, slivers count too much (180k triangles at 1366x767: 95 us,
 * 150 at 8 by boxes). Batched modules mix their draws' small and large
 * primitives in a batch, where the lists are better for longer
 * (compose_module: 32): 512 draws at 2560x1440 take 2436 us without it, 2878
 * at 8, 2588 at 16, 2485 at 24, 2437 at 32. */
#define CPV_DENSE 8
#endif
#ifndef CPV_RT_WARPS
#define CPV_RT_WARPS 8
#endif
#ifndef CPV_BATCH
#define CPV_BATCH 128
#endif
#ifndef CPV_ANY_FS_CONSTANT
#define CPV_ANY_FS_CONSTANT 0 /* some pipeline of the module shades once per primitive */
#endif
#ifndef CPV_LINEAR_BLEND
#define CPV_LINEAR_BLEND 0 /* the module's pipeline blends a constant colour linearly (cpv_linear_blend) and does nothing else */
#endif
#ifndef CPV_QUICK_DIV
#define CPV_QUICK_DIV 0 /* fragments divide by reciprocals prepared at set-up */
#endif
#define CPV_TILE (1 << CPV_TILE_SHIFT)
#define CPV_RT_THREADS ((CPV_TILE * CPV_TILE) < (32 * CPV_RT_WARPS) ? (CPV_TILE * CPV_TILE) : (32 * CPV_RT_WARPS))
#define CPV_PPT ((CPV_TILE * CPV_TILE) / CPV_RT_THREADS)
/* register budget of the persistent batched raster: 32 resident warps per
 * SM (64 registers a thread) */
#ifndef CPV_RT_MIN_BLOCKS
#define CPV_RT_MIN_BLOCKS (1024 / CPV_RT_THREADS)
#endif

#define CPV_ROWS_PER_PASS (CPV_RT_THREADS / CPV_TILE)
#define CPV_WARP_ROWS (32 / CPV_TILE > 0 ? 32 / CPV_TILE : 1) /* tile rows one warp covers per pass */
/* immediate schedule with one pixel a thread: each warp owns an 8 x 4 block
 * of the tile instead of whole rows (a compact block is more often wholly
 * inside or outside a primitive, so fewer visits cover few lanes) */
#define CPV_WARP_BLOCKS (CPV_WARP_LISTS && CPV_PPT == 1 && CPV_TILE >= 8)
#define CPV_BLOCK_W 8
#define CPV_BLOCK_H 4
#ifndef CPV_ANY_LINES
#define CPV_ANY_LINES 0 /* some pipeline of the module draws lines */
#endif
#ifndef CPV_NUM_CA
#define CPV_NUM_CA 1 /* colour attachments of the module's subpass (up to 8; 1 also for a depth-only pass) */
#endif
/* fragment shader outputs: 4 floats per colour attachment */
#define CPV_COLOUR_FLOATS (4 * CPV_NUM_CA)
#define CPV_NV_ALLOC (CPV_NV_MAX > 0 ? CPV_NV_MAX : 1)
#define CPV_NV_ROOM0 (CPV_ANY_FS_CONSTANT && CPV_NV_ALLOC < 4 ? 4 : CPV_NV_ALLOC)
#define CPV_NV_ROOM (CPV_ANY_LINES && CPV_NV_ROOM0 < 7 ? 7 : CPV_NV_ROOM0)
#define CPV_NV_PAD ((CPV_NV_ROOM + 3) & ~3)
#define CPV_SLOTS 4
#define CPV_NSLOT (CPV_RT_THREADS * CPV_SLOTS)

/* One primitive after set-up, in the reference's terms
 * (CPVulkan/CommandBuffer.Draw.cpp:1510-1594, 874-954). 16-byte aligned
 * groups so that the coverage loop reads them with 128-bit loads.
 *
 * Points and lines reuse the record (Draw.cpp:1315-1508):
 *   point — its box is exactly the set of pixels the reference covers and the
 *           edges are zero (every pixel of the box passes); za.x = NDC z,
 *           wf.x = clip w, var[0] = the vertex's outputs;
 *   line  — e[0..2] and za are the four edges of the line's quad, wf.x/y
 *           the two clip w, var[0..1] the vertices' outputs, var[2][0..6] =
 *           p0.x, p0.y, (p1 - p0).x, (p1 - p0).y, |p1 - p0|², z0, z1; the
 *           provoking slot field holds 3 (a line's provoking vertex is its
 *           first). */
struct __align__(16) CpvTri {
    float4 e[3];     /* edge k: start vertex (x, y) and b - a (dx, dy), NDC */
    float4 za;       /* NDC z of p0..p2 (after the CW swap), |area| */
    float4 wf;       /* clip w of p0..p2, flags (see below) */
#if CPV_QUICK_DIV
    float4 rc;       /* triangles: 1 / wf.xyz and 1 / area, correctly rounded; w = 0: divide (cpv_tri_reciprocals) */
#endif
    float var[3][CPV_NV_PAD]; /* varyings per vertex; for a pipeline whose fragment
                                 shader is constant per primitive, var[0][0..3]
                                 holds the shaded colour instead */
#if (CPV_QUICK_DIV + 3 * CPV_NV_PAD / 4) % 2 == 1
    /* an odd number of 16-byte units: 8 lanes that read a unit each of 8
     * records then use all 32 banks once (the 500k-triangle request's raster
     * 196 us at 12 units, 168 at 11; the 512-draw pass's 4.25 ms at 8 units,
     * 3.0 at 9) */
    float4 pad;
#endif
};

/* A primitive's pixel bounding box within its tile, one byte each: x0, y0,
 * x1 | 0x80, y1 | 0x80 (ends exclusive). The high bits make the subtraction of
 * cpv_in_box borrow-free; a dead primitive has the empty box. */
#define CPV_BOX_DEAD 0x80800000u
__device__ __forceinline__ uint32_t cpv_box_pack(int32_t x0, int32_t y0, int32_t x1, int32_t y1) {
    return static_cast<uint32_t>(x0) | (static_cast<uint32_t>(y0) << 8) | (static_cast<uint32_t>(x1) << 16) | (static_cast<uint32_t>(y1) << 24) | CPV_BOX_DEAD;
}
__device__ __forceinline__ int32_t cpv_box_x0(uint32_t b) { return static_cast<int32_t>(b & 0xFFu); }
__device__ __forceinline__ int32_t cpv_box_y0(uint32_t b) { return static_cast<int32_t>((b >> 8) & 0xFFu); }
__device__ __forceinline__ int32_t cpv_box_x1(uint32_t b) { return static_cast<int32_t>((b >> 16) & 0x7Fu); }
__device__ __forceinline__ int32_t cpv_box_y1(uint32_t b) { return static_cast<int32_t>((b >> 24) & 0x7Fu); }
/* A pixel of the tile as cpv_in_box takes it. */
__device__ __forceinline__ uint32_t cpv_box_pixel(uint32_t lx, uint32_t ly) { return (lx | 0x80u) | ((ly | 0x80u) << 8) | ((lx + 1u) << 16) | ((ly + 1u) << 24); }
/* x0 <= lx, y0 <= ly, lx + 1 <= x1 and ly + 1 <= y1, a byte each. */
__device__ __forceinline__ bool cpv_in_box(uint32_t box, uint32_t pixel) {
    const uint32_t hi = __byte_perm(pixel, box, 0x7610), lo = __byte_perm(box, pixel, 0x7610);
    return ((hi - lo) & 0x80808080u) == 0x80808080u;
}

/* Flag word (wf.w bits): 1 live, 2 front facing, bits 2-5 pipeline index in
 * the module, bits 6-7 provoking-vertex slot (3: a line), bits 8-31 draw
 * index in the batch (0 for a per-draw module). */
__device__ __forceinline__ uint32_t cpv_tri_flags(const CpvTri& t) { return __float_as_uint(t.wf.w); }
__device__ __forceinline__ bool cpv_tri_live(const CpvTri& t) { return (cpv_tri_flags(t) & 1u) != 0u; }
__device__ __forceinline__ bool cpv_tri_front(const CpvTri& t) { return (cpv_tri_flags(t) & 2u) != 0u; }
__device__ __forceinline__ uint32_t cpv_tri_pipeline(const CpvTri& t) { return (cpv_tri_flags(t) >> 2) & 15u; }
__device__ __forceinline__ uint32_t cpv_tri_pslot(const CpvTri& t) { return (cpv_tri_flags(t) >> 6) & 3u; }
__device__ __forceinline__ uint32_t cpv_tri_draw(const CpvTri& t) { return cpv_tri_flags(t) >> 8; }
__device__ __forceinline__ void cpv_tri_tag(CpvTri& t, uint32_t pipeline, uint32_t draw) {
    t.wf.w = __uint_as_float((cpv_tri_flags(t) & 0xC3u) | (pipeline << 2) | (draw << 8));
}

/* Pixel centre in NDC (CPVulkan/CommandBuffer.Draw.cpp:1524, 1573-1580):
 * (x / width + halfPixel) * 2 - 1, halfPixel = (1 / width) * 0.5. */
__device__ __forceinline__ float cpv_pixel_ndc(int32_t x, float extent) {
    const float half = __fmul_rn(__fdiv_rn(1.0f, extent), 0.5f);
    return __fsub_rn(__fmul_rn(__fadd_rn(__fdiv_rn(static_cast<float>(x), extent), half), 2.0f), 1.0f);
}

/* Edge functions at a pixel centre (CPVulkan/CommandBuffer.Draw.cpp:882-902):
 * w_k = (p.x - a.x) * (b.y - a.y) - (p.y - a.y) * (b.x - a.x); covered when
 * no w_k is negative (inclusive on every edge). */
__device__ __forceinline__ bool cpv_covers(const CpvTri& t, float xf, float yf, float w[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float4 e = t.e[k];
        const float t0 = __fmul_rn(__fsub_rn(xf, e.x), e.w);
        const float t1 = __fmul_rn(__fsub_rn(yf, e.y), e.z);
        w[k] = __fsub_rn(t0, t1);
    }
#if CPV_ANY_LINES
    /* a line's quad has a fourth edge (CPVulkan/CommandBuffer.Draw.cpp:1437):
     * every edge must be >= 0, which also rejects NaN */
    if (((__float_as_uint(t.wf.w) >> 6) & 3u) == 3u) {
        const float4 e = t.za;
        const float w3 = __fsub_rn(__fmul_rn(__fsub_rn(xf, e.x), e.w), __fmul_rn(__fsub_rn(yf, e.y), e.z));
        return w[0] >= 0.0f && w[1] >= 0.0f && w[2] >= 0.0f && w3 >= 0.0f;
    }
#endif
    return !(w[0] < 0.0f || w[1] < 0.0f || w[2] < 0.0f);
}

/* The same without the values. A rounded difference is negative where its
 * first operand is the smaller and nowhere else (equal or NaN operands give 0
 * or NaN, also for infinities), so a triangle's products are compared and not
 * subtracted. */
__device__ __forceinline__ bool cpv_covers_pixel(const CpvTri& t, float xf, float yf) {
#if CPV_ANY_LINES
    float w[3];
    return cpv_covers(t, xf, yf, w);
#else
    bool out = false;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float4 e = t.e[k];
        out = out | (__fmul_rn(__fsub_rn(xf, e.x), e.w) < __fmul_rn(__fsub_rn(yf, e.y), e.z));
    }
    return !out;
#endif
}

/* Whether a primitive covers any pixel centre of a box of at most four by
 * four pixels (cpv_covers): every column and row of the first three by
 * three, a smaller box's repeated, so that no loop's trips differ between
 * lanes; the rest where the box is larger and none is covered yet. Products
 * are compared as in cpv_covers_pixel. Pixel centres come from the tables
 * when given (the box lies inside the attachment). */
__device__ __forceinline__ bool cpv_covers_any(const CpvTri& t, int4 b, float vw, float vh, const float* ndc_x, const float* ndc_y) {
    auto column = [&](int32_t i) {
        const int32_t x = min(b.x + i, b.z - 1);
        return ndc_x ? __ldg(ndc_x + x) : cpv_pixel_ndc(x, vw);
    };
    auto row = [&](int32_t i) {
        const int32_t y = min(b.y + i, b.w - 1);
        return ndc_y ? __ldg(ndc_y + y) : cpv_pixel_ndc(y, vh);
    };
    bool any = false;
#if CPV_ANY_LINES
    if (((__float_as_uint(t.wf.w) >> 6) & 3u) == 3u) {
        for (int32_t i = 0; i < 16; i++) {
            float w[3];
            any = cpv_covers(t, column(i & 3), row(i >> 2), w) || any;
        }
        return any;
    }
#endif
    float tx[4][3];
    auto set_column = [&](int32_t c) {
        const float xf = column(c);
#pragma unroll
        for (int k = 0; k < 3; k++) tx[c][k] = __fmul_rn(__fsub_rn(xf, t.e[k].x), t.e[k].w);
    };
    auto test_row = [&](int32_t r, int32_t c0, int32_t c1) {
        const float yf = row(r);
        float ty[3];
#pragma unroll
        for (int k = 0; k < 3; k++) ty[k] = __fmul_rn(__fsub_rn(yf, t.e[k].y), t.e[k].z);
#pragma unroll
        for (int32_t c = 0; c < 4; c++)
            if (c >= c0 && c < c1) any = any | !((tx[c][0] < ty[0]) | (tx[c][1] < ty[1]) | (tx[c][2] < ty[2]));
    };
#pragma unroll
    for (int32_t c = 0; c < 3; c++) set_column(c);
#pragma unroll
    for (int32_t r = 0; r < 3; r++) test_row(r, 0, 3);
    if (!any && (b.z - b.x > 3 || b.w - b.y > 3)) {
        set_column(3);
#pragma unroll
        for (int32_t r = 0; r < 3; r++) test_row(r, 3, 4);
        test_row(3, 0, 4);
    }
    return any;
}

/* Tile rectangle of a set-up primitive with pixel box b (empty when culled, off screen, or
 * when none of the pixel centres of a box of at most four by four is covered
 * — the raster would find no fragment there either). Packed as
 * x0 | y0 << 16, x1 | y1 << 16 in tile units, end exclusive. */
__device__ __forceinline__ uint2 cpv_tile_rect(const CpvTri& t, int4 b, float vw, float vh, const float* ndc_x = nullptr, const float* ndc_y = nullptr) {
    uint32_t r[4] = {0, 0, 0, 0};
    if (cpv_tri_live(t)) {
        bool any = true;
        if (b.z - b.x <= 4 && b.w - b.y <= 4) any = cpv_covers_any(t, b, vw, vh, ndc_x, ndc_y);
        if (any) {
            r[0] = static_cast<uint32_t>(b.x >> CPV_TILE_SHIFT);
            r[1] = static_cast<uint32_t>(b.y >> CPV_TILE_SHIFT);
            r[2] = static_cast<uint32_t>(((b.z - 1) >> CPV_TILE_SHIFT) + 1);
            r[3] = static_cast<uint32_t>(((b.w - 1) >> CPV_TILE_SHIFT) + 1);
        }
    }
    return make_uint2(r[0] | (r[1] << 16), r[2] | (r[3] << 16));
}

/* Whether primitive t may cover a pixel of the rectangle [rx0, rx1) x
 * [ry0, ry1) (inside its box). Each rounded edge function
 * w = fl(fl(xf - a.x) * dy) - fl(fl(yf - a.y) * dx) is monotonic along a
 * row and along a column (the pixel-centre values are monotonic in the
 * pixel index, and IEEE subtraction and multiplication by a fixed value are
 * monotonic), so its largest value over the rectangle is at the corner
 * picked by the signs of dy and dx; if that value is negative, every pixel
 * of the rectangle fails the edge and none is covered. Exact: it only
 * drops pixels the coverage test rejects. Edges with a non-finite
 * coefficient keep the primitive (NaN counts as covered). The rectangle is
 * relative to the tile; col/row hold the tile's pixel-centre NDC values. */
__device__ __forceinline__ bool cpv_may_cover(const CpvTri& t, int32_t rx0, int32_t ry0, int32_t rx1, int32_t ry1, const float* col,
                                              const float* row) {
    /* the pixel-centre sequences are monotonic (in either direction for a
     * negative extent): their extremes over a range are its ends */
    const float c0 = col[rx0], c1 = col[rx1 - 1];
    const float r0 = row[ry0], r1 = row[ry1 - 1];
    const float xa = fminf(c0, c1), xb = fmaxf(c0, c1), ya = fminf(r0, r1), yb = fmaxf(r0, r1);
    if (!(fabsf(c0) <= 3.4e38f && fabsf(c1) <= 3.4e38f && fabsf(r0) <= 3.4e38f && fabsf(r1) <= 3.4e38f)) return true;
    bool may = true;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float4 e;
        if (k < 3) {
            e = t.e[k];
        } else {
#if CPV_ANY_LINES
            if (((__float_as_uint(t.wf.w) >> 6) & 3u) != 3u) break;
            e = t.za; /* a line's fourth edge */
#else
            break;
#endif
        }
        if (!(fabsf(e.x) <= 3.4e38f && fabsf(e.y) <= 3.4e38f && fabsf(e.z) <= 3.4e38f && fabsf(e.w) <= 3.4e38f)) continue;
        const float xf = e.w > 0.0f ? xb : xa;
        const float yf = e.z > 0.0f ? ya : yb;
        const float w = __fsub_rn(__fmul_rn(__fsub_rn(xf, e.x), e.w), __fmul_rn(__fsub_rn(yf, e.y), e.z));
        may = may && !(w < 0.0f);
    }
    return may;
}

/* Whether cpv_block_edges may be asked: every coefficient of the triangle's
 * edges is finite (a line has a fourth edge and is tested pixel by pixel). */
__device__ __forceinline__ bool cpv_edges_finite(const CpvTri& t) {
#if CPV_ANY_LINES
    if (((__float_as_uint(t.wf.w) >> 6) & 3u) == 3u) return false;
#endif
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float4 e = t.e[k];
        finite = finite && fmaxf(fmaxf(fabsf(e.x), fabsf(e.y)), fmaxf(fabsf(e.z), fabsf(e.w))) <= 3.4e38f && e.x == e.x && e.y == e.y && e.z == e.z && e.w == e.w;
    }
    return finite;
}

/* A triangle's edges over the rectangle of pixel centres [xa, xb] x [ya, yb]
 * (finite, in either order): bit 3 when an edge is negative at every pixel
 * (none is covered), else bit k for each edge that some pixel may fail. By
 * the monotonicity cpv_may_cover uses, an edge function
 * (xf - a.x) * dy - (yf - a.y) * dx has its extremes at the products' extremes,
 * and its rounded difference is negative exactly when the one is less than
 * the other. */
__device__ __forceinline__ uint32_t cpv_block_edges(const CpvTri& t, float xa, float xb, float ya, float yb) {
    uint32_t open = 0u;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float4 e = t.e[k];
        const float p0 = __fmul_rn(__fsub_rn(xa, e.x), e.w), p1 = __fmul_rn(__fsub_rn(xb, e.x), e.w);
        const float q0 = __fmul_rn(__fsub_rn(ya, e.y), e.z), q1 = __fmul_rn(__fsub_rn(yb, e.y), e.z);
        if (fmaxf(p0, p1) < fminf(q0, q1)) open |= 8u;
        if (fminf(p0, p1) < fmaxf(q0, q1)) open |= 1u << k;
    }
    return open;
}

/* ---- per-fragment operation helpers (LLVMRuntime/PipelineCompiler.cpp:1020-1429) ---- */

__device__ __forceinline__ bool cpv_fcompare(float a, float b, uint32_t op) {
    switch (op) {
    case 0: return false;
    case 1: return a < b;
    case 2: return a == b;
    case 3: return a <= b;
    case 4: return a > b;
    case 5: return (a < b) || (a > b);
    case 6: return a >= b;
    default: return true;
    }
}

__device__ __forceinline__ bool cpv_icompare(uint32_t a, uint32_t b, uint32_t op) {
    switch (op) {
    case 0: return false;
    case 1: return a < b;
    case 2: return a == b;
    case 3: return a <= b;
    case 4: return a > b;
    case 5: return a != b;
    case 6: return a >= b;
    default: return true;
    }
}

/* Stencil ops; increment/decrement-and-clamp saturate as signed i8
 * (LLVMRuntime/PipelineCompiler.cpp:1382-1413). */
__device__ __forceinline__ uint32_t cpv_stencil_op(uint32_t op, uint32_t cur, uint32_t ref) {
    const int32_t sc = static_cast<int8_t>(cur);
    switch (op) {
    case 0: return cur;
    case 1: return 0u;
    case 2: return ref & 0xFFu;
    case 3: return static_cast<uint32_t>(static_cast<uint8_t>(sc == 127 ? 127 : sc + 1));
    case 4: return static_cast<uint32_t>(static_cast<uint8_t>(sc == -128 ? -128 : sc - 1));
    case 5: return (~cur) & 0xFFu;
    case 6: return (cur + 1u) & 0xFFu;
    case 7: return (cur - 1u) & 0xFFu;
    default: return cur;
    }
}

/* ApplyBlendFactor / ApplyBlend (CPVulkan/CommandBuffer.Draw.cpp:956-1262). */
__device__ __forceinline__ void cpv_blend_factor(const float s[4], const float d[4], const float c[4], uint32_t cf, uint32_t af, float o[4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = 0.0f;
    switch (cf) {
    case 0: break;
    case 1: for (int i = 0; i < 4; i++) o[i] = 1.0f; break;
    case 2: for (int i = 0; i < 4; i++) o[i] = s[i]; break;
    case 3: for (int i = 0; i < 4; i++) o[i] = __fsub_rn(1.0f, s[i]); break;
    case 4: for (int i = 0; i < 4; i++) o[i] = d[i]; break;
    case 5: for (int i = 0; i < 4; i++) o[i] = __fsub_rn(1.0f, d[i]); break;
    case 6: for (int i = 0; i < 4; i++) o[i] = s[3]; break;
    case 7: { const float v = __fsub_rn(1.0f, s[3]); for (int i = 0; i < 4; i++) o[i] = v; break; }
    case 8: for (int i = 0; i < 4; i++) o[i] = d[3]; break;
    case 9: { const float v = __fsub_rn(1.0f, d[3]); for (int i = 0; i < 4; i++) o[i] = v; break; }
    case 10: for (int i = 0; i < 4; i++) o[i] = c[i]; break;
    case 11: for (int i = 0; i < 4; i++) o[i] = __fsub_rn(1.0f, c[i]); break;
    case 12: for (int i = 0; i < 4; i++) o[i] = c[3]; break;
    case 13: { const float v = __fsub_rn(1.0f, c[3]); for (int i = 0; i < 4; i++) o[i] = v; break; }
    case 14: { const float f = cpv_std_min(s[3], __fsub_rn(1.0f, d[3])); o[0] = f; o[1] = f; o[2] = f; o[3] = 1.0f; break; }
    default: break;
    }
    if (cf != af) {
        switch (af) {
        case 0: o[3] = 0.0f; break;
        case 1: case 14: o[3] = 1.0f; break;
        case 2: case 6: o[3] = s[3]; break;
        case 3: case 7: o[3] = __fsub_rn(1.0f, s[3]); break;
        case 4: case 8: o[3] = d[3]; break;
        case 5: case 9: o[3] = __fsub_rn(1.0f, d[3]); break;
        case 10: case 12: o[3] = c[3]; break;
        case 11: case 13: o[3] = __fsub_rn(1.0f, c[3]); break;
        default: break;
        }
    }
}

__device__ __forceinline__ float cpv_blend_op(float s, float sf, float d, float df, uint32_t op) {
    const float a = __fmul_rn(s, sf);
    const float b = __fmul_rn(d, df);
    switch (op) {
    case 0: return __fadd_rn(a, b);
    case 1: return __fsub_rn(a, b);
    case 2: return __fsub_rn(b, a);
    case 3: return cpv_std_min(s, d);
    case 4: return cpv_std_max(s, d);
    default: return 0.0f;
    }
}

/* Two binary32 values in a 64-bit register, and the packed operations on
 * them: each lane is rounded as the scalar operation rounds it. */
struct CpvPair {
    unsigned long long v;
};
__device__ __forceinline__ CpvPair cpv_pair(float a, float b) {
    CpvPair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void cpv_unpair(CpvPair p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v)); }
__device__ __forceinline__ CpvPair cpv_mul2(CpvPair a, CpvPair b) {
    CpvPair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ CpvPair cpv_add2(CpvPair a, CpvPair b) {
    CpvPair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ CpvPair cpv_add2_rz(CpvPair a, CpvPair b) {
    CpvPair r;
    asm("add.rz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ CpvPair cpv_fma2(CpvPair a, CpvPair b, CpvPair c) {
    CpvPair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

/* The 8-bit UNORM channels that a + d * f encodes to, decoded again, for two
 * channels: the blend of a colour that is constant over a primitive, for
 * destination channels d with factors that do not read the destination (a:
 * source times its factor, f: the destination's factor, signs as the blend
 * operation has them). The reference's steps: multiply, add, clamp (NaN →
 * 0), times 255, round half away from zero — floor(x + 0.5), both additions
 * rounded toward zero — and over 255 as cpv_decode_unorm8. */
__device__ __forceinline__ CpvPair cpv_linear_blend(CpvPair d, CpvPair a, CpvPair f) {
    float a0, a1, p0, p1;
    cpv_unpair(a, a0, a1);
    cpv_unpair(cpv_mul2(d, f), p0, p1);
    const CpvPair x = cpv_mul2(cpv_pair(__saturatef(__fadd_rn(a0, p0)), __saturatef(__fadd_rn(a1, p1))), cpv_pair(255.0f, 255.0f));
    const CpvPair n = cpv_add2(cpv_add2_rz(cpv_add2_rz(x, cpv_pair(0.5f, 0.5f)), cpv_pair(8388608.0f, 8388608.0f)), cpv_pair(-8388608.0f, -8388608.0f));
    return cpv_fma2(n, cpv_pair(0x1.010102p-8f, 0x1.010102p-8f), cpv_mul2(n, cpv_pair(-0x1.fdfdfep-33f, -0x1.fdfdfep-33f)));
}

/* Register-resident attachment state of one pixel. */
#ifndef CPV_COLOUR_WORDS
#define CPV_COLOUR_WORDS 1 /* 32-bit words of the module's widest first-attachment texel (8- and 16-byte formats: 2, 4) */
#endif
struct CpvPixel {
    uint32_t colour[CPV_COLOUR_WORDS];
    float depth;        /* decoded depth (D16: u16 / 65535) */
    uint32_t depth_raw; /* stored bits */
    uint32_t stencil;
#if CPV_NUM_CA > 1
    uint32_t extra[CPV_NUM_CA - 1]; /* texels of colour attachments 1 .. */
#endif
};

/* Block-wide exclusive sum over CPV_RT_THREADS threads. */
__device__ __forceinline__ uint32_t cpv_block_scan(uint32_t v, uint32_t& total, uint32_t* warp_sums) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= static_cast<uint32_t>(o)) incl += t;
    }
    if (lane == 31u) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t base = 0, sum = 0;
    for (uint32_t k = 0; k < CPV_RT_THREADS / 32; k++) {
        const uint32_t s = warp_sums[k];
        if (k < warp) base += s;
        sum += s;
    }
    total = sum;
    return base + incl - v;
}

/* Sparse schedule: class of a primitive in the tile by its box — 0 dead or
 * outside the tile, 1 small (at most CPV_SMALL_PX pixels of the tile), 2
 * large. */
__device__ __forceinline__ uint32_t cpv_tile_class(uint32_t box) {
    const int32_t px = (cpv_box_x1(box) - cpv_box_x0(box)) * (cpv_box_y1(box) - cpv_box_y0(box));
    return px == 0 ? 0u : (px > CPV_SMALL_PX ? 2u : 1u);
}

/* Sparse schedule: the small primitives j0 .. j0 + 31 of a batch (one per
 * lane of the calling warp) test the pixels of their boxes inside the tile
 * and append each covered pixel's primitive to its list — as one list of
 * (primitive, pixel) tests spread evenly over the warp's lanes, so that a
 * lane's large box does not hold the other 31 lanes. The primitives are put
 * in the first lanes, in order; test i belongs to the last of them that
 * starts at or before i — of those that start within the step, by the bits
 * that they set at their starts — and is pixel i - (its start) of its box,
 * row-major. Issue-bound: a binary search over the lanes' sums, four shuffles
 * and differences instead of comparisons a test made the rasters of 500k
 * triangles at 2048x2048 164 us (155 now), of 2 M at 1920x1080 170 (164), of
 * 64 draws at 640x360 149 (139), of 512 at 2560x1440 2593 (2472). A pixel's
 * list is applied in batch order whatever the order of its appends. */
__device__ __forceinline__ void cpv_list_small_warp(const CpvTri* tris, const uint32_t* boxes, uint32_t j0, uint32_t n, const float* col_ndc,
                                                     const float* row_ndc, uint32_t* list_count, uint8_t* list_j) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t own_box = j0 + lane < n ? boxes[j0 + lane] : CPV_BOX_DEAD;
    const uint32_t small = __ballot_sync(0xFFFFFFFFu, cpv_tile_class(own_box) == 1u);
    const uint32_t prims = __popc(small);
    /* the lane of the lane-th small primitive */
    uint32_t from = 0u;
#pragma unroll
    for (uint32_t s = 16u; s > 0u; s >>= 1)
        if (__popc(small & ((1u << (from + s)) - 1u)) <= lane) from += s;
    const uint32_t box = __shfl_sync(0xFFFFFFFFu, own_box, from);
    const uint32_t bw = static_cast<uint32_t>(cpv_box_x1(box) - cpv_box_x0(box));
    const uint32_t size = lane < prims ? bw * static_cast<uint32_t>(cpv_box_y1(box) - cpv_box_y0(box)) : 0u;
    uint32_t incl = size;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= static_cast<uint32_t>(o)) incl += t;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    const uint32_t start = incl - size;
    /* start (up to 31 * 1024), lane; x0, y0, width and the width's reciprocal.
     * row = (k * magic) >> 16 = floor(k / bw) for every k < 1024 and bw <= 32:
     * magic = ceil(2^16 / bw) exceeds 2^16 / bw by less than 1, so the product
     * exceeds k * 2^16 / bw by less than k < 2^16 / 64, under the 2^16 / bw gap
     * from a non-integer k / bw to the next integer. A width of 1 is stored
     * with magic 0 and its pixels are column 0 of row k. */
    const uint32_t pack0 = start | (from << 16) | (static_cast<uint32_t>(cpv_box_x0(box)) << 21) | (static_cast<uint32_t>(cpv_box_y0(box)) << 26);
    const uint32_t pack1 = lane < prims && bw > 1u ? ((65536u + bw - 1u) / bw) | (bw << 16) : 1u << 16;
    uint32_t before = 0u;  /* primitives that start before the step */
    for (uint32_t base = 0; base < total; base += 32u) {
        const uint32_t i = base + lane, at = start - base;
        const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, size != 0u && at < 32u ? 1u << at : 0u);
        const uint32_t owner = before + __popc(starts & (0xFFFFFFFFu >> (31u - lane))) - 1u;
        before += __popc(starts);
        const uint32_t o0 = __shfl_sync(0xFFFFFFFFu, pack0, owner), o1 = __shfl_sync(0xFFFFFFFFu, pack1, owner);
        if (i >= total) continue;
        const uint32_t k = i - (o0 & 0xFFFFu), w = o1 >> 16;
        const uint32_t row = w == 1u ? k : (k * (o1 & 0xFFFFu)) >> 16;
        const uint32_t lx = ((o0 >> 21) & 31u) + k - row * w, ly = (o0 >> 26) + row;
        const uint32_t j = j0 + ((o0 >> 16) & 31u);
        if (!cpv_covers_pixel(tris[j], col_ndc[lx], row_ndc[ly])) continue;
        const uint32_t p = ly * CPV_TILE + lx;
        const uint32_t s = atomicAdd(&list_count[p], 1u);
        if (s < CPV_SLOT_DEPTH) list_j[p * CPV_SLOT_DEPTH + s] = static_cast<uint8_t>(j);
    }
}

/* Dynamic shared memory of the raster kernels: CPV_BATCH primitives and
 * their boxes in the tile, then the schedule's buffers (deferred: fragment slots; sparse: per-pixel
 * primitive lists, pixel-centre tables, the large-primitive list). */
#define CPV_TILE_PX (CPV_TILE * CPV_TILE)
#define CPV_SPARSE_BYTES (4u * CPV_TILE_PX + CPV_TILE_PX * CPV_SLOT_DEPTH + CPV_BATCH)
#define CPV_RASTER_SMEM_BYTES \
    (CPV_BATCH * (sizeof(CpvTri) + 4u) + (CPV_DEFERRED ? CPV_NSLOT * (4u + 20u + 2u) : 0u) + (CPV_SPARSE ? CPV_SPARSE_BYTES : 0u))

/* A tile without primitives under a pending clear (CpvClear). */
template <class Source>
__device__ __forceinline__ void cpv_clear_tile(const Source& src, uint32_t tx, uint32_t ty) {
    for (uint32_t i = threadIdx.x; i < CPV_TILE_PX; i += CPV_RT_THREADS) {
        const uint32_t x = tx * CPV_TILE + i % CPV_TILE, y = ty * CPV_TILE + i / CPV_TILE;
        if (x < src.fb_width && y < src.fb_height) src.clear_pixel(static_cast<uint64_t>(y) * src.fb_width + x);
    }
}

/* One screen tile (tx, ty) whose first batch holds `first` > 0 primitives:
 * loads the tile's attachment texels into registers, walks the tile's
 * primitives from `src` in API order in batches of CPV_BATCH (set-up into shared memory, then coverage, shading and the
 * per-fragment operations of each pixel in primitive order) and stores the
 * texels back once.
 *
 * Source supplies:
 *   uint32_t next(uint32_t* warp_sums)       the size of the tile's next batch (up to CPV_BATCH; 0: done)
 *   void setup(uint32_t i, CpvTri& t, int4& box)  set up the batch's i-th primitive and its pixel box (or mark it dead)
 *   bool shade(const CpvTri&, const float w[3], int x, int y, float colour[CPV_COLOUR_FLOATS], float& mapped, const CpvPixel* early)
 *                                            (true: discarded, or failed the early depth
 *                                            test against *early when given)
 *   void rop(const CpvTri&, const float colour[CPV_COLOUR_FLOATS], float mapped, CpvPixel&)
 *   bool table_only()                        a covered fragment is a blend-table lookup alone:
 *   uint32_t table_lookup(const CpvTri&, uint32_t texel)  the texel after it
 *   void load_pixel(uint64_t pix, CpvPixel&) / store_pixel(uint64_t pix, const CpvPixel&)
 *                                            (the load gives the pending clear's texel, if there is one)
 *   void clear_pixel(uint64_t pix)           writes the pending clear
 *   float vw, vh                             viewport extent (pixel centres)
 *   uint32_t fb_width, fb_height
 *
 * Three fragment schedules (CPV_SCHEDULE):
 *   0 immediate — each pixel's thread tests every primitive of the batch and
 *               shades its covered fragments as it finds them (cheap
 *               shaders, large primitives);
 *   1 deferred — per batch of primitives, threads first record up to
 *               CPV_SLOTS covered fragments each, the CTA then shades all
 *               recorded fragments densely (full warps, whatever the
 *               coverage pattern), and finally every pixel's thread applies
 *               its own fragments' per-fragment operations in primitive
 *               order (expensive shaders);
 *   2 sparse  — coverage is found per primitive instead of per pixel: the
 *               primitives whose bounding boxes cover at most CPV_SMALL_PX
 *               pixels of the tile are rasterised by warps, 32 primitives'
 *               pixels spread over the lanes; larger ones are tested by the
 *               pixels' threads. Either appends the primitive's batch index
 *               to each covered pixel's list (up to CPV_SLOT_DEPTH per
 *               batch); each pixel's thread then shades and applies its list
 *               in primitive order (tiny primitives, heavy overdraw). A pixel
 *               whose list overflowed walks the whole batch instead, and a
 *               batch dense in large primitives (CPV_DENSE) runs the
 *               immediate schedule.
 * All apply each pixel's fragments in API primitive order, as the
 * reference's serial loop does. */
template <class Source>
__device__ __forceinline__ void cpv_raster_tile(Source& src, uint32_t first, uint32_t tx, uint32_t ty, CpvTri* tris, uint32_t* warp_sums) {
    /* pixel-centre NDC of the tile's columns and rows (the values of
     * cpv_pixel_ndc); the barrier keeps the previous tile's readers of a
     * persistent CTA ahead of the rewrite */
    __shared__ float col_ndc[CPV_TILE], row_ndc[CPV_TILE];
    const int32_t tile_x0 = static_cast<int32_t>(tx * CPV_TILE), tile_y0 = static_cast<int32_t>(ty * CPV_TILE);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < CPV_TILE; i += CPV_RT_THREADS) {
        col_ndc[i] = cpv_pixel_ndc(tile_x0 + static_cast<int32_t>(i), src.vw);
        row_ndc[i] = cpv_pixel_ndc(tile_y0 + static_cast<int32_t>(i), src.vh);
    }
    uint32_t* boxes = reinterpret_cast<uint32_t*>(tris + CPV_BATCH);  /* per primitive: its box in the tile */
    int32_t px[CPV_PPT], py[CPV_PPT];
    uint32_t bp[CPV_PPT];  /* the pixel as cpv_in_box takes it */
    float xf[CPV_PPT], yf[CPV_PPT];
    bool inside[CPV_PPT];
    CpvPixel st[CPV_PPT];
#pragma unroll
    for (int k = 0; k < CPV_PPT; k++) {
#if CPV_WARP_BLOCKS
        /* warp w: block (w % blocks a row, w / blocks a row); lane: x = lane % 8, y = lane / 8 */
        const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
        px[k] = static_cast<int32_t>(tx * CPV_TILE + (warp % (CPV_TILE / CPV_BLOCK_W)) * CPV_BLOCK_W + (lane % CPV_BLOCK_W));
        py[k] = static_cast<int32_t>(ty * CPV_TILE + (warp / (CPV_TILE / CPV_BLOCK_W)) * CPV_BLOCK_H + (lane / CPV_BLOCK_W));
#else
        px[k] = static_cast<int32_t>(tx * CPV_TILE + (threadIdx.x % CPV_TILE));
        py[k] = static_cast<int32_t>(ty * CPV_TILE + (threadIdx.x / CPV_TILE) + k * CPV_ROWS_PER_PASS);
#endif
        bp[k] = cpv_box_pixel(static_cast<uint32_t>(px[k] - tile_x0), static_cast<uint32_t>(py[k] - tile_y0));
        inside[k] = px[k] < static_cast<int32_t>(src.fb_width) && py[k] < static_cast<int32_t>(src.fb_height);
        xf[k] = cpv_pixel_ndc(px[k], src.vw);
        yf[k] = cpv_pixel_ndc(py[k], src.vh);
#if !CPV_LINEAR_BLEND
        if (inside[k]) src.load_pixel(static_cast<uint64_t>(py[k]) * src.fb_width + px[k], st[k]);
#endif
    }
#if CPV_LINEAR_BLEND
    static_assert(CPV_WARP_BLOCKS, "a linear-blend module runs the immediate schedule with one pixel a thread");
    float lin[4] = {0.0f, 0.0f, 0.0f, 0.0f};  /* the pixel's decoded colour */
    if (inside[0]) src.load_linear(static_cast<uint64_t>(py[0]) * src.fb_width + px[0], lin);
    CpvPair lin01 = cpv_pair(lin[0], lin[1]), lin23 = cpv_pair(lin[2], lin[3]);
#endif

#if CPV_DEFERRED
    uint8_t* slot_base = reinterpret_cast<uint8_t*>(boxes + CPV_BATCH);
    uint32_t* slot_jk = reinterpret_cast<uint32_t*>(slot_base);          /* batch index | pixel k << 8 | discard << 31 */
    float* slot_f = reinterpret_cast<float*>(slot_jk + CPV_NSLOT);       /* 5 floats per slot: w0 w1 w2 → rgba + mapped */
    uint16_t* dense = reinterpret_cast<uint16_t*>(slot_f + 5 * CPV_NSLOT);
#endif
#if CPV_SPARSE
    static_assert(CPV_BATCH <= 256, "batch indices are stored in bytes");
    uint32_t* list_count = boxes + CPV_BATCH;  /* per tile pixel: fragments listed this batch */
    uint8_t* list_j = reinterpret_cast<uint8_t*>(list_count + CPV_TILE_PX);  /* per tile pixel: CPV_SLOT_DEPTH batch indices */
    uint8_t* large = list_j + CPV_TILE_PX * CPV_SLOT_DEPTH;                  /* batch indices of large primitives */
    __shared__ uint32_t large_count[2];  /* of this batch and the next, by turns: their number (at most 256), and from bit 9 their pixels */
    if (threadIdx.x == 0u) large_count[0] = 0u;
    uint32_t turn = 0u;
    for (uint32_t i = threadIdx.x; i < CPV_TILE_PX; i += CPV_RT_THREADS) list_count[i] = 0u;
    uint32_t lp[CPV_PPT]; /* this thread's pixels, as tile pixel indices */
#pragma unroll
    for (int k = 0; k < CPV_PPT; k++) lp[k] = static_cast<uint32_t>((py[k] - tile_y0) * CPV_TILE + (px[k] - tile_x0));
#endif

#if CPV_WARP_LISTS
    /* immediate schedule: per warp, the batch's primitives reaching its rows
     * (batch index; for a warp's block bits 8-10: the edges its pixels have to
     * test, bit 11: the box, too; none set: the whole block is covered) */
    static_assert(CPV_BATCH <= 256, "batch indices take 8 bits");
    __shared__ uint16_t warp_list[(CPV_RT_THREADS / 32) * CPV_BATCH];
#if CPV_WARP_BLOCKS
    __shared__ uint16_t live_flags[CPV_BATCH], live_list[CPV_BATCH];
    /* every pixel centre of the tile is finite (their sequences are monotonic) */
    const bool centres_finite = fabsf(cpv_pixel_ndc(tile_x0, src.vw)) <= 3.4e38f && fabsf(cpv_pixel_ndc(tile_x0 + CPV_TILE - 1, src.vw)) <= 3.4e38f &&
                                fabsf(cpv_pixel_ndc(tile_y0, src.vh)) <= 3.4e38f && fabsf(cpv_pixel_ndc(tile_y0 + CPV_TILE - 1, src.vh)) <= 3.4e38f;
    const int32_t warp_x0 = static_cast<int32_t>(((threadIdx.x >> 5) % (CPV_TILE / CPV_BLOCK_W)) * CPV_BLOCK_W);
    const int32_t warp_y0 = static_cast<int32_t>(((threadIdx.x >> 5) / (CPV_TILE / CPV_BLOCK_W)) * CPV_BLOCK_H);
#else
    const int32_t warp_y0 = static_cast<int32_t>((threadIdx.x & ~31u) / CPV_TILE);
#endif
#endif

    for (uint32_t n = first; n != 0u; n = src.next(warp_sums)) {
        __syncthreads();
#if CPV_SPARSE
        if (threadIdx.x == 0u) large_count[turn ^ 1u] = 0u;
#endif
        /* a tile of 8 × 8 has fewer threads than CPV_BATCH: stride the set-up;
         * a primitive reaching beyond the tile that covers no pixel of it
         * (its box ∩ the tile) is dropped for this tile; one inside the tile
         * is left to the pixel tests, which is cheaper for small primitives */
        for (uint32_t i = threadIdx.x; i < n; i += CPV_RT_THREADS) {
            CpvTri& t = tris[i];
            int4 b = make_int4(0, 0, 0, 0);
            src.setup(i, t, b);
            const int32_t rx0 = max(b.x - tile_x0, 0), ry0 = max(b.y - tile_y0, 0);
            const int32_t rx1 = min(b.z - tile_x0, CPV_TILE), ry1 = min(b.w - tile_y0, CPV_TILE);
            bool live = cpv_tri_live(t) && rx1 > rx0 && ry1 > ry0;
            /* worth a test when the primitive spans much of the tile */
            if (live && (b.x < tile_x0 || b.y < tile_y0 || b.z > tile_x0 + CPV_TILE || b.w > tile_y0 + CPV_TILE) &&
                (rx1 - rx0) * (ry1 - ry0) >= CPV_TILE_PX / 8)
                live = cpv_may_cover(t, rx0, ry0, rx1, ry1, col_ndc, row_ndc);
            boxes[i] = live ? cpv_box_pack(rx0, ry0, rx1, ry1) : CPV_BOX_DEAD;
#if CPV_SPARSE
            /* 1. large primitives (box covering more than CPV_SMALL_PX pixels
             *    of the tile) are collected, in any order (by a block scan and
             *    three barriers after the set-up: rasters 2 to 4% longer), and
             *    the pixels they may cover summed: the triangle's area, if
             *    that is less than the box's (an estimate that only chooses
             *    the schedule; NaN counts as none) */
            if (cpv_tile_class(boxes[i]) == 2u) {
                const float px = fminf(fmaxf(t.za.w * (src.vw * src.vh * 0.125f), 0.0f), static_cast<float>((rx1 - rx0) * (ry1 - ry0)));
                large[atomicAdd(&large_count[turn], 1u + (static_cast<uint32_t>(px) << 9)) & 0x1FFu] = static_cast<uint8_t>(i);
            }
#endif
#if CPV_WARP_BLOCKS
            live_flags[i] = live ? (0x100u | (centres_finite && cpv_edges_finite(t) ? 1u : 0u)) : 0u;
#endif
        }
        __syncthreads();
#if CPV_WARP_BLOCKS
        /* the batch's live primitives in order (index; bit 8: cpv_block_edges
         * applies): each warp compacts the whole batch's flags for itself up
         * to its 32, then writes those (half of a large triangle's tiles hold
         * none of it, so half the primitives of a batch are dead) */
        uint32_t alive = 0u;
        for (uint32_t b = 0; b < n; b += 32u) {
            const uint32_t i = b + (threadIdx.x & 31u);
            const uint32_t flags = i < n ? live_flags[i] : 0u;
            const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, flags != 0u);
            if (flags != 0u && (b >> 5) % (CPV_RT_THREADS / 32) == (threadIdx.x >> 5))
                live_list[alive + __popc(ballot & ((1u << (threadIdx.x & 31u)) - 1u))] = static_cast<uint16_t>(i | ((flags & 1u) << 8));
            alive += __popc(ballot);
        }
        __syncthreads();
#endif
#if CPV_SPARSE
        const uint32_t nlarge = large_count[turn] & 0x1FFu, large_px = large_count[turn] >> 9;
        turn ^= 1u;
        /* mostly large primitives, or enough of them over each pixel that its
         * list may overflow: this batch runs the immediate schedule */
        const bool immediate_batch = nlarge * 4u >= 3u * n || large_px >= CPV_DENSE * static_cast<uint32_t>(CPV_TILE_PX);
        if (!immediate_batch) {
            /* 2. small primitives: each warp lists the pixels its 32 cover */
            for (uint32_t j0 = threadIdx.x & ~31u; j0 < n; j0 += CPV_RT_THREADS)
                cpv_list_small_warp(tris, boxes, j0, n, col_ndc, row_ndc, list_count, list_j);
            /* 3. large primitives: every pixel's thread tests its pixels */
            for (uint32_t m = 0; m < nlarge; m++) {
                const uint32_t j = large[m];
                const CpvTri& t = tris[j];
                const uint32_t box = boxes[j];
#pragma unroll
                for (int k = 0; k < CPV_PPT; k++) {
                    if (!cpv_in_box(box, bp[k]) || !cpv_covers_pixel(t, xf[k], yf[k])) continue;
                    const uint32_t s = atomicAdd(&list_count[lp[k]], 1u);
                    if (s < CPV_SLOT_DEPTH) list_j[lp[k] * CPV_SLOT_DEPTH + s] = static_cast<uint8_t>(j);
                }
            }
            __syncthreads();
            /* 4. each pixel shades and applies its list in batch (API) order */
#pragma unroll
            for (int k = 0; k < CPV_PPT; k++) {
                const uint32_t c = list_count[lp[k]];
                if (c == 0u) continue;
                if (c <= CPV_SLOT_DEPTH) {
                    const uint8_t* lj = list_j + lp[k] * CPV_SLOT_DEPTH;
                    int32_t last = -1;
                    for (uint32_t it = 0; it < c; it++) {
                        /* next batch index after `last` (a primitive covers a pixel once) */
                        int32_t j = lj[0];
                        if (c > 1u) {
                            j = 0x7FFFFFFF;
                            for (uint32_t e = 0; e < c; e++) {
                                const int32_t v = lj[e];
                                if (v > last && v < j) j = v;
                            }
                            last = j;
                        }
                        const CpvTri& t = tris[j];
                        float w[3], colour[CPV_COLOUR_FLOATS], mapped;
                        cpv_covers(t, xf[k], yf[k], w);
                        if (src.shade(t, w, px[k], py[k], colour, mapped, &st[k])) continue;
                        src.rop(t, colour, mapped, st[k]);
                    }
                } else {
                    /* list overflow: walk the whole batch for this pixel */
                    for (uint32_t j = 0; j < n; j++) {
                        if (!cpv_in_box(boxes[j], bp[k])) continue;
                        const CpvTri& t = tris[j];
                        float w[3], colour[CPV_COLOUR_FLOATS], mapped;
                        if (!cpv_covers(t, xf[k], yf[k], w)) continue;
                        if (src.shade(t, w, px[k], py[k], colour, mapped, &st[k])) continue;
                        src.rop(t, colour, mapped, st[k]);
                    }
                }
                list_count[lp[k]] = 0u;
            }
        }
#else
        const bool immediate_batch = true;
        (void)immediate_batch;
#endif
#if !CPV_DEFERRED
        /* immediate: every pixel's thread tests each primitive in order,
         * shading and applying what it covers. In modules of the immediate
         * schedule each warp first lists, in order, the batch's live
         * primitives that may reach its pixels, and walks only those; a dense
         * batch of a sparse module walks all. */
        if (immediate_batch) {
#if CPV_WARP_LISTS
            const uint32_t lane = threadIdx.x & 31u;
            uint16_t* mine = warp_list + (threadIdx.x >> 5) * CPV_BATCH;
            uint32_t count = 0;
#if CPV_WARP_BLOCKS
            for (uint32_t b = 0; b < alive; b += 32u) {
                bool hit = false;
                uint32_t entry = 0u;
                if (b + lane < alive) {
                    entry = live_list[b + lane];
                    const uint32_t j = entry & 0xFFu;
                    const uint32_t box = boxes[j];
                    /* the warp's block, within the box */
                    const int32_t rx0 = max(cpv_box_x0(box), warp_x0), rx1 = min(cpv_box_x1(box), warp_x0 + CPV_BLOCK_W);
                    const int32_t ry0 = max(cpv_box_y0(box), warp_y0), ry1 = min(cpv_box_y1(box), warp_y0 + CPV_BLOCK_H);
                    if (rx1 > rx0 && ry1 > ry0) {
                        /* of a block inside the box (so inside the attachment) only the open edges are left to test */
                        const bool in_box = rx0 == warp_x0 && rx1 == warp_x0 + CPV_BLOCK_W && ry0 == warp_y0 && ry1 == warp_y0 + CPV_BLOCK_H;
                        uint32_t open = 7u;
                        if (entry & 0x100u) open = cpv_block_edges(tris[j], col_ndc[rx0], col_ndc[rx1 - 1], row_ndc[ry0], row_ndc[ry1 - 1]);
                        hit = open < 8u;
                        entry = j | (open << 8) | (in_box ? 0u : 0x800u);
                    }
                }
                const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, hit);
                if (hit) mine[count + __popc(ballot & ((1u << lane) - 1u))] = static_cast<uint16_t>(entry);
                count += __popc(ballot);
            }
#else
            for (uint32_t b = 0; b < n; b += 32u) {
                const uint32_t j = b + lane;
                bool hit = false;
                if (j < n) {
                    const CpvTri& t = tris[j];
                    const uint32_t box = boxes[j];  /* a dead primitive's is empty */
                    const int32_t rx0 = cpv_box_x0(box), rx1 = cpv_box_x1(box);
#pragma unroll
                    for (int k = 0; k < CPV_PPT; k++) {
                        /* the warp's rows of pass k, within the box */
                        const int32_t ry0 = max(cpv_box_y0(box), warp_y0 + k * CPV_ROWS_PER_PASS);
                        const int32_t ry1 = min(cpv_box_y1(box), warp_y0 + k * CPV_ROWS_PER_PASS + CPV_WARP_ROWS);
                        hit = hit || (ry1 > ry0 && cpv_may_cover(t, rx0, ry0, rx1, ry1, col_ndc, row_ndc));
                    }
                }
                const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, hit);
                if (hit) mine[count + __popc(ballot & ((1u << lane) - 1u))] = static_cast<uint16_t>(j);
                count += __popc(ballot);
            }
#endif
            __syncwarp();
#else
            const uint32_t count = n;
#endif
#if CPV_WARP_BLOCKS && (CPV_LINEAR_BLEND || CPV_ANY_FS_CONSTANT)
            /* The entry's tests for this thread's pixel. */
            auto passes = [&](uint32_t entry, const CpvTri& t) {
                bool covered = true;
                if (entry & 0x800u) covered = cpv_in_box(boxes[entry & 0xFFu], bp[0]);
#if CPV_ANY_LINES
                float w[3];
                if (entry & 0x700u) covered = cpv_covers(t, xf[0], yf[0], w) && covered;
#else
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    if (entry & (0x100u << k)) {
                        const float4 e = t.e[k];
                        /* the rounded difference is negative exactly when the one is less */
                        covered = covered && !(__fmul_rn(__fsub_rn(xf[0], e.x), e.w) < __fmul_rn(__fsub_rn(yf[0], e.y), e.z));
                    }
                }
#endif
                return covered;
            };
#endif
#if CPV_LINEAR_BLEND
            /* The blend of a constant colour as two constants per channel
             * (cpv_shade_constant): eight binary32 operations a channel on the
             * decoded colour, two channels an instruction, and nothing else in
             * the loop. Issue-bound: the 200k-quad scene at 1920x1080 takes 2.10
             * ms of raster (2.38 with scalar operations; with blend tables
             * 2.51, and 0.12 to build them), 1.3 of it in this loop, 0.4 in
             * set-up and filter, the rest in the lists and their barriers. */
            for (uint32_t m = 0; m < count; m++) {
                const uint32_t entry = mine[m];
                const CpvTri& t = tris[entry & 0xFFu];
                if (entry > 0xFFu && !passes(entry, t)) continue;
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(t.var[0]), f = *reinterpret_cast<const ulonglong2*>(t.var[1]);
                lin01 = cpv_linear_blend(lin01, CpvPair{a.x}, CpvPair{f.x});
                lin23 = cpv_linear_blend(lin23, CpvPair{a.y}, CpvPair{f.y});
            }
#else
#if CPV_WARP_BLOCKS && CPV_ANY_FS_CONSTANT
            /* A pipeline whose covered fragments are a blend-table lookup each:
             * a loop of its own, so that the general one's registers do not
             * spill it (a byte permute makes each lookup's address). */
            if (src.table_only()) {
                uint32_t texel = st[0].colour[0];
                for (uint32_t m = 0; m < count; m++) {
                    const uint32_t entry = mine[m];
                    const CpvTri& t = tris[entry & 0xFFu];
                    if (entry > 0xFFu && !passes(entry, t)) continue;
                    texel = src.table_lookup(t, texel);
                }
                st[0].colour[0] = texel;
                continue;
            }
#endif
            for (uint32_t m = 0; m < count; m++) {
#if CPV_WARP_LISTS
                const uint32_t entry = mine[m];
                const uint32_t j = entry & 0xFFu;
#if CPV_WARP_BLOCKS
                if (entry <= 0xFFu) {
                    /* the whole block is covered (one pixel a thread, all inside) */
                    const CpvTri& t = tris[j];
                    float w[3], colour[CPV_COLOUR_FLOATS], mapped;
                    cpv_covers(t, xf[0], yf[0], w);
                    if (src.shade(t, w, px[0], py[0], colour, mapped, &st[0])) continue;
                    src.rop(t, colour, mapped, st[0]);
                    continue;
                }
#endif
#else
                const uint32_t j = m;
#endif
                const CpvTri& t = tris[j];
                const uint32_t box = boxes[j];
#pragma unroll
                for (int k = 0; k < CPV_PPT; k++) {
                    if (!cpv_in_box(box, bp[k])) continue;
                    float w[3];
                    if (!cpv_covers(t, xf[k], yf[k], w)) continue;
                    float colour[CPV_COLOUR_FLOATS], mapped;
                    if (src.shade(t, w, px[k], py[k], colour, mapped, &st[k])) continue;
                    src.rop(t, colour, mapped, st[k]);
                }
            }
#endif
        }
#else
        const uint32_t limit = n * CPV_PPT;
        uint32_t cursor = 0;
        while (__syncthreads_or(cursor < limit)) {
            /* 1. coverage: record up to CPV_SLOTS fragments, in primitive order */
            uint32_t cnt = 0;
            while (cursor < limit && cnt < CPV_SLOTS) {
                const uint32_t j = cursor / CPV_PPT, k = cursor - j * CPV_PPT;
                cursor++;
                const CpvTri& t = tris[j];
                uint32_t bpk = bp[0];
                float xfk = xf[0], yfk = yf[0];
#pragma unroll
                for (int kk = 1; kk < CPV_PPT; kk++)
                    if (k == static_cast<uint32_t>(kk)) { bpk = bp[kk]; xfk = xf[kk]; yfk = yf[kk]; }
                if (!cpv_in_box(boxes[j], bpk)) continue;
                float w[3];
                if (!cpv_covers(t, xfk, yfk, w)) continue;
                const uint32_t s = threadIdx.x * CPV_SLOTS + cnt;
                slot_jk[s] = j | (k << 8);
                slot_f[5 * s + 0] = w[0];
                slot_f[5 * s + 1] = w[1];
                slot_f[5 * s + 2] = w[2];
                cnt++;
            }
            /* 2. dense shading of every recorded fragment */
            uint32_t total;
            const uint32_t pos = cpv_block_scan(cnt, total, warp_sums);
            for (uint32_t i = 0; i < cnt; i++) dense[pos + i] = static_cast<uint16_t>(threadIdx.x * CPV_SLOTS + i);
            __syncthreads();
            for (uint32_t d = threadIdx.x; d < total; d += CPV_RT_THREADS) {
                const uint32_t s = dense[d];
                const uint32_t owner = s / CPV_SLOTS;
                const uint32_t jk = slot_jk[s];
                const uint32_t j = jk & 0xFFu, k = (jk >> 8) & 0xFFu;
                const int32_t x = static_cast<int32_t>(tx * CPV_TILE + (owner % CPV_TILE));
                const int32_t y = static_cast<int32_t>(ty * CPV_TILE + (owner / CPV_TILE) + k * CPV_ROWS_PER_PASS);
                const float w[3] = {slot_f[5 * s + 0], slot_f[5 * s + 1], slot_f[5 * s + 2]};
                float colour[CPV_COLOUR_FLOATS], mapped;
                const bool discard = src.shade(tris[j], w, x, y, colour, mapped);
                slot_f[5 * s + 0] = colour[0];
                slot_f[5 * s + 1] = colour[1];
                slot_f[5 * s + 2] = colour[2];
                slot_f[5 * s + 3] = colour[3];
                slot_f[5 * s + 4] = mapped;
                if (discard) slot_jk[s] = jk | 0x80000000u;
            }
            __syncthreads();
            /* 3. per-fragment operations of this thread's pixels, in order */
            for (uint32_t i = 0; i < cnt; i++) {
                const uint32_t s = threadIdx.x * CPV_SLOTS + i;
                const uint32_t jk = slot_jk[s];
                if (jk >> 31) continue;
                const uint32_t j = jk & 0xFFu, k = (jk >> 8) & 0xFFu;
                const float colour[4] = {slot_f[5 * s + 0], slot_f[5 * s + 1], slot_f[5 * s + 2], slot_f[5 * s + 3]};
#pragma unroll
                for (int kk = 0; kk < CPV_PPT; kk++)
                    if (k == static_cast<uint32_t>(kk)) src.rop(tris[j], colour, slot_f[5 * s + 4], st[kk]);
            }
        }
#endif
    }
#if CPV_LINEAR_BLEND
    cpv_unpair(lin01, lin[0], lin[1]);
    cpv_unpair(lin23, lin[2], lin[3]);
    if (inside[0]) src.store_linear(static_cast<uint64_t>(py[0]) * src.fb_width + px[0], lin);
    return;
#endif
#pragma unroll
    for (int k = 0; k < CPV_PPT; k++) {
        if (inside[k]) src.store_pixel(static_cast<uint64_t>(py[k]) * src.fb_width + px[k], st[k]);
    }
}

#endif /* CPV_RASTER_CUH */
