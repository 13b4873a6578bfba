// bm_device.cuh -- device code shared by the single-pair kernels (bm_kernels.cu)
// and the batched kernels (bm_batch.cu): per-pixel and per-block bodies of every
// stage, so both launch paths run the same arithmetic.  Included only by units
// compiled with -use_fast_math (the reference's flags, CMakeLists.txt:50).
#pragma once

#include <curand_kernel.h>
#include <type_traits>

#include "bm_internal.h"

namespace bmk {
namespace dev {

// util_cuda.h:61
#define BM_PI 3.141592653589793115997963468544

constexpr int TX = 32;  // block width: one warp per row of a tile
constexpr int TY = 8;   // block height

__device__ __forceinline__ int lo16(uint32_t w) { return (int)(int16_t)(w & 0xffffu); }
__device__ __forceinline__ int hi16(uint32_t w) { return (int)(int16_t)(w >> 16); }

template <int NSP>
__device__ __forceinline__ void store_desc(uint32_t* dst, const uint32_t (&w)[NSP])
{
    if constexpr (NSP >= 4) {
#pragma unroll
        for (int k = 0; k < NSP / 4; k++)
            reinterpret_cast<uint4*>(dst)[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
    } else if constexpr (NSP == 2) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    } else {
        dst[0] = w[0];
    }
}

template <int NSP, bool L2 = false>
__device__ __forceinline__ void load_desc(uint32_t (&w)[NSP], const uint32_t* src)
{
    if constexpr (NSP >= 4) {
#pragma unroll
        for (int k = 0; k < NSP / 4; k++) {
            uint4 v = L2 ? __ldcg(reinterpret_cast<const uint4*>(src) + k) : __ldg(reinterpret_cast<const uint4*>(src) + k);
            w[4 * k] = v.x;
            w[4 * k + 1] = v.y;
            w[4 * k + 2] = v.z;
            w[4 * k + 3] = v.w;
        }
    } else if constexpr (NSP == 2) {
        uint2 v = L2 ? __ldcg(reinterpret_cast<const uint2*>(src)) : __ldg(reinterpret_cast<const uint2*>(src));
        w[0] = v.x;
        w[1] = v.y;
    } else {
        w[0] = L2 ? __ldcg(src) : __ldg(src);
    }
}

template <int NSP, bool L2 = false>
__device__ __forceinline__ int hamming(const uint32_t (&a)[NSP], const uint32_t* pb)
{
    uint32_t b[NSP];
    load_desc<NSP, L2>(b, pb);
    int h = 0;
#pragma unroll
    for (int k = 0; k < NSP; k++) h += __popc(a[k] ^ b[k]);
    return h;
}

__device__ __forceinline__ void rs_normals(const RsArgs& rs, unsigned int id, float& n1, float& n2)
{
    if (rs.mode == BM_RNG_PHILOX) {
        curandStatePhilox4_32_10_t st;
        curand_init(rs.seed, (unsigned long long)id, 2ull * rs.call, &st);
        float2 v = curand_normal2(&st);
        n1 = v.x;
        n2 = v.y;
    } else {
        // The reference state: curand_init(id, 0, 0) (briefmatch_cuda.cu:57) advanced by
        // two uniforms per earlier call (two curand_normal per call, :240-241).  Each
        // branch has a state of its own: skipahead takes its state's address, which
        // would keep a shared one in local memory through every step of the loop.
        const unsigned long long skip = 2ull * rs.call;
        if (skip <= 512ull) {
            curandStateXORWOW_t st;
            curand_init((unsigned long long)id, 0ull, 0ull, &st);
            for (unsigned int k = 0; k < (unsigned int)skip; k++) (void)curand(&st);
            n1 = curand_normal(&st);
            n2 = curand_normal(&st);
        } else {
            curandStateXORWOW_t st;
            curand_init((unsigned long long)id, 0ull, 0ull, &st);
            skipahead(skip, &st);
            n1 = curand_normal(&st);
            n2 = curand_normal(&st);
        }
    }
}

// Descriptor loads for the own pixel: read once per level and never again, so
// they are marked evict-first to leave L2 to the gathered descriptors.
template <int NSP>
__device__ __forceinline__ void load_desc_stream(uint32_t (&w)[NSP], const uint32_t* __restrict__ src)
{
    if constexpr (NSP >= 4) {
#pragma unroll
        for (int k = 0; k < NSP / 4; k++) {
            uint4 v = __ldcs(reinterpret_cast<const uint4*>(src) + k);
            w[4 * k] = v.x;
            w[4 * k + 1] = v.y;
            w[4 * k + 2] = v.z;
            w[4 * k + 3] = v.w;
        }
    } else if constexpr (NSP == 2) {
        uint2 v = __ldcs(reinterpret_cast<const uint2*>(src));
        w[0] = v.x;
        w[1] = v.y;
    } else {
        w[0] = __ldcs(src);
    }
}

// Descriptor gather that is issued only when `pred` holds (the words stay zero
// otherwise); written as predicated PTX loads so that several gathers of one
// thread are in flight together instead of waiting behind each other's branches.
template <int NSP>
__device__ __forceinline__ void gather_desc_pred(uint32_t (&w)[NSP], const uint32_t* __restrict__ src, bool pred)
{
    const int pr = pred ? 1 : 0;
#pragma unroll
    for (int k = 0; k < NSP; k++) w[k] = 0;
    if constexpr (NSP >= 4) {
#pragma unroll
        for (int k = 0; k < NSP / 4; k++)
            asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t@p ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%5];\n\t}"
                : "+r"(w[4 * k]), "+r"(w[4 * k + 1]), "+r"(w[4 * k + 2]), "+r"(w[4 * k + 3])
                : "r"(pr), "l"(src + 4 * k));
    } else if constexpr (NSP == 2) {
        asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.global.nc.v2.u32 {%0, %1}, [%3];\n\t}"
            : "+r"(w[0]), "+r"(w[1])
            : "r"(pr), "l"(src));
    } else {
        asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\t@p ld.global.nc.u32 %0, [%2];\n\t}"
            : "+r"(w[0])
            : "r"(pr), "l"(src));
    }
}

typedef unsigned long long f2x;  // two packed floats (low = first)

__device__ __forceinline__ f2x pk2(float a, float b) { f2x r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float lo2(f2x v) { return __uint_as_float((unsigned int)(v & 0xffffffffull)); }
__device__ __forceinline__ float hi2(f2x v) { return __uint_as_float((unsigned int)(v >> 32)); }
__device__ __forceinline__ f2x add2(f2x a, f2x b) { f2x d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2x mul2(f2x a, f2x b) { f2x d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2x fma2(f2x a, f2x b, f2x c)
{
    f2x d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}


// ---------------------------------------------------------------------------
// Lanczos-3 up-sampling (util_cuda.cu:126-158): output pixel (x, y).  The weights
// are tabulated per output column/row with the reference's expression; the 6x6
// accumulation runs in the reference's order (i outer, j inner).
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float upsample_val(const T* __restrict__ in, int sxi, int syi,
                                              const float* __restrict__ lx, const int* __restrict__ ix,
                                              const float* __restrict__ ly, const int* __restrict__ iy, int x, int y)
{
    int x1 = ix[x], y1 = iy[y];
    float Ly[6];
    int row[6];
#pragma unroll
    for (int b = 0; b < 6; b++) {
        Ly[b] = ly[y * 6 + b];
        row[b] = min(syi - 1, max(0, y1 - 2 + b)) * sxi;
    }
    float v = 0.0f, w = 0.0f;
#pragma unroll
    for (int a = 0; a < 6; a++) {
        float Lx = lx[x * 6 + a];
        int ci = min(sxi - 1, max(0, x1 - 2 + a));
#pragma unroll
        for (int b = 0; b < 6; b++) {
            w += Lx * Ly[b];
            v += float(in[ci + row[b]]) * Lx * Ly[b];
        }
    }
    return v / w;
}

template <typename T>
__device__ __forceinline__ void upsample_px(const T* __restrict__ in, float* __restrict__ out, int sxi, int syi,
                                            int sxo, const float* __restrict__ lx, const int* __restrict__ ix,
                                            const float* __restrict__ ly, const int* __restrict__ iy, int x, int y)
{
    out[x + (size_t)y * sxo] = upsample_val<T>(in, sxi, syi, lx, ix, ly, iy, x, y);
}

// ---------------------------------------------------------------------------
// 16-bit keys of image samples: a monotone map of the float value to a half-precision
// bit pattern, so that keys compare two at a time; different keys order as their floats
// do, equal keys leave the order open.  The 63487 finite halves from -0x7bff to 0x7bff
// cover 128 +- 158.7 grey levels (Lanczos overshoot included) in steps of 1/200;
// values beyond share the end keys.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t sample_key(float v)
{
    const int i = __float2int_rn(fminf(fmaxf(__fmaf_rn(v, 200.0f, -25600.0f), -31743.0f), 31743.0f));
    return i < 0 ? 0x8000u | (uint32_t)(-i) : (uint32_t)i;
}
// 1.0 or 0.0 per half
__device__ __forceinline__ uint32_t half2_gt(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("set.gt.f16x2.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t half2_eq(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("set.eq.f16x2.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// 2 * acc + bit per half
__device__ __forceinline__ uint32_t half2_shift_in(uint32_t acc, uint32_t bit)
{
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(acc), "r"(0x40004000u), "r"(bit));
    return r;
}
// Four accumulators that hold 1024 + byte in each half (0x6400 | byte): the words of the
// low and of the high halves' bytes.
__device__ __forceinline__ void half2_bytes(const uint32_t (&a)[4], uint32_t& lo, uint32_t& hi)
{
    const uint32_t p = __byte_perm(a[0], a[1], 0x6240), q = __byte_perm(a[2], a[3], 0x6240);
    lo = __byte_perm(p, q, 0x5410);
    hi = __byte_perm(p, q, 0x7632);
}

// ---------------------------------------------------------------------------
// BRIEF descriptors (briefmatch_cuda.cu:82-124).
// Interior pixels (at least rmax from every border, rmax = the largest |offset|)
// read the image at the precomputed linear offsets `off` with no clamping -- the
// reference's clamped reads give the same addresses there; samples past N carry
// offset 0 and give 0 bits.  Border pixels clamp each coordinate as the reference.
// A warp reads 32 consecutive pixels at one offset: one coalesced L1 request.
// ---------------------------------------------------------------------------
template <int NSP, typename OffArray>
__device__ __forceinline__ void features_interior_px(const float* __restrict__ I, uint32_t* __restrict__ F, int sx,
                                                     int x, int y, const OffArray& off)
{
    const float* base = I + (size_t)y * sx + x;
    uint32_t word[NSP];
#pragma unroll
    for (int wd = 0; wd < NSP; wd++) {
        uint32_t acc = 0;
#pragma unroll
        for (int b = 0; b < 32; b++) {
            const int2 o = off[wd * 32 + b];
            const float i1 = __ldg(base + o.x);
            const float i2 = __ldg(base + o.y);
            if (i1 > i2) acc |= 1u << b;
        }
        word[wd] = acc;
    }
    store_desc<NSP>(F + ((size_t)y * sx + x) * NSP, word);
}

template <int NSP>
__device__ __forceinline__ void features_border_px(const float* __restrict__ I, uint32_t* __restrict__ F, int sx,
                                                   int sy, int N, const int4* __restrict__ s_pat, int x, int y)
{
    const float* base = I + (size_t)y * sx + x;
    uint32_t word[NSP];
#pragma unroll
    for (int wd = 0; wd < NSP; wd++) {
        const int s0 = wd * 32;
        const int cnt = min(32, N - s0);
        uint32_t acc = 0;
#pragma unroll 4
        for (int b = 0; b < cnt; b++) {
            int4 q = s_pat[s0 + b];
            int ox1 = max(-x, min(sx - x - 1, q.x));
            int oy1 = max(-y, min(sy - y - 1, q.y));
            int ox2 = max(-x, min(sx - x - 1, q.z));
            int oy2 = max(-y, min(sy - y - 1, q.w));
            float i1 = __ldg(base + ox1 + (long)oy1 * sx);
            float i2 = __ldg(base + ox2 + (long)oy2 * sx);
            acc |= (i1 > i2 ? 1u : 0u) << b;
        }
        word[wd] = acc;
    }
    store_desc<NSP>(F + ((size_t)y * sx + x) * NSP, word);
}

// True when every pixel of the TX x TY tile at (bx, by) lies rmax or more inside.
__device__ __forceinline__ bool tile_interior(int bx, int by, int sx, int sy, int rmax)
{
    return (bx - rmax >= 0) && (bx + TX - 1 + rmax < sx) && (by - rmax >= 0) && (by + TY - 1 + rmax < sy);
}

// Chained launches (programmatic dependent launch): a kernel may start while the one
// before it runs its last blocks, and waits here for that one to be complete.  The
// trigger for the next kernel comes after the wait, so everything older than a kernel's
// immediate predecessor is complete when it starts; only what that predecessor wrote
// (or read) has to be touched after the wait, and never by the read-only path.  A pair's
// levels are 17 or more launches in a row, 2.5 us apart on small frames: chained, a pair of
// 96x64 frames took 166 us (207), 320x240 263 (299), 1024x436 u2.9 1209 (1254).
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------------------
// PatchMatch (briefmatch_cuda.cu:126-246).
// ---------------------------------------------------------------------------
// Zero or temporal initialisation (briefmatch_cuda.cu:149-184); temporal init reads
// the previous field from flow_prev (a snapshot) and writes flow_out.  CHAINED: the
// launch before may have written the descriptors after this one started; they are read
// through L2.
template <int NSP, bool CHAINED = false>
__device__ __forceinline__ void init_px(const uint32_t* F1, const uint32_t* F2,
                                        const uint32_t* __restrict__ flow_prev, uint32_t* __restrict__ flow_out,
                                        uint16_t* __restrict__ cost, int sx, int sy, int first, int x, int y)
{
    const long n = (long)sx * sy;
    const long pix = x + (long)y * sx;
    int nx = 0, ny = 0;
    if (!first) {
        uint32_t own = flow_prev[pix];
        long q = pix + lo16(own) + (long)hi16(own) * sx;
        uint32_t t = (q >= 0 && q < n) ? flow_prev[q] : 0u;
        nx = min(max(lo16(t), -x), sx - x - 1);
        ny = min(max(hi16(t), -y), sy - y - 1);
    }
    uint32_t f1[NSP];
    load_desc<NSP, CHAINED>(f1, F1 + pix * NSP);
    cost[pix] = (uint16_t)hamming<NSP, CHAINED>(f1, F2 + (pix + nx + (long)ny * sx) * NSP);
    flow_out[pix] = pack_flow(nx, ny);
}

// Seeded initialisation: first the plain initialisation (zero vector, or the
// temporal candidate when !first, exactly as init_px), then the network's proposal
// for this pixel -- pred is [h4][w4][3] (u, v in quarter-resolution input pixels,
// confidence logit) -- where its confidence logit reaches logit_min; the proposal
// replaces the plain vector only if its Hamming cost is strictly lower.  CHAINED: as
// init_px.
template <int NSP, bool CHAINED>
__device__ __forceinline__ void seed_px(const uint32_t* F1, const uint32_t* F2,
                                        const uint32_t* __restrict__ flow_prev, uint32_t* __restrict__ flow_out,
                                        uint16_t* __restrict__ cost, int sx, int sy, int first, int x, int y,
                                        const float* __restrict__ pred, int w4, int h4, float scale_x, float scale_y,
                                        float inv_x, float inv_y, float logit_min)
{
    const long n = (long)sx * sy;
    const long pix = x + (long)y * sx;
    int nx = 0, ny = 0;
    if (!first) {
        uint32_t own = flow_prev[pix];
        long q = pix + lo16(own) + (long)hi16(own) * sx;
        uint32_t t = (q >= 0 && q < n) ? flow_prev[q] : 0u;
        nx = min(max(lo16(t), -x), sx - x - 1);
        ny = min(max(hi16(t), -y), sy - y - 1);
    }
    uint32_t f1[NSP];
    load_desc<NSP, CHAINED>(f1, F1 + pix * NSP);
    int h = hamming<NSP, CHAINED>(f1, F2 + (pix + nx + (long)ny * sx) * NSP);
    // quarter-resolution cell of this up-sampled pixel (scale = up-sampled px per
    // quarter-resolution px, inv = its reciprocal from the host, so the cell index
    // is one IEEE add and multiply: no approximate division)
    const int qx = min(w4 - 1, max(0, (int)((x + 0.5f) * inv_x)));
    const int qy = min(h4 - 1, max(0, (int)((y + 0.5f) * inv_y)));
    const float* pr = pred + ((size_t)qy * w4 + qx) * 3;
    if (pr[2] >= logit_min) {
        const int sxv = min(max(__float2int_rn(pr[0] * scale_x), -x), sx - x - 1);
        const int syv = min(max(__float2int_rn(pr[1] * scale_y), -y), sy - y - 1);
        if (sxv != nx || syv != ny) {
            const int hs = hamming<NSP, CHAINED>(f1, F2 + (pix + sxv + (long)syv * sx) * NSP);
            if (hs < h) {
                h = hs;
                nx = sxv;
                ny = syv;
            }
        }
    }
    cost[pix] = (uint16_t)h;
    flow_out[pix] = pack_flow(nx, ny);
}

// One jump-flood level at step p (briefmatch_cuda.cu:206-219) for pixel (x, y).
// Neighbours are read from flow_in (the previous level's field) and the result is
// written to flow_out, so the outcome does not depend on the schedule.  All
// neighbour reads are issued together, then all candidate descriptors are gathered
// together, and only then are the candidates accepted in the reference's order
// (d = -1, +1; vertical then horizontal; strictly lower cost wins, insert()
// :126-147).  Candidates equal to the current vector (the reference's own skip) or
// to an earlier candidate cannot change a decision, so their gathers are elided.
// With RS the iteration's random-search candidate (:237-243) is evaluated last; it
// reads only this pixel's own state, so fusing it into the last level gives the
// reference's result.
// INLAUNCH: the field and cost were written after this kernel started -- by an earlier
// phase of the same launch (the persistent batched kernel), or by the level before it
// (chained launches); they are then read through L2 (ld.global.cg), never through the
// non-coherent read-only path.  (Ordinary loads instead: a batch of 12 pairs 0.7 % slower.)
template <bool INLAUNCH>
__device__ __forceinline__ uint32_t field_load(const uint32_t* p)
{
    if constexpr (INLAUNCH)
        return __ldcg(p);
    else
        return __ldg(p);
}

// Linear offsets of a level's neighbours, down a column (v) and along a row (h), for
// d = +1 (d = -1 negates them).  An offset of n = sx * sy or more leaves the plane
// from every pixel; it is held at n, so that pixel + offset fits 32 bits
// (n <= 32767^2).
struct JumpStep {
    int v, h;
};
__device__ __forceinline__ JumpStep jump_step(int sx, int sy, int p, int pd)
{
    const long n = (long)sx * sy;
    const long h = (long)pd * p, v = h * sx;
    return {(int)max(-n, min(n, v)), (int)max(-n, min(n, h))};
}

// A register with no defined value and no instruction to define it: the words of a
// gather whose predicate is off are never looked at.
__device__ __forceinline__ uint32_t undefined_word()
{
    uint32_t r;
    asm("" : "=r"(r));
    return r;
}

// 16 bytes of a descriptor, read only when `pred` holds (undefined words otherwise).
__device__ __forceinline__ uint4 gather16_pred(const uint32_t* __restrict__ src, bool pred)
{
    uint4 w = make_uint4(undefined_word(), undefined_word(), undefined_word(), undefined_word());
    asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t@p ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%5];\n\t}"
        : "+r"(w.x), "+r"(w.y), "+r"(w.z), "+r"(w.w)
        : "r"(pred ? 1 : 0), "l"(src));
    return w;
}

// The same for data read once (evict-first), as load_desc_stream.
__device__ __forceinline__ uint4 stream16_pred(const uint32_t* __restrict__ src, bool pred)
{
    uint4 w = make_uint4(undefined_word(), undefined_word(), undefined_word(), undefined_word());
    asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t@p ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%5];\n\t}"
        : "+r"(w.x), "+r"(w.y), "+r"(w.z), "+r"(w.w)
        : "r"(pred ? 1 : 0), "l"(src));
    return w;
}

__device__ __forceinline__ int hamming16(const uint4& a, const uint4& b)
{
    return __popc(a.x ^ b.x) + __popc(a.y ^ b.y) + __popc(a.z ^ b.z) + __popc(a.w ^ b.w);
}

// Candidates of a level for one pixel: the four neighbours' vectors (0 outside the
// plane), clamped into the image two components at a time (16-bit pairs), and the
// random-search candidate.  A candidate equal to `own` or to an earlier one is not
// live; with doubleProp off the d = -1 neighbours become `own`.
template <bool RS, bool INLAUNCH>
__device__ __forceinline__ void jump_candidates(const uint32_t* flow_in, uint32_t own, int sx, int sy, JumpStep js,
                                                int doubleProp, const RsArgs& rs, int x, int y, int pix,
                                                uint32_t (&cand)[RS ? 5 : 4], bool (&live)[RS ? 5 : 4])
{
    constexpr int NC = RS ? 5 : 4;
    const unsigned int n = (unsigned int)(sx * sy);
    const uint32_t lo = pack_flow(-x, -y), hi = pack_flow(sx - x - 1, sy - y - 1);
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int off = (c & 1) ? js.h : js.v;
        const int q = pix + (c < 2 ? -off : off);
        const bool active = c >= 2 || doubleProp;
        const uint32_t nb = (active && (unsigned int)q < n) ? field_load<INLAUNCH>(flow_in + q) : 0u;
        cand[c] = active ? __vmaxs2(__vmins2(nb, hi), lo) : own;
    }
    if constexpr (RS) {
        float n1, n2;
        rs_normals(rs, (unsigned int)pix, n1, n2);
        const int nx = min(max((int)round(rs.dist * n1), -x), sx - x - 1);
        const int ny = min(max((int)round(rs.dist * n2), -y), sy - y - 1);
        cand[NC - 1] = pack_flow(nx, ny);
    }
#pragma unroll
    for (int c = 0; c < NC; c++) {
        bool dup = cand[c] == own;
#pragma unroll
        for (int k = 0; k < c; k++) dup = dup || cand[k] == cand[c];
        live[c] = !dup;
    }
}

// Descriptors of up to 16 bytes: one thread reads its pixel's descriptor and its
// candidates' whole; a thread without a live candidate reads none.  The level is bound
// by the L1 data pipe (a gather of 32 scattered 16-byte vectors takes ~18 wavefronts)
// with the integer pipe next to it: 32-bit indices and clamps on 16-bit pairs took the
// integer pipe from 74 % to 52 % and a level at 1024x436 u2.9 N128 from 42.0 to 36.8 us
// (67.1 to 56.9 with the random search, whose state now stays in registers).
template <int NSP, bool RS, bool INLAUNCH = false>
__device__ __forceinline__ void jump_px(const uint32_t* __restrict__ F1, const uint32_t* __restrict__ F2,
                                        const uint32_t* flow_in, uint32_t* flow_out, uint16_t* cost, int sx, int sy,
                                        JumpStep js, int doubleProp, const RsArgs& rs, int x, int y)
{
    static_assert(NSP <= 4, "longer descriptors go through jump_row");
    constexpr int NC = RS ? 5 : 4;
    const int pix = x + y * sx;
    const uint32_t own = field_load<INLAUNCH>(flow_in + pix);
    uint32_t cand[NC];
    bool live[NC];
    jump_candidates<RS, INLAUNCH>(flow_in, own, sx, sy, js, doubleProp, rs, x, y, pix, cand, live);
    bool any = live[0];
#pragma unroll
    for (int c = 1; c < NC; c++) any = any || live[c];
    uint32_t best = own;
    if (any) {
        const int h0 = INLAUNCH ? (int)__ldcg(cost + pix) : (int)cost[pix];
        uint32_t f1[NSP];
        load_desc_stream<NSP>(f1, F1 + (size_t)(unsigned int)pix * NSP);
        // predicated gathers, all in flight at once
        uint32_t g[NC][NSP];
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const int t = pix + lo16(cand[c]) + hi16(cand[c]) * sx;
            gather_desc_pred<NSP>(g[c], F2 + (size_t)(unsigned int)t * NSP, live[c]);
        }
        int h = h0;
#pragma unroll
        for (int c = 0; c < NC; c++) {
            int acc = 0;
#pragma unroll
            for (int k = 0; k < NSP; k++) acc += __popc(f1[k] ^ g[c][k]);
            if (live[c] && acc < h) {
                h = acc;
                best = cand[c];
            }
        }
        if (h != h0) cost[pix] = (uint16_t)h;
    }
    flow_out[pix] = best;
}

// Descriptors of 32 or 64 bytes: a warp takes 32 consecutive pixels of a row (lane =
// pixel for the candidates and the decision) and reads descriptors L = NSP / 4 lanes
// to one, 16 bytes each, so that one load instruction covers 32 / L whole descriptors
// in consecutive sectors.  One lane reading a 64-byte descriptor alone touches a line
// of its own with every 16-byte load: at N = 512 that kept the L1 data pipe 91 % busy
// with HBM at 52 % (3136x1764 pixels, 249 us under ncu); this form is bound by HBM
// (the same level in the engine: 132 us, 116 us at the measured copy bandwidth for its
// 140 bytes per pixel; the whole 1920x1080 u4.9 N512 pair 56.8 -> 47.2 ms).  Step s serves pixels s * (32 / L) ...; each lane's partial distances
// of the L steps are summed over the L lanes by a reduce-scatter that leaves step k's
// sums with the group's lane k, and one shuffle hands them to the pixel's lane.  All
// 32 lanes take part; `valid` says which pixels lie in the image (x, y are then theirs).
template <int NSP, bool RS, bool INLAUNCH = false>
__device__ __forceinline__ void jump_row(const uint32_t* __restrict__ F1, const uint32_t* __restrict__ F2,
                                         const uint32_t* flow_in, uint32_t* flow_out, uint16_t* cost, int sx, int sy,
                                         JumpStep js, int doubleProp, const RsArgs& rs, int x, int y, bool valid)
{
    static_assert(NSP == 8 || NSP == 16, "two or four lanes per descriptor");
    constexpr int NC = RS ? 5 : 4;
    constexpr int L = NSP / 4;      // lanes per descriptor
    constexpr int PPS = 32 / L;     // pixels per step
    constexpr int NP = (NC + 1) / 2;  // packed pairs of distances (each at most 512)
    const unsigned int FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int pix = x + y * sx;
    uint32_t own = 0, cand[NC];
    int h0 = 0;
    int t[NC];   // target pixel of a live candidate, else -1
    bool any = false;
#pragma unroll
    for (int c = 0; c < NC; c++) t[c] = -1;
    if (valid) {
        bool live[NC];
        own = field_load<INLAUNCH>(flow_in + pix);
        h0 = INLAUNCH ? (int)__ldcg(cost + pix) : (int)cost[pix];
        jump_candidates<RS, INLAUNCH>(flow_in, own, sx, sy, js, doubleProp, rs, x, y, pix, cand, live);
#pragma unroll
        for (int c = 0; c < NC; c++) {
            if (live[c]) t[c] = pix + lo16(cand[c]) + hi16(cand[c]) * sx;
            any = any || live[c];
        }
    }
    uint32_t best = own;
    if (__any_sync(FULL, any)) {
        const int part = lane & (L - 1), slot = lane / L;
        const int pix0 = __shfl_sync(FULL, pix, 0);   // lane 0's pixel; the row's others follow
        uint32_t sum[L][NP];
        constexpr int G = NSP == 8 ? 2 : 1;   // steps in flight together (measured; 64 bytes spill with two)
#pragma unroll
        for (int s0 = 0; s0 < L; s0 += G) {
            uint4 f1[G], g[G][NC];
#pragma unroll
            for (int i = 0; i < G; i++) {
                const int j = (s0 + i) * PPS + slot;
                int tj[NC];
                bool aj = false;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    tj[c] = __shfl_sync(FULL, t[c], j);
                    aj = aj || tj[c] >= 0;
                }
                f1[i] = stream16_pred(F1 + (size_t)(unsigned int)(pix0 + j) * NSP + part * 4, aj);
#pragma unroll
                for (int c = 0; c < NC; c++)
                    g[i][c] = gather16_pred(F2 + (size_t)(unsigned int)tj[c] * NSP + part * 4, tj[c] >= 0);
            }
#pragma unroll
            for (int i = 0; i < G; i++)
#pragma unroll
                for (int k = 0; k < NP; k++) {
                    sum[s0 + i][k] = (uint32_t)hamming16(f1[i], g[i][2 * k]);
                    if (2 * k + 1 < NC) sum[s0 + i][k] |= (uint32_t)hamming16(f1[i], g[i][2 * k + 1]) << 16;
                }
        }
        uint32_t mine[NP];
#pragma unroll
        for (int k = 0; k < NP; k++) {
            uint32_t v[L];
#pragma unroll
            for (int s = 0; s < L; s++) v[s] = sum[s][k];
            // halve the steps held per lane until one is left: step == part
#pragma unroll
            for (int w = L / 2; w > 0; w /= 2) {
                const bool up = (part & w) != 0;
#pragma unroll
                for (int s = 0; s < w; s++) {
                    const uint32_t give = up ? v[s] : v[s + w];
                    const uint32_t keep = up ? v[s + w] : v[s];
                    v[s] = keep + __shfl_xor_sync(FULL, give, w);
                }
            }
            // lane slot * L + part now holds pixel part * PPS + slot
            mine[k] = __shfl_sync(FULL, v[0], (lane % PPS) * L + lane / PPS);
        }
        int h = h0;
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const int hc = (int)((c & 1) ? mine[c / 2] >> 16 : mine[c / 2] & 0xffffu);
            if (t[c] >= 0 && hc < h) {
                h = hc;
                best = cand[c];
            }
        }
        if (h != h0) cost[pix] = (uint16_t)h;
    }
    if (valid) flow_out[pix] = best;
}

// One level for the warp's 32 pixels, by descriptor length.
template <int NSP, bool RS, bool INLAUNCH = false>
__device__ __forceinline__ void jump_level_px(const uint32_t* __restrict__ F1, const uint32_t* __restrict__ F2,
                                              const uint32_t* flow_in, uint32_t* flow_out, uint16_t* cost, int sx,
                                              int sy, int p, int pd, int doubleProp, const RsArgs& rs, int x, int y)
{
    const JumpStep js = jump_step(sx, sy, p, pd);
    const bool valid = x < sx && y < sy;
    if constexpr (NSP >= 8)
        jump_row<NSP, RS, INLAUNCH>(F1, F2, flow_in, flow_out, cost, sx, sy, js, doubleProp, rs, x, y, valid);
    else if (valid)
        jump_px<NSP, RS, INLAUNCH>(F1, F2, flow_in, flow_out, cost, sx, sy, js, doubleProp, rs, x, y);
}

// Local refinement step of the seeded schedule (no reference counterpart): the
// pixel's own vector moved by r up-sampled pixels left, right, up and down (clamped
// into the image), in that order, each kept only when strictly cheaper than the
// best so far.  Reads flow_in (a snapshot) and writes flow_out, like a jump level.
template <int NSP>
__device__ __forceinline__ void local_px(const uint32_t* __restrict__ F1, const uint32_t* __restrict__ F2,
                                         const uint32_t* flow_in, uint32_t* flow_out,
                                         uint16_t* cost, int sx, int sy, int r, int x, int y)
{
    const long pix = x + (long)y * sx;
    const uint32_t own = __ldcg(flow_in + pix);
    const int h0 = (int)__ldcg(cost + pix);
    const int ox = lo16(own), oy = hi16(own);
    uint32_t cand[4];
    bool live[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int dx = c == 0 ? -r : (c == 1 ? r : 0);
        const int dy = c == 2 ? -r : (c == 3 ? r : 0);
        const int nx = min(max(ox + dx, -x), sx - x - 1);
        const int ny = min(max(oy + dy, -y), sy - y - 1);
        cand[c] = pack_flow(nx, ny);
        bool dup = cand[c] == own;
#pragma unroll
        for (int k = 0; k < c; k++) dup = dup || cand[k] == cand[c];
        live[c] = !dup;
    }
    uint32_t f1[NSP];
    load_desc_stream<NSP>(f1, F1 + pix * NSP);
    uint32_t g[4][NSP];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const long t = pix + lo16(cand[c]) + (long)hi16(cand[c]) * sx;
        gather_desc_pred<NSP>(g[c], F2 + t * NSP, live[c]);
    }
    int h = h0;
    uint32_t best = own;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        int acc = 0;
#pragma unroll
        for (int k = 0; k < NSP; k++) acc += __popc(f1[k] ^ g[c][k]);
        if (live[c] && acc < h) {
            h = acc;
            best = cand[c];
        }
    }
    flow_out[pix] = best;
    if (h != h0) cost[pix] = (uint16_t)h;
}

// ---------------------------------------------------------------------------
// Down-sampling (briefmatch.cpp:296-324) for input-resolution pixel (x, y):
// int16 -> float, Gaussian H then V evaluated only where the nearest-neighbour
// decimation samples (source index tables nnx/nny), scaled by (mx, my).  Each
// pass keeps the reference's float rounding and fused multiply-adds.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void downsample_px(const uint32_t* flow, float* __restrict__ U,
                                              float* __restrict__ V, int sx, int sy, int sx_in,
                                              const float* __restrict__ taps, int P, float mx, float my,
                                              const unsigned int* __restrict__ nnx, const unsigned int* __restrict__ nny,
                                              int x, int y)
{
    const unsigned int x1 = nnx[x], y1 = nny[y];
    const size_t o = (size_t)x + (size_t)y * sx_in;
    if (x1 >= (unsigned)sx || y1 >= (unsigned)sy) {
        U[o] = 0.0f;
        V[o] = 0.0f;
        return;
    }
    const int ks2 = P / 2;
    float su = 0, sv = 0;
    for (int i = 0; i < P; i++) {
        const int yy = min(sy - 1, max(0, (int)y1 + i - ks2));
        const uint32_t* row = flow + (size_t)yy * sx;
        float hu = 0, hv = 0;
        for (int k = 0; k < P; k++) {
            const uint32_t f = row[min(sx - 1, max(0, (int)x1 + k - ks2))];
            const float tk = taps[k];
            hu += tk * float(lo16(f));
            hv += tk * float(hi16(f));
        }
        su += taps[i] * hu;
        sv += taps[i] * hv;
    }
    U[o] = su * mx;
    V[o] = sv * my;
}

// The same for a block of TX x TY threads and the TX x rows outputs whose first is
// (x0, y0): neighbouring outputs of a column share most of their window's rows, so each
// row's horizontal sum is formed once, in `h` (down_smem_bytes of shared memory), and the
// vertical sums read it.  Per output (rows - 1) * u / rows + P / rows horizontal sums
// instead of P; what bounds it is their loads, u words apart (twelve of them in flight per
// thread instead of four: 198 us).  1920x1080 u4.9, 32 rows: 426 -> 186 us.
__host__ __device__ inline int down_rows_up(int rows, int sy, int sy_in, int P)
{
    // source rows of `rows` outputs: the index table rounds, so one more at either end
    return (int)((long)(rows - 1) * sy / sy_in) + 2 + P;
}
__host__ __device__ inline size_t down_smem_bytes(int rows, int sy, int sy_in, int P)
{
    return (size_t)down_rows_up(rows, sy, sy_in, P) * TX * sizeof(float2);
}
constexpr size_t DOWN_SMEM_MAX = 48 * 1024;   // what a launch may use without an opt-in
__device__ __forceinline__ void downsample_block(const uint32_t* flow, float* __restrict__ U, float* __restrict__ V,
                                                 int sx, int sy, int sx_in, int sy_in, const float* __restrict__ taps,
                                                 int P, float mx, float my, const unsigned int* __restrict__ nnx,
                                                 const unsigned int* __restrict__ nny, int x0, int y0, int rows,
                                                 float2* h)
{
    const int ks2 = P / 2;
    const int x = x0 + threadIdx.x;
    const int first = (int)__ldg(nny + y0), last = (int)__ldg(nny + min(y0 + rows, sy_in) - 1);
    const unsigned int x1 = x < sx_in ? __ldg(nnx + x) : 0xffffffffu;
    if (x1 < (unsigned)sx) {
        for (int j = threadIdx.y; j < last - first + P; j += TY) {
            const uint32_t* row = flow + (size_t)min(sy - 1, max(0, first + j - ks2)) * sx;
            float hu = 0, hv = 0;
#pragma unroll 4
            for (int k = 0; k < P; k++) {
                const uint32_t f = row[min(sx - 1, max(0, (int)x1 + k - ks2))];
                const float tk = __ldg(taps + k);
                hu = __fmaf_rn(tk, float(lo16(f)), hu);
                hv = __fmaf_rn(tk, float(hi16(f)), hv);
            }
            h[j * TX + threadIdx.x] = make_float2(hu, hv);
        }
    }
    __syncthreads();
    if (x >= sx_in) return;
    for (int y = y0 + threadIdx.y; y < min(y0 + rows, sy_in); y += TY) {
        const unsigned int y1 = __ldg(nny + y);
        const size_t o = (size_t)x + (size_t)y * sx_in;
        float su = 0, sv = 0;
        if (x1 < (unsigned)sx && y1 < (unsigned)sy) {
            const float2* col = h + ((int)y1 - first) * TX + threadIdx.x;
#pragma unroll 4
            for (int i = 0; i < P; i++) {
                const float ti = __ldg(taps + i);
                const float2 v = col[i * TX];
                su = __fmaf_rn(ti, v.x, su);
                sv = __fmaf_rn(ti, v.y, sv);
            }
            su *= mx;
            sv *= my;
        }
        U[o] = su;
        V[o] = sv;
    }
}

// ---------------------------------------------------------------------------
// 1-D median (util_cuda.cu:75-111) of the two outputs at linear indices p and
// p + step (the second only when `second`): each window is fsize samples at linear
// offsets -ks .. fsize-1-ks (ks = fsize/2), guard 0 outside the plane, and the median
// is the (ks+1)-th smallest.  The two windows share the fsize-1 samples S between
// them; with a the first output's own sample and b the second's, the (ks+1)-th
// smallest of S + {a} is min(max(a, S(ks-1)), S(ks)), S(i) the (i+1)-th smallest of
// S, so one partial selection (positions 0..ks, in registers padded with +inf up to
// FS-1) serves both outputs.
// ---------------------------------------------------------------------------
template <int FS>
__device__ __forceinline__ void median2_px(const float* in, float* __restrict__ out, long p, long step,
                                           long n, int fsize, bool second)
{
    const int ks = fsize / 2;
    auto sample = [&](long idx) { return (idx >= 0 && idx < n) ? in[idx] : 0.0f; };
    const float a = sample(p - (long)ks * step);
    const float b = second ? sample(p + (long)(fsize - ks) * step) : 0.0f;
    if (fsize == 1) {
        out[p] = a;
        if (second) out[p + step] = b;
        return;
    }
    float v[FS - 1];
#pragma unroll
    for (int k = 0; k < FS - 1; k++)
        v[k] = (k < fsize - 1) ? sample(p + (long)(k - ks + 1) * step) : __int_as_float(0x7f800000);
#pragma unroll
    for (int i = 0; i < (FS + 1) / 2; i++) {
        if (i <= ks) {
#pragma unroll
            for (int j = i + 1; j < FS - 1; j++) {
                const float x = v[i], y = v[j];
                v[i] = fminf(x, y);
                v[j] = fmaxf(x, y);
            }
        }
    }
    float lo = v[0], hi = v[1];
#pragma unroll
    for (int i = 1; i < (FS + 1) / 2; i++)
        if (i == ks) {
            lo = v[i - 1];
            hi = v[i];
        }
    out[p] = fminf(fmaxf(a, lo), hi);
    if (second) out[p + step] = fminf(fmaxf(b, lo), hi);
}

// ---------------------------------------------------------------------------
// Cross-trilateral filter (briefmatch_cuda.cu:248-297): one block filters the TX x
// 4 TY outputs whose top-left pixel is (bx0, by0).  Each thread owns four vertically
// adjacent outputs and walks the window column by column, two source rows at a time:
// packed f32x2 registers hold the two rows, so a sample pair is used as it is read from
// shared memory (the tile is stored column by column) and serves all four outputs.
// TRI_G = 2 groups of TX x TY threads share a tile, each taking half of the window's
// columns; their sums meet in shared memory (small windows: one group, G = 1).  The
// neighbourhood is staged with clamp-to-edge addressing, `smem` must hold
// tri_smem_bytes(s, TY).
//
// The three Gaussians are one exp2 of the summed exponents,
// r q = r (du^2 + dv^2 + dI^2 + j^2 cS / r) over scaled differences: kE is the power of two
// nearest sqrt(cE), r = cE / kE^2 the factor that leaves, kI = sqrt(cI / r).  With it a flow's
// scaled difference is exact but for one rounding: a scale that rounds, kE = sqrt(cE) and no
// factor, saves the multiplication, but puts an error of q's size into the weights far from
// the centre, and where only such are left (a sum of weights under the floor of 1e-5) the
// output was up to 4e-4 px off at flows of 18 px.
//
// What is summed are the weighted differences du and dv to the output's own median value,
// which is added back to the quotient: the sums are of small numbers whatever the flow is,
// and a value depends on nothing outside its window.  Error against 64 bits: 2.6e-8 of the
// norm of a 1920x1080 field, which is the rounding of the result (sums of the flow itself
// 2.2e-7; sums relative to one reference flow per block 3.1 to 5.0e-8, but up to 3e-4 px off
// at small flows beside a fast object, where these stay at 6e-10).  The column factor
// exp2(-cS i^2) is applied once per column.  Ten FP32 lane operations per tap and output.
//
// What bounds it is the FP32 pipe's operand reads: a packed FMA with three different
// 64-bit registers takes three cycles, with two it takes two (measured; an operand that is
// the same for the whole grid does not count).  So flow differences are additions, the
// intensity's an FMA with the grid's scale, squares read one register twice, and only the two
// weighted sums need three registers: 22 cycles per pair of taps, 20 by operation count.
// 1920x1080 with a 94 x 94 window: 7.16 -> 6.12 ms; 1024x436 (48 x 48): 400 -> 372 us (without
// the factor r 5.61 and 342).  The tile's loads are eight in flight per thread, the medians'
// before them; one after the other they took 0.1 ms of the former, and half the time of
// small windows.
//
// Flows beyond TRI_FAR of a standard deviation (and infinite ones) as a centre: the sums
// over differences would meet 0 * inf, so such an output takes its sums over the flow.
//
// Row pairs: source row m lies in output r's window when 0 <= m - r < 2s.  Outputs 0
// and 2 take whole pairs; outputs 1 and 3 have a single row in their first and last
// pair, whose other half is taken as zero with an infinite row term, so no sample
// outside a window is touched.
// ---------------------------------------------------------------------------
constexpr int TRI_R = 4;       // outputs per thread
constexpr int TRI_UNROLL = 8;  // row pairs per turn of the column walk (measured: 1, 2, 4, 8, 16)
constexpr int TRI_MAX_S = 52;  // largest half window whose tile fits an SM's shared memory (226 KB)
constexpr int TRI_G = 2;       // thread groups per block, each taking half of the window's columns (small windows: 1)

// Rows of a tile of TY thread rows, and floats per tile column: the rows, padded to 2
// modulo 4 so that the 16 lanes of a 64-bit read phase fall on 32 different banks.
__host__ __device__ constexpr int tri_rows(int ty) { return ty * TRI_R; }
__host__ __device__ inline int tri_pitch(int s, int ty) { return tri_rows(ty) + 2 * s + ((s & 1) ? 0 : 2); }

__host__ __device__ inline size_t tri_smem_bytes(int s, int ty)
{
    const size_t tile = (size_t)(TX + 2 * s) * tri_pitch(s, ty) * 3;
    const size_t sums = (size_t)(TRI_G - 1) * TX * ty * TRI_R * 3;   // the groups' partial sums reuse the tile
    return (size_t)(s + 1) * sizeof(float4) + (tile > sums ? tile : sums) * sizeof(float);
}

constexpr float TRI_FAR = 1e30f;
// A finite flow held where its scaled difference stays finite.
__device__ __forceinline__ float tri_held(float v, float most)
{
    return fabsf(v) > most && fabsf(v) <= 3.402823466e38f ? copysignf(most, v) : v;
}

// Exponent scales of the trilateral weights: exp(-d/(2 sigma2)) = exp2(-d * c)
// with intensities divided by 255 folded into cI; kE, r and kI as trilateral_block has them.
struct TriCoef {
    float cE, cI, cS;
    float kE, r, kI, cSr;   // cSr = cS / r
    bool scaled;            // kE and r are ordinary numbers (cE is neither 0 nor infinite)
};
inline TriCoef tri_coef(float sigmaEPE2, float sigmaI2, float sigmaS2)
{
    const float LOG2E = 1.4426950408889634f;
    TriCoef t;
    t.cE = LOG2E / (2.0f * sigmaEPE2);
    t.cI = LOG2E / (2.0f * sigmaI2 * 255.0f * 255.0f);
    t.cS = LOG2E / (2.0f * sigmaS2);
    t.scaled = t.cE > 0.0f && t.cE < 3.0e38f;
    const double cE = t.scaled ? (double)t.cE : 1.0;
    const double kE = __builtin_exp2(__builtin_rint(0.5 * __builtin_log2(cE))), r = cE / (kE * kE);
    t.kE = (float)kE;
    t.r = (float)r;
    t.kI = (float)__builtin_sqrt((double)t.cI / r);
    t.cSr = (float)((double)t.cS / r);
    return t;
}

// 2^-x per half.  The negation is spelled without .ftz, which makes it a modifier of the
// exponential's operand: under -use_fast_math a C++ minus is neg.ftz, an addition of its
// own on the FP32 pipe (two of them per pair of taps were 19 % of that pipe's work).
__device__ __forceinline__ float ex2n(float x)
{
    float r;
    asm("{\n\t.reg .f32 t;\n\tneg.f32 t, %1;\n\tex2.approx.ftz.f32 %0, t;\n\t}" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ f2x ex2n_2(f2x a) { return pk2(ex2n(lo2(a)), ex2n(hi2(a))); }

template <int TY, int G>
__device__ __forceinline__ void trilateral_block(const float* __restrict__ U, const float* __restrict__ V,
                                                 const float* Um, const float* Vm,
                                                 const float* __restrict__ I, float* __restrict__ Uo,
                                                 float* __restrict__ Vo, int sx, int sy, int s, const TriCoef& tc,
                                                 int bx0, int by0, float4* smem4)
{
    const float kE = tc.kE, kI = tc.kI;
    const int TW = TX + 2 * s, TH = tri_rows(TY) + 2 * s, P = tri_pitch(s, TY);
    // row terms of pair p: outputs 0 (.x .y: rows 2p, 2p + 1) and 1 (.z .w: rows 2p - 1,
    // 2p); outputs 2 and 3 use pair p - 1's
    float4* rowf = smem4;                                     // [s + 1]
    float* sU = reinterpret_cast<float*>(smem4 + s + 1);      // [TW][P], column by column
    float* sV = sU + TW * P;
    float* sI = sV + TW * P;
    const int x0 = bx0 - s, y0 = by0 - s;
    const float most = kE > 1.0f ? 1e38f / kE : 3.402823466e38f;
    const int x = bx0 + threadIdx.x;
    const int yb = by0 + threadIdx.y * TRI_R;
    // (pixels outside the image compute on clamped centres and store nothing)
    f2x um[TRI_R], vm[TRI_R], ic[TRI_R];   // negated scaled centres, twice
#pragma unroll
    for (int r = 0; r < TRI_R; r++) {
        const size_t o = (size_t)min(sx - 1, x) + (size_t)min(sy - 1, yb + r) * sx;
        const float a = __fmul_rn(-kE, Um[o]), b = __fmul_rn(-kE, Vm[o]);
        um[r] = pk2(a, a);
        vm[r] = pk2(b, b);
    }
    // four rows of two columns at a time: their loads are in flight together
    constexpr int STEP = TY * G, ROWS = 4;
    for (int c0 = threadIdx.x; c0 < TW; c0 += 2 * TX) {
        const int gx[2] = {min(sx - 1, max(0, x0 + c0)), min(sx - 1, max(0, x0 + c0 + TX))};
        const int cols = c0 + TX < TW ? 2 : 1;
        for (int r0 = threadIdx.z * TY + threadIdx.y; r0 < TH; r0 += STEP * ROWS) {
            float a[ROWS][2], b[ROWS][2], i[ROWS][2];
#pragma unroll
            for (int k = 0; k < ROWS; k++) {
                const size_t row = (size_t)min(sy - 1, max(0, y0 + r0 + k * STEP)) * sx;
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (r0 + k * STEP < TH && h < cols) {
                        a[k][h] = __ldg(U + row + gx[h]);
                        b[k][h] = __ldg(V + row + gx[h]);
                        i[k][h] = __ldg(I + row + gx[h]);
                    }
            }
#pragma unroll
            for (int k = 0; k < ROWS; k++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (r0 + k * STEP < TH && h < cols) {
                        const int at = (c0 + h * TX) * P + r0 + k * STEP;
                        sU[at] = __fmul_rn(kE, tri_held(a[k][h], most));
                        sV[at] = __fmul_rn(kE, tri_held(b[k][h], most));
                        sI[at] = i[k][h];
                    }
        }
    }
    for (int p = threadIdx.y * TX + threadIdx.x; p <= s; p += TX * TY) {
        auto term = [&](int n) {
            return n >= 0 && n < 2 * s ? (float)((n - s) * (n - s)) * tc.cSr : __int_as_float(0x7f800000);
        };
        rowf[p] = make_float4(term(2 * p), term(2 * p + 1), term(2 * p - 1), term(2 * p));
    }
    __syncthreads();

#pragma unroll
    for (int r = 0; r < TRI_R; r++) {
        const float i0 = __fmul_rn(-kI, sI[(threadIdx.x + s) * P + threadIdx.y * TRI_R + r + s]);
        ic[r] = pk2(i0, i0);
    }
    float su[TRI_R], sv[TRI_R], sw[TRI_R];
#pragma unroll
    for (int r = 0; r < TRI_R; r++) su[r] = sv[r] = sw[r] = 0.0f;

    const f2x kII = pk2(kI, kI), rr = pk2(tc.r, tc.r);
    struct Pair {
        f2x u, v, i;
    };
    const ulonglong2* terms = reinterpret_cast<const ulonglong2*>(rowf);
    auto column = [&](int i) {
        const float* cu = sU + (threadIdx.x + s + i) * P + threadIdx.y * TRI_R;
        const int plane = TW * P;
        f2x au[TRI_R], av[TRI_R], aw[TRI_R];
#pragma unroll
        for (int r = 0; r < TRI_R; r++) au[r] = av[r] = aw[r] = 0;   // 0 bits = (0.0f, 0.0f)
        auto load = [&](int p) {
            Pair t;
            t.u = *reinterpret_cast<const f2x*>(cu + 2 * p);
            t.v = *reinterpret_cast<const f2x*>(cu + plane + 2 * p);
            t.i = *reinterpret_cast<const f2x*>(cu + 2 * plane + 2 * p);
            return t;
        };
        auto sums = [&](int r, const Pair& t, f2x row) {
            const f2x du = add2(t.u, um[r]), dv = add2(t.v, vm[r]), dI = fma2(t.i, kII, ic[r]);
            const f2x w = ex2n_2(mul2(fma2(dI, dI, fma2(dv, dv, fma2(du, du, row))), rr));
            au[r] = fma2(w, du, au[r]);
            av[r] = fma2(w, dv, av[r]);
            aw[r] = add2(aw[r], w);
        };
        auto upper = [&](const Pair& t) { return Pair{pk2(0.0f, hi2(t.u)), pk2(0.0f, hi2(t.v)), pk2(0.0f, hi2(t.i))}; };
        auto lower = [&](const Pair& t) { return Pair{pk2(lo2(t.u), 0.0f), pk2(lo2(t.v), 0.0f), pk2(lo2(t.i), 0.0f)}; };
        ulonglong2 f = terms[0];
        f2x e0 = f.x, e1 = f.y;                       // the previous pair's terms
        Pair t = load(0);                             // rows 0, 1
        sums(0, t, e0);
        Pair h = upper(t);
        sums(1, h, e1);
        if (s > 1) {
            f = terms[1];
            t = load(1);                              // rows 2, 3
            f2x t0 = f.x, t1 = f.y;
            sums(0, t, t0);
            sums(1, t, t1);
            sums(2, t, e0);
            h = upper(t);
            sums(3, h, e1);
#pragma unroll TRI_UNROLL
            for (int p = 2; p < s; p++) {
                f = terms[p];
                t0 = f.x;
                t1 = f.y;
                f = terms[p - 1];   // reloaded, not carried over: a copy per step costs more
                e0 = f.x;
                e1 = f.y;
                t = load(p);
                sums(0, t, t0);
                sums(1, t, t1);
                sums(2, t, e0);
                sums(3, t, e1);
            }
            f = terms[s - 1];
            e0 = f.x;
            e1 = f.y;
        }
        f = terms[s];
        t = load(s);                                  // rows 2s, 2s + 1
        const f2x last = f.y;
        h = lower(t);
        sums(1, h, last);
        sums(2, t, e0);
        if (s > 1) {
            sums(3, t, e1);
        } else {
            h = upper(t);
            sums(3, h, e1);
        }
        t = load(s + 1);                              // row 2s + 2
        h = lower(t);
        sums(3, h, last);
        const float wi = exp2f(-(float)(i * i) * tc.cS);
#pragma unroll
        for (int r = 0; r < TRI_R; r++) {
            su[r] = __fmaf_rn(wi, lo2(au[r]) + hi2(au[r]), su[r]);
            sv[r] = __fmaf_rn(wi, lo2(av[r]) + hi2(av[r]), sv[r]);
            sw[r] = __fmaf_rn(wi, lo2(aw[r]) + hi2(aw[r]), sw[r]);
        }
    };
    // the columns [-s, 0) and [0, s) are summed apart, by two groups or one after the other,
    // and added at the end: a value is the same either way
    const int tid = threadIdx.y * TX + threadIdx.x;
    float other_u[TRI_R], other_v[TRI_R], other_w[TRI_R];
    if constexpr (G == 2) {
        for (int k = 0; k < s; k++) column(threadIdx.z ? k : k - s);
        __syncthreads();   // every group is done with the tile
        if (threadIdx.z) {
#pragma unroll
            for (int r = 0; r < TRI_R; r++) {
                sU[(3 * r + 0) * TX * TY + tid] = su[r];
                sU[(3 * r + 1) * TX * TY + tid] = sv[r];
                sU[(3 * r + 2) * TX * TY + tid] = sw[r];
            }
        }
    } else {
#pragma unroll 1
        for (int half = 0; half < 2; half++) {
            for (int k = 0; k < s; k++) column(half ? k : k - s);
            if (half == 0) {
#pragma unroll
                for (int r = 0; r < TRI_R; r++) {
                    other_u[r] = su[r];
                    other_v[r] = sv[r];
                    other_w[r] = sw[r];
                    su[r] = sv[r] = sw[r] = 0.0f;
                }
            }
        }
    }
    float a[TRI_R], b[TRI_R];
#pragma unroll
    for (int r = 0; r < TRI_R; r++) {
        const size_t o = (size_t)min(sx - 1, x) + (size_t)min(sy - 1, yb + r) * sx;
        a[r] = threadIdx.z ? 0.0f : Um[o];
        b[r] = threadIdx.z ? 0.0f : Vm[o];
    }
    if constexpr (G == 2) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < TRI_R; r++) {
            other_u[r] = sU[(3 * r + 0) * TX * TY + tid];
            other_v[r] = sU[(3 * r + 1) * TX * TY + tid];
            other_w[r] = sU[(3 * r + 2) * TX * TY + tid];
        }
    }
    if (threadIdx.z || x >= sx || yb >= sy) return;
    const float inv_k = __frcp_rn(kE);
#pragma unroll
    for (int r = 0; r < TRI_R; r++) {
        const float w = sw[r] + other_w[r];
        const float mu = su[r] + other_u[r];
        const float mv = sv[r] + other_v[r];
        if (yb + r < sy) {
            const size_t o = (size_t)x + (size_t)(yb + r) * sx;
            // sum of w u over max(1e-5, sum of w), with u = centre + scaled difference / kE
            auto quotient = [&](float centre, float m) {
                return w < 1e-5f ? __fdiv_rn(__fmaf_rn(centre, w, m * inv_k), 1e-5f)
                                 : __fmaf_rn(__fdiv_rn(m, w), inv_k, centre);
            };
            float u = quotient(a[r], mu), v = quotient(b[r], mv);
            if (fabsf(lo2(um[r])) > TRI_FAR || fabsf(lo2(vm[r])) > TRI_FAR) {
                float fu = 0.0f, fv = 0.0f, fw = 0.0f;
#pragma unroll 1
                for (int k = 0; k < 4 * s * s; k++) {
                    const int i = k / (2 * s) - s, j = k % (2 * s) - s;
                    const size_t g = (size_t)min(sx - 1, max(0, x + i)) + (size_t)min(sy - 1, max(0, yb + r + j)) * sx;
                    const float du = __fmaf_rn(kE, U[g], lo2(um[r])), dv = __fmaf_rn(kE, V[g], lo2(vm[r]));
                    const float dI = __fmaf_rn(kI, I[g], lo2(ic[r]));
                    const float f = exp2f(-(tc.r * (du * du + dv * dv + dI * dI) + (float)(i * i + j * j) * tc.cS));
                    fu = __fmaf_rn(f, U[g], fu);
                    fv = __fmaf_rn(f, V[g], fv);
                    fw += f;
                }
                u = __fdiv_rn(fu, fmaxf(1e-5f, fw));
                v = __fdiv_rn(fv, fmaxf(1e-5f, fw));
            }
            Uo[o] = u;
            Vo[o] = v;
        }
    }
}

}  // namespace dev
}  // namespace bmk
