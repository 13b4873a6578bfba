// bm_kernels.cu -- sm_103a kernels of the BriefMatch flow engine, single frame pair.
//
// This unit is compiled with -use_fast_math, the flags the reference kernels are
// built with (CMakeLists.txt:50), so that expressions whose rounding the reference
// fixes (Lanczos weights, the nearest-neighbour index of the down-sampler, the
// curand normals) produce the same bits as the reference build.  The per-pixel
// bodies live in bm_device.cuh, shared with the batched kernels.
//
// Layouts (all row-major, x fastest):
//   descriptors  uint32 [sx*sy][nsp], nsp = ceil(N/32) rounded up to a power of two,
//                padding words zero -- one pixel's descriptor is one or more uint4
//   flow         uint32 per pixel, int16 nx in the low half, int16 ny in the high half
//   cost         uint16 per pixel, the Hamming distance of the current candidate
//                (the reference's D is cost/N)
#include <climits>
#include <cstring>
#include <mutex>

#include "bm_device.cuh"

namespace bmk {

namespace {

using namespace dev;

inline dim3 grid2d(int w, int h) { return dim3((w + TX - 1) / TX, (h + TY - 1) / TY); }

// Tile visited by this block.  Full-frame passes alternate their visiting order
// (raster, then reverse raster): a pass that follows one in the other direction
// starts on the tiles its predecessor touched last, which are still in L2.
__device__ __forceinline__ int2 block_tile(int rev)
{
    int bx = blockIdx.x, by = blockIdx.y;
    if (rev) {
        bx = gridDim.x - 1 - bx;
        by = gridDim.y - 1 - by;
    }
    return make_int2(bx * TX, by * TY);
}

// Lanczos weight tables (util_cuda.cu:134-151): per output column (or row) the six
// weights with the reference's expression and the first tap index.
__global__ void k_lanczos_tables(float* __restrict__ w, int* __restrict__ idx, int n_in, int n_out)
{
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n_out) return;
    float xp = x * float(n_in) / n_out;
    int x1 = floor(xp);
    int a = 3;
    for (int k = 0; k < 6; k++) {
        int i = x1 - a + 1 + k;
        float xx = BM_PI * (xp - i);
        float L = a * sin(xx) * sin(xx / a) / (xx * xx);
        if (L != L) L = 1;
        w[x * 6 + k] = L;
    }
    idx[x] = x1;
}


template <typename T>
__global__ void __launch_bounds__(256) k_upsample(const T* __restrict__ in, float* __restrict__ out,
                                                  int sxi, int syi, int sxo, int syo,
                                                  const float* __restrict__ lx, const int* __restrict__ ix,
                                                  const float* __restrict__ ly, const int* __restrict__ iy)
{
    const int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
    if (x >= sxo || y >= syo) return;
    upsample_px<T>(in, out, sxi, syi, sxo, lx, ix, ly, iy, x, y);
}

// Up-sampling into an edge-replicated image: the output covers (sxo + 2m) x
// (syo + 2m) pixels at row pitch `pitch`; a pixel of the margin holds the value of
// the nearest image pixel (each coordinate clamped), computed by the same Lanczos
// expression, so every read of the margin equals a clamped read of the image.
// Each thread computes UP_R output rows of one column (a block covers
// TX x (TY * UP_R) outputs).  The rows share the column's six weights and source
// columns and the products input * Lx: those of the first row's Lanczos window are formed
// once (36 multiplies), and a window one source row further on moves them by a row and
// forms six more.  Each output takes its 36 multiply-adds onto them in the reference's
// order (util_cuda.cu:140-152: over source columns, then rows; v += (in * Lx) * Ly as one
// rounded product and an FMA, w += Lx * Ly as an FMA), so every value equals
// upsample_val's bit for bit.
//
// The rows' sums are kept and divided, keyed and stored together after the last row: with
// that the loads of later rows run ahead, and two blocks per SM at 121 registers take
// 39.5 us at 1024x436 u2.9 where three at 79 with a division per row took 47.6 (1920x1080
// u4.9 434 -> 393, 320x240 u2.9 14.8 -> 12.7; three blocks spill: 41.7 and 387).
//
// Beside the float image the kernel writes the key image the descriptors read: a word
// per pixel with the 16-bit key (sample_key) of the pixel in its low half and of the
// pixel below it in its high half (if it has one: it may be missing where memory is short).
// A thread pairs the keys of its own rows; the word that spans two threads' rows is written
// as two halves.  Beside that
// the threads write the frame itself as float into `frame` (if any), for the refinement:
// 2 us at 1024x436 where a launch of its own took 4 to 6.  (Extra blocks for it: as fast
// on large frames, 4 us slower on small ones.)
template <int UP_R, bool KEYS>
__global__ void __launch_bounds__(TX * TY, 2) k_upsample_pad_rows(const uint8_t* __restrict__ in, float* __restrict__ frame,
                                                               float* __restrict__ out,
                                                               uint32_t* __restrict__ keys, int pitch, int m, int sxi,
                                                               int syi, int sxo, int syo,
                                                               const float* __restrict__ lx, const int* __restrict__ ix,
                                                               const float* __restrict__ ly, const int* __restrict__ iy)
{
    chain_trigger();   // launched unchained: what is older is complete
    const int X = blockIdx.x * TX + threadIdx.x;
    const int Y0 = (blockIdx.y * TY + threadIdx.y) * UP_R;
    if (frame) {
        const size_t n = (size_t)sxi * syi, threads = (size_t)gridDim.x * gridDim.y * (TX * TY);
        const size_t block = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
        for (size_t i = block * (TX * TY) + threadIdx.y * TX + threadIdx.x; i < n; i += threads) frame[i] = (float)in[i];
    }
    if (X >= sxo + 2 * m || Y0 >= syo + 2 * m) return;
    const int x = min(sxo - 1, max(0, X - m));
    const int x1 = __ldg(ix + x);
    float Lx[6];
    int col[6];
#pragma unroll
    for (int a = 0; a < 6; a++) {
        Lx[a] = __ldg(lx + x * 6 + a);
        col[a] = min(sxi - 1, max(0, x1 - 2 + a));
    }
    float P[6][6];  // P[a][b] = in[row b of the window][col a] * Lx[a]
    auto products = [&](int win, int b) {
        const uint8_t* src = in + (size_t)min(syi - 1, max(0, win - 2 + b)) * sxi;
#pragma unroll
        for (int a = 0; a < 6; a++) P[a][b] = __fmul_rn((float)__ldg(src + col[a]), Lx[a]);
    };
    int win = __ldg(iy + min(syo - 1, max(0, Y0 - m)));   // uniform across the warp
#pragma unroll
    for (int b = 0; b < 6; b++) products(win, b);
    float v[UP_R], w[UP_R];
#pragma unroll
    for (int r = 0; r < UP_R; r++) {
        const int y = min(syo - 1, max(0, Y0 + r - m));
        for (const int y1 = __ldg(iy + y); win < y1;) {   // windows only move down
            win++;
#pragma unroll
            for (int a = 0; a < 6; a++)
#pragma unroll
                for (int b = 0; b < 5; b++) P[a][b] = P[a][b + 1];
            products(win, 5);
        }
        float Ly[6];
#pragma unroll
        for (int b = 0; b < 6; b++) Ly[b] = __ldg(ly + y * 6 + b);
        v[r] = w[r] = 0.0f;
#pragma unroll
        for (int a = 0; a < 6; a++)
#pragma unroll
            for (int b = 0; b < 6; b++) {
                w[r] = __fmaf_rn(Lx[a], Ly[b], w[r]);
                v[r] = __fmaf_rn(P[a][b], Ly[b], v[r]);
            }
    }
    uint32_t key_above = 0;
#pragma unroll
    for (int r = 0; r < UP_R; r++) {
        const int Y = Y0 + r;
        if (Y >= syo + 2 * m) break;
        const float val = v[r] / w[r];
        const size_t o = X + (size_t)Y * pitch;
        out[o] = val;
        const uint32_t key = sample_key(val);
        if constexpr (!KEYS) continue;
        if (r > 0)
            keys[o - pitch] = key_above | (key << 16);
        else if (Y > 0)
            reinterpret_cast<uint16_t*>(keys + (o - pitch))[1] = (uint16_t)key;
        if (r == UP_R - 1 || Y == syo + 2 * m - 1) reinterpret_cast<uint16_t*>(keys + o)[0] = (uint16_t)key;
        key_above = key;
    }
}

__global__ void k_u8_to_f32(const uint8_t* __restrict__ in, float* __restrict__ out, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)in[i];
}


// BRIEF descriptors: interior tiles read the linear offsets from the kernel's
// parameter space (fully unrolled, immediate operands); border tiles stage the
// pattern in shared memory and clamp.
template <int NSP>
__global__ void __launch_bounds__(256) k_features(const float* __restrict__ I, uint32_t* __restrict__ F,
                                                  int sx, int sy, int N, const int4* __restrict__ pat, int rmax,
                                                  const __grid_constant__ PatternOffsets po, int rev)
{
    __shared__ int4 s_pat[BM_PATCH_MAX / 4];
    const int2 t0 = block_tile(rev);
    const int x = t0.x + threadIdx.x, y = t0.y + threadIdx.y;
    if (tile_interior(t0.x, t0.y, sx, sy, rmax)) {
        features_interior_px<NSP>(I, F, sx, x, y, po.off);
    } else {
        const int tid = threadIdx.y * TX + threadIdx.x;
        for (int k = tid; k < N; k += TX * TY) s_pat[k] = pat[k];
        __syncthreads();
        if (x >= sx || y >= sy) return;
        features_border_px<NSP>(I, F, sx, sy, N, s_pat, x, y);
    }
}

// BRIEF descriptors from the key image of an edge-replicated frame (k_upsample_pad_rows)
// whose margin is at least the pattern's largest offset: every pixel reads at the
// linear offsets (no clamping, no border tiles).  A thread takes the pixels (x, y) and
// (x, y + 1): one key word per sample serves both.
//
// Per sample pair, four half-precision instructions: `set.gt` and `set.eq` (1.0 or 0.0
// per half) and an FMA each that shifts the result into an accumulator
// (acc = 2 acc + bit; from 4.0, eight results leave 1024 + their byte, exact in a
// half).  Equal keys do not say which sample is larger: those pairs (and only those)
// are compared again on the float image, so every bit is the float comparison's.
// Samples whose two points coincide (and the padding past N) are equal by construction;
// their bits are masked out of that by the pattern (po.differ).  On textured frames one
// pair in a thousand ties and each lane repairs its own; saturated or flat parts tie
// throughout, and there (a lane with more than MANY_TIES) the warp goes sample by
// sample, and past FLAT_TIES samples of a word reads the next words of the chunk from
// the float image outright.
//
// Reading two keys per 4 bytes halves the load requests that bound the float form
// (70 % of the load unit's rate, and 13 % of its instructions branches around the
// strip's end): 144 -> 99 us at 2969x1264 N128, 280 -> 191 at N256, 980 -> 557 at
// 3136x1764 N512.  What bounds it now is issue; without the ties' repair and detection
// it would be 68 us at N128.  Measured beside it: four pixels per thread (32 columns
// on, sharing the addresses) 101, 203 and 606 us, its code twice as long for the
// instruction cache; all sixteen words of N512 unrolled 17 % slower; a repair that
// always goes sample by sample 102 and 575.  Six blocks per SM (40 registers) measured
// 1-3 % better than five, seven or eight.
constexpr int FLAT_TIES = 12, MANY_TIES = 12;
template <int NSP>
__global__ void __launch_bounds__(256, 6) k_features_keys(const uint32_t* W, const float* I,
                                                          int pitch, uint32_t* __restrict__ F, int sx, int sy,
                                                          const __grid_constant__ KeyOffsets po, int rev)
{
    chain_wait();
    chain_trigger();
    int bx = blockIdx.x, by = blockIdx.y;
    if (rev) {
        bx = gridDim.x - 1 - bx;
        by = gridDim.y - 1 - by;
    }
    const int x = bx * TX + threadIdx.x;
    const int y = 2 * (by * TY + threadIdx.y);
    const bool inside = x < sx && y < sy;
    const unsigned int warp = __ballot_sync(0xffffffffu, inside);
    if (!inside) return;
    // the pixel less the margin; each sample adds an unsigned 32-bit byte offset
    const size_t origin = (size_t)y * pitch + x;
    const char* base = reinterpret_cast<const char*>(W + origin);
    const char* fbase = reinterpret_cast<const char*>(I + origin);
    const size_t down = (size_t)pitch * sizeof(float);
    const bool second = y + 1 < sy;
    // sample b of word w of pixel v on the float image
    auto larger = [&](uint2 o, int v) {
        const char* f = fbase + v * down;
        return *reinterpret_cast<const float*>(f + o.x) > *reinterpret_cast<const float*>(f + o.y);
    };
    auto compare = [&](int w, int b, const uint32_t (&ask)[2], uint32_t (&bits)[2]) {
        const uint2 o = po.off[w * 32 + b];
#pragma unroll
        for (int v = 0; v < 2; v++)
            if ((ask[v] >> b & 1u) && larger(o, v)) bits[v] |= 1u << b;
    };
    constexpr int CW = NSP < 4 ? NSP : 4;   // words formed before they are stored
#pragma unroll 1
    for (int c = 0; c < NSP / CW; c++) {
        uint32_t word[2][CW];
        bool flat = false;
#pragma unroll
        for (int wd = 0; wd < CW; wd++) {
            const int w = c * CW + wd;
            uint32_t bits[2], ask[2];
            if (flat) {
                bits[0] = bits[1] = 0;
                ask[0] = 0xffffffffu;
                ask[1] = second ? 0xffffffffu : 0;
#pragma unroll 4
                for (int b = 0; b < 32; b++) compare(w, b, ask, bits);
            } else {
                uint32_t gt[4], eq[4];
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    gt[g] = eq[g] = 0x44004400u;     // 4.0, 4.0
#pragma unroll
                    for (int b = 7; b >= 0; b--) {   // the byte's low bit is its first sample
                        const uint2 o = po.off[w * 32 + g * 8 + b];
                        const uint32_t k1 = *reinterpret_cast<const uint32_t*>(base + o.x);
                        const uint32_t k2 = *reinterpret_cast<const uint32_t*>(base + o.y);
                        gt[g] = half2_shift_in(gt[g], half2_gt(k1, k2));
                        eq[g] = half2_shift_in(eq[g], half2_eq(k1, k2));
                    }
                }
                half2_bytes(gt, bits[0], bits[1]);
                half2_bytes(eq, ask[0], ask[1]);
                ask[0] &= po.differ[w];
                ask[1] = second ? ask[1] & po.differ[w] : 0;
                if (__any_sync(warp, max(__popc(ask[0]), __popc(ask[1])) > MANY_TIES)) {
                    uint32_t any = __reduce_or_sync(warp, ask[0] | ask[1]);
                    flat = __popc(any) > FLAT_TIES;
                    while (any) {
                        const int b = __ffs(any) - 1;
                        any &= any - 1;
                        compare(w, b, ask, bits);
                    }
                } else {
#pragma unroll
                    for (int v = 0; v < 2; v++)
                        while (ask[v]) {
                            const int b = __ffs(ask[v]) - 1;
                            ask[v] &= ask[v] - 1;
                            if (larger(po.off[w * 32 + b], v)) bits[v] |= 1u << b;
                        }
                }
            }
            word[0][wd] = bits[0];
            word[1][wd] = bits[1];
        }
        store_desc<CW>(F + ((size_t)y * sx + x) * NSP + c * CW, word[0]);
        if (second) store_desc<CW>(F + ((size_t)(y + 1) * sx + x) * NSP + c * CW, word[1]);
    }
}

// The same without a key image (memory is short): every pair on the float image.  A kernel
// of its own, as another branch to the float image costs the one above 1-3 % of its time.
template <int NSP>
__global__ void __launch_bounds__(256) k_features_float(const float* I, int pitch, uint32_t* __restrict__ F, int sx, int sy,
                                                        const __grid_constant__ KeyOffsets po, int rev)
{
    chain_wait();
    chain_trigger();
    int bx = blockIdx.x, by = blockIdx.y;
    if (rev) {
        bx = gridDim.x - 1 - bx;
        by = gridDim.y - 1 - by;
    }
    const int x = bx * TX + threadIdx.x, y = by * TY + threadIdx.y;
    if (x >= sx || y >= sy) return;
    const char* base = reinterpret_cast<const char*>(I + ((size_t)y * pitch + x));
    uint32_t* out = F + ((size_t)y * sx + x) * NSP;
#pragma unroll 1
    for (int w = 0; w < NSP; w++) {
        uint32_t bits = 0;
#pragma unroll
        for (int b = 0; b < 32; b++) {
            const uint2 o = po.off[w * 32 + b];
            if (*reinterpret_cast<const float*>(base + o.x) > *reinterpret_cast<const float*>(base + o.y)) bits |= 1u << b;
        }
        out[w] = bits;
    }
}

// CHAINED (k_seed alike): the launch before may be writing the descriptors (init_px); else
// they are read through L1: 9408x5292 N512 922 us instead of 958, its seed 1204 instead of 1282.
template <int NSP, bool CHAINED>
__global__ void __launch_bounds__(256) k_initialize(const uint32_t* F1, const uint32_t* F2,
                                                    const uint32_t* __restrict__ flow_prev, uint32_t* __restrict__ flow_out,
                                                    uint16_t* __restrict__ cost, int sx, int sy, int first, int rev)
{
    const int2 t0 = block_tile(rev);
    const int x = t0.x + threadIdx.x, y = t0.y + threadIdx.y;
    chain_wait();
    chain_trigger();
    if (x >= sx || y >= sy) return;
    init_px<NSP, CHAINED>(F1, F2, flow_prev, flow_out, cost, sx, sy, first, x, y);
}

template <int NSP, bool CHAINED>
__global__ void __launch_bounds__(256) k_seed(const uint32_t* F1, const uint32_t* F2,
                                              const uint32_t* __restrict__ flow_prev, uint32_t* __restrict__ flow_out,
                                              uint16_t* __restrict__ cost, int sx, int sy, int first,
                                              const float* __restrict__ pred, int w4, int h4, float scale_x,
                                              float scale_y, float inv_x, float inv_y, float logit_min)
{
    const int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
    chain_wait();
    chain_trigger();
    if (x >= sx || y >= sy) return;
    seed_px<NSP, CHAINED>(F1, F2, flow_prev, flow_out, cost, sx, sy, first, x, y, pred, w4, h4, scale_x, scale_y, inv_x, inv_y,
                 logit_min);
}

// Blocks per SM the level is compiled for (its time falls with the loads in flight up
// to the line where registers spill into them): 5 for 32- and 64-byte descriptors (at
// N512, 3136x1764: 156 us uncapped at 100 registers, 132 at 5 blocks, 156 at 6), 6 with
// the random search (229 us at 5 blocks, 217 at 6).
template <int NSP, bool RS>
__host__ __device__ constexpr int jump_blocks() { return NSP <= 4 ? (RS ? 6 : 8) : (NSP == 16 && RS ? 6 : 5); }
template <int NSP, bool RS>
__global__ void __launch_bounds__(256, (jump_blocks<NSP, RS>())) k_jump_level(const uint32_t* __restrict__ F1, const uint32_t* __restrict__ F2,
                                                    const uint32_t* flow_in, uint32_t* flow_out, uint16_t* cost,
                                                    int sx, int sy, int p, int pd, int doubleProp, RsArgs rs, int rev)
{
    const int2 t0 = block_tile(rev);
    const int x = t0.x + threadIdx.x, y = t0.y + threadIdx.y;
    chain_wait();
    chain_trigger();
    jump_level_px<NSP, RS, true>(F1, F2, flow_in, flow_out, cost, sx, sy, p, pd, doubleProp, rs, x, y);
}

template <int NSP>
__global__ void __launch_bounds__(256) k_local_step(const uint32_t* __restrict__ F1, const uint32_t* __restrict__ F2,
                                                    const uint32_t* flow_in, uint32_t* flow_out, uint16_t* cost,
                                                    int sx, int sy, int r, int rev)
{
    const int2 t0 = block_tile(rev);
    const int x = t0.x + threadIdx.x, y = t0.y + threadIdx.y;
    chain_wait();
    chain_trigger();
    if (x >= sx || y >= sy) return;
    local_px<NSP>(F1, F2, flow_in, flow_out, cost, sx, sy, r, x, y);
}

template <int NSP>
__global__ void __launch_bounds__(256) k_random_search(const uint32_t* __restrict__ F1, const uint32_t* __restrict__ F2,
                                                       uint32_t* __restrict__ flow, uint16_t* __restrict__ cost,
                                                       int sx, int sy, RsArgs rs)
{
    const int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
    if (x >= sx || y >= sy) return;
    const long pix = x + (long)y * sx;
    const uint32_t own = flow[pix];
    const int cx = lo16(own), cy = hi16(own);
    float n1, n2;
    rs_normals(rs, (unsigned int)pix, n1, n2);
    const int nx = min(max((int)round(rs.dist * n1), -x), sx - x - 1);
    const int ny = min(max((int)round(rs.dist * n2), -y), sy - y - 1);
    if (nx == cx && ny == cy) return;
    uint32_t f1[NSP];
    load_desc<NSP>(f1, F1 + pix * NSP);
    const int hc = hamming<NSP>(f1, F2 + (pix + nx + (long)ny * sx) * NSP);
    if (hc < cost[pix]) {
        cost[pix] = (uint16_t)hc;
        flow[pix] = pack_flow(nx, ny);
    }
}

__global__ void k_normals(float2* __restrict__ out, int sx, int sy, RsArgs rs)
{
    const int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
    if (x >= sx || y >= sy) return;
    const long pix = x + (long)y * sx;
    float n1, n2;
    rs_normals(rs, (unsigned int)pix, n1, n2);
    out[pix] = make_float2(n1, n2);
}

// resizeNN's source index, util_cuda.cu:165-166 (sxi = up-sampled size, sxo = input size),
// tabulated per output column / row with the reference's expression.
__global__ void k_nn_table(unsigned int* __restrict__ idx, int n_up, int n_in)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n_in) return;
    unsigned int x1 = round(x * float(n_up) / n_in);
    idx[x] = x1;
}


__global__ void __launch_bounds__(256) k_downsample(const uint32_t* flow, float* __restrict__ U,
                                                    float* __restrict__ V, int sx, int sy, int sx_in, int sy_in,
                                                    const float* __restrict__ taps, int P, float mx, float my,
                                                    const unsigned int* __restrict__ nnx,
                                                    const unsigned int* __restrict__ nny, int rows)
{
    chain_wait();
    chain_trigger();
    extern __shared__ float2 down_h[];
    downsample_block(flow, U, V, sx, sy, sx_in, sy_in, taps, P, mx, my, nnx, nny, blockIdx.x * TX, blockIdx.y * rows,
                     rows, down_h);
}
// Small frames, and scales whose window does not fit shared memory.
__global__ void __launch_bounds__(256) k_downsample_px(const uint32_t* flow, float* __restrict__ U,
                                                       float* __restrict__ V, int sx, int sy, int sx_in, int sy_in,
                                                       const float* __restrict__ taps, int P, float mx, float my,
                                                       const unsigned int* __restrict__ nnx,
                                                       const unsigned int* __restrict__ nny)
{
    chain_wait();
    chain_trigger();
    const int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
    if (x >= sx_in || y >= sy_in) return;
    downsample_px(flow, U, V, sx, sy, sx_in, taps, P, mx, my, nnx, nny, x, y);
}

// CUDA_convert, util_cuda.cu:174-183, for both components when no resampling is needed.
__global__ void k_flow_to_planes(const uint32_t* flow, float* __restrict__ U, float* __restrict__ V, size_t n)
{
    chain_wait();
    chain_trigger();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t f = flow[i];
    U[i] = (float)lo16(f);
    V[i] = (float)hi16(f);
}


// Separable 1-D median, both components in one launch (blockIdx.z).  Each thread
// computes two outputs adjacent along the filter direction (median2_px): down a
// column (dir 0) the rows y and y+1; along the rows (dir 1) the linear indices 2t and
// 2t+1 (the reference's window runs over linear indices, so a pair may span a row
// end).
template <int FS>
__global__ void __launch_bounds__(256) k_median_pass(const float* inU, const float* inV,
                                                     float* __restrict__ outU, float* __restrict__ outV,
                                                     int dir, int fsize, int sx, int sy)
{
    static_assert(FS % 2 == 1, "median register windows are odd");
    chain_wait();
    chain_trigger();
    const float* in = blockIdx.z ? inV : inU;
    float* out = blockIdx.z ? outV : outU;
    const long n = (long)sx * sy;
    if (dir) {
        const long p = 2 * ((long)blockIdx.x * (TX * TY) + threadIdx.y * TX + threadIdx.x);
        if (p >= n) return;
        median2_px<FS>(in, out, p, 1, n, fsize, p + 1 < n);
    } else {
        const int x = blockIdx.x * TX + threadIdx.x, y = 2 * (blockIdx.y * TY + threadIdx.y);
        if (x >= sx || y >= sy) return;
        median2_px<FS>(in, out, x + (long)y * sx, sx, n, fsize, y + 1 < sy);
    }
}

template <int TY, int G>
__global__ void __launch_bounds__(TX * TY * G, 16 / (TY * G)) k_trilateral(const float* __restrict__ U,
                                                                       const float* __restrict__ V,
                                                                       const float* Um,
                                                                       const float* Vm,
                                                                       const float* __restrict__ I,
                                                                       float* __restrict__ Uo, float* __restrict__ Vo,
                                                                       int sx, int sy, int s,
                                                                       const __grid_constant__ TriCoef tc)
{
    chain_wait();
    chain_trigger();
    extern __shared__ float4 smem4[];
    trilateral_block<TY, G>(U, V, Um, Vm, I, Uo, Vo, sx, sy, s, tc, blockIdx.x * TX, blockIdx.y * tri_rows(TY), smem4);
}

__global__ void __launch_bounds__(256) k_trilateral_global(const float* __restrict__ U, const float* __restrict__ V,
                                                           const float* Um, const float* Vm,
                                                           const float* __restrict__ I, float* __restrict__ Uo,
                                                           float* __restrict__ Vo, int sx, int sy, int s,
                                                           float cE, float cI, float cS)
{
    chain_wait();
    chain_trigger();
    const int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
    if (x >= sx || y >= sy) return;
    const size_t o = (size_t)x + (size_t)y * sx;
    const float um0 = Um[o], vm0 = Vm[o], I0 = I[o];
    // sums of the differences to the centre, as trilateral_block's; of the flow itself where
    // that is far or NaN (an empty window gives 0 all the same)
    const bool far_u = !(fabsf(um0) <= TRI_FAR), far_v = !(fabsf(vm0) <= TRI_FAR);
    float uf = 0.0f, vf = 0.0f, W = 0.0f;
    auto walk = [&](auto flow) {
        constexpr bool FLOW = decltype(flow)::value;
        for (int i = -s; i < s; i++) {
            const int gx = min(sx - 1, max(0, x + i));
            const float si = (float)(i * i) * cS;
            for (int j = -s; j < s; j++) {
                const size_t g = (size_t)gx + (size_t)min(sy - 1, max(0, y + j)) * sx;
                const float u1 = __ldg(U + g), v1 = __ldg(V + g);
                const float dI = __ldg(I + g) - I0;
                const float du = u1 - um0, dv = v1 - vm0;
                const float e = du * du + dv * dv;
                const float sp = si + (float)(j * j) * cS;
                const float w = exp2f(fmaf(e, -cE, fmaf(dI * dI, -cI, -sp)));
                uf = fmaf(w, FLOW && far_u ? u1 : du, uf);
                vf = fmaf(w, FLOW && far_v ? v1 : dv, vf);
                W += w;
            }
        }
    };
    walk(std::false_type{});
    if (far_u || far_v) {
        uf = vf = W = 0.0f;
        walk(std::true_type{});
    }
    const float bu = far_u ? 0.0f : um0, bv = far_v ? 0.0f : vm0;
    Uo[o] = W < 1e-5f ? fmaf(bu, W, uf) / 1e-5f : bu + uf / W;
    Vo[o] = W < 1e-5f ? fmaf(bv, W, vf) / 1e-5f : bv + vf / W;
}

// ---------------------------------------------------------------------------
// Reference-layout export/import (briefmatch.h:139-141).
// ---------------------------------------------------------------------------
__global__ void k_export_field(const uint32_t* __restrict__ flow, const uint16_t* __restrict__ cost,
                               int16_t* __restrict__ nx, int16_t* __restrict__ ny, float* __restrict__ dist,
                               size_t n, int N)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t f = flow[i];
    if (nx) nx[i] = (int16_t)lo16(f);
    if (ny) ny[i] = (int16_t)hi16(f);
    // featDist's return value, briefmatch_cuda.cu:79
    if (dist) dist[i] = float((int)cost[i]) / N;
}

__global__ void k_import_field(const int16_t* __restrict__ nx, const int16_t* __restrict__ ny,
                               const uint16_t* __restrict__ cost_in, uint32_t* __restrict__ flow,
                               uint16_t* __restrict__ cost, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    flow[i] = pack_flow(nx[i], ny[i]);
    if (cost_in) cost[i] = cost_in[i];
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
// SMs of the current device.
static cudaError_t sm_count(int* sms)
{
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    return e == cudaSuccess ? cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) : e;
}

// Launch of a kernel that waits for its predecessor itself (chain_wait); `chained`: that
// predecessor is the kernel launched last on the stream, and this one may start under its
// last blocks.
template <typename Kernel, typename... Args>
static cudaError_t launch(Kernel kernel, dim3 grid, dim3 block, size_t smem, bool chained, cudaStream_t st, Args... args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t lanczos_tables(float* w, int* idx, int n_in, int n_out, cudaStream_t st)
{
    k_lanczos_tables<<<(n_out + 127) / 128, 128, 0, st>>>(w, idx, n_in, n_out);
    return cudaGetLastError();
}

cudaError_t upsample_f32(const float* in, float* out, int sxi, int syi, int sxo, int syo,
                         const float* lx, const int* ix, const float* ly, const int* iy, cudaStream_t st)
{
    k_upsample<float><<<grid2d(sxo, syo), dim3(TX, TY), 0, st>>>(in, out, sxi, syi, sxo, syo, lx, ix, ly, iy);
    return cudaGetLastError();
}

cudaError_t upsample_u8(const uint8_t* in, float* out, int sxi, int syi, int sxo, int syo,
                        const float* lx, const int* ix, const float* ly, const int* iy, cudaStream_t st)
{
    k_upsample<uint8_t><<<grid2d(sxo, syo), dim3(TX, TY), 0, st>>>(in, out, sxi, syi, sxo, syo, lx, ix, ly, iy);
    return cudaGetLastError();
}

cudaError_t upsample_u8_pad(const uint8_t* in, float* frame, float* out, uint32_t* keys, int pitch, int m, int sxi, int syi, int sxo,
                            int syo, const float* lx, const int* ix, const float* ly, const int* iy, cudaStream_t st)
{
    if (m < 0 || pitch < sxo + 2 * m) return cudaErrorInvalidValue;
    // Eight rows a thread share the most products; a grid of fewer blocks than SMs takes
    // four or two rows a thread and with them less time for its chain of rows (96x64 u1.5:
    // 10.6 us with eight, 8.8 and 7.2 with four and two, 7.3 with one; 1024x436 u2.9 39.4,
    // 43.6, 56.2, 1920x1080 u4.9 394, 492, 662).
    int sms = 0;
    const cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) return e;
    auto rows = [&](auto kernel, int r) {
        const dim3 g((sxo + 2 * m + TX - 1) / TX, (syo + 2 * m + TY * r - 1) / (TY * r));
        kernel<<<g, dim3(TX, TY), 0, st>>>(in, frame, out, keys, pitch, m, sxi, syi, sxo, syo, lx, ix, ly, iy);
    };
    const long columns = (sxo + 2 * m + TX - 1) / TX, eights = (syo + 2 * m + TY - 1) / TY;
    if (!keys) rows(k_upsample_pad_rows<8, false>, 8);   // memory is short
    else if (columns * eights >= 8L * sms) rows(k_upsample_pad_rows<8, true>, 8);
    else if (columns * eights >= 4L * sms) rows(k_upsample_pad_rows<4, true>, 4);
    else rows(k_upsample_pad_rows<2, true>, 2);
    return cudaGetLastError();
}

cudaError_t u8_to_f32(const uint8_t* in, float* out, size_t n, cudaStream_t st)
{
    k_u8_to_f32<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}

#define BM_DISPATCH_NSP(nsp, ...)                          \
    switch (nsp) {                                         \
    case 1: { constexpr int NSP = 1; __VA_ARGS__; } break;   \
    case 2: { constexpr int NSP = 2; __VA_ARGS__; } break;   \
    case 4: { constexpr int NSP = 4; __VA_ARGS__; } break;   \
    case 8: { constexpr int NSP = 8; __VA_ARGS__; } break;   \
    case 16: { constexpr int NSP = 16; __VA_ARGS__; } break; \
    default: return cudaErrorInvalidValue;                 \
    }

cudaError_t features(const float* up, uint32_t* F, int sx, int sy, int N, int nsp,
                     const int4* pat, int rmax, const PatternOffsets& po, int rev, cudaStream_t st)
{
    BM_DISPATCH_NSP(nsp, k_features<NSP><<<grid2d(sx, sy), dim3(TX, TY), 0, st>>>(up, F, sx, sy, N, pat, rmax, po, rev));
    return cudaGetLastError();
}

bool key_image_fits(int m, int pitch) { return (2 * (size_t)m + 1) * (size_t)pitch < ((size_t)1 << 30); }

void key_offsets(KeyOffsets& ko, const int4* pat, int N, int m, int pitch)
{
    std::memset(&ko, 0, sizeof(ko));
    auto at = [&](int dx, int dy) { return (uint32_t)((size_t)(dy + m) * pitch + (dx + m)) * 4u; };
    for (int s = 0; s < BM_PATCH_MAX / 4; s++) {
        const int4 q = s < N ? pat[s] : make_int4(0, 0, 0, 0);
        ko.off[s] = make_uint2(at(q.x, q.y), at(q.z, q.w));
        if (ko.off[s].x != ko.off[s].y) ko.differ[s / 32] |= 1u << (s % 32);
    }
}

cudaError_t features_keys(const uint32_t* keys, const float* up, int pitch, uint32_t* F, int sx, int sy, int nsp,
                          const KeyOffsets& ko, int rev, bool chained, cudaStream_t st)
{
    if (!keys) {
        BM_DISPATCH_NSP(nsp, return launch(k_features_float<NSP>, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, up, pitch, F, sx, sy, ko, rev));
    }
    const dim3 g((sx + TX - 1) / TX, (sy + 2 * TY - 1) / (2 * TY));
    BM_DISPATCH_NSP(nsp, return launch(k_features_keys<NSP>, g, dim3(TX, TY), 0, chained, st, keys, up, pitch, F, sx, sy, ko, rev));
    return cudaSuccess;
}

cudaError_t initialize(const uint32_t* F1, const uint32_t* F2, const uint32_t* flow_prev,
                       uint32_t* flow_out, uint16_t* cost, int sx, int sy, int nsp, int first, int rev,
                       bool chained, cudaStream_t st)
{
    if (chained) {
        BM_DISPATCH_NSP(nsp, return launch(k_initialize<NSP, true>, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, F1, F2, flow_prev, flow_out, cost, sx, sy, first, rev));
    }
    BM_DISPATCH_NSP(nsp, return launch(k_initialize<NSP, false>, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, F1, F2, flow_prev, flow_out, cost, sx, sy, first, rev));
    return cudaSuccess;
}

cudaError_t seed_field(const uint32_t* F1, const uint32_t* F2, const uint32_t* flow_prev, uint32_t* flow_out,
                       uint16_t* cost, int sx, int sy, int nsp, int first, const float* pred, int w4, int h4,
                       float scale_x, float scale_y, float logit_min, bool chained, cudaStream_t st)
{
    // host IEEE reciprocals: the device cell lookup multiplies by them
    const float inv_x = 1.0f / scale_x, inv_y = 1.0f / scale_y;
    if (chained) {
        BM_DISPATCH_NSP(nsp, return launch(k_seed<NSP, true>, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, F1, F2, flow_prev, flow_out, cost, sx, sy, first, pred, w4, h4, scale_x, scale_y, inv_x, inv_y, logit_min));
    }
    BM_DISPATCH_NSP(nsp, return launch(k_seed<NSP, false>, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, F1, F2, flow_prev, flow_out, cost, sx, sy, first, pred, w4, h4, scale_x, scale_y, inv_x, inv_y, logit_min));
    return cudaSuccess;
}

cudaError_t jump_level(const uint32_t* F1, const uint32_t* F2, const uint32_t* flow_in,
                       uint32_t* flow_out, uint16_t* cost, int sx, int sy, int nsp,
                       int p, int pd, int doubleProp, const RsArgs& rs, int rev, bool chained, cudaStream_t st)
{
    if (rs.enabled) {
        BM_DISPATCH_NSP(nsp, return launch(k_jump_level<NSP, true>, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, F1, F2, flow_in, flow_out, cost, sx, sy, p, pd, doubleProp, rs, rev));
    } else {
        BM_DISPATCH_NSP(nsp, return launch(k_jump_level<NSP, false>, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, F1, F2, flow_in, flow_out, cost, sx, sy, p, pd, doubleProp, rs, rev));
    }
    return cudaSuccess;
}

cudaError_t local_step(const uint32_t* F1, const uint32_t* F2, const uint32_t* flow_in, uint32_t* flow_out,
                       uint16_t* cost, int sx, int sy, int nsp, int r, int rev, bool chained, cudaStream_t st)
{
    BM_DISPATCH_NSP(nsp, return launch(k_local_step<NSP>, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, F1, F2, flow_in, flow_out, cost, sx, sy, r, rev));
    return cudaSuccess;
}

cudaError_t random_search(const uint32_t* F1, const uint32_t* F2, uint32_t* flow, uint16_t* cost,
                          int sx, int sy, int nsp, const RsArgs& rs, cudaStream_t st)
{
    BM_DISPATCH_NSP(nsp, k_random_search<NSP><<<grid2d(sx, sy), dim3(TX, TY), 0, st>>>(F1, F2, flow, cost, sx, sy, rs));
    return cudaGetLastError();
}

cudaError_t normals(float2* out, int sx, int sy, const RsArgs& rs, cudaStream_t st)
{
    k_normals<<<grid2d(sx, sy), dim3(TX, TY), 0, st>>>(out, sx, sy, rs);
    return cudaGetLastError();
}

cudaError_t nn_table(unsigned int* idx, int n_up, int n_in, cudaStream_t st)
{
    k_nn_table<<<(n_in + 127) / 128, 128, 0, st>>>(idx, n_up, n_in);
    return cudaGetLastError();
}

cudaError_t downsample(const uint32_t* flow, float* U, float* V, int sx, int sy, int sx_in, int sy_in,
                       const float* taps, int P, float mx, float my, const unsigned int* nnx,
                       const unsigned int* nny, bool chained, cudaStream_t st)
{
    // By blocks of 32 rows, or as many as fit the 48 KB that need no opt-in, for windows
    // of 16 taps and more where those give every SM two blocks: 1920x1080 u4.9, 19 taps,
    // 426 us per pixel, 184 by blocks.  With few taps a pass per pixel is as fast
    // (1024x436 u2.9, 7 taps: 22.5 and 21.5; 584x388 u1.5, 3 taps: 8.2 and 8.8), and it does
    // not change the SMs' split between L1 and shared memory: blocks from 11 taps on made
    // a batch of 12 pairs on several streams 0.8 % slower.
    int sms = 0;
    const cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) return e;
    int rows = 4 * TY;
    while (rows > TY && down_smem_bytes(rows, sy, sy_in, P) > DOWN_SMEM_MAX) rows /= 2;
    const size_t smem = down_smem_bytes(rows, sy, sy_in, P);
    if (P < 16 || smem > DOWN_SMEM_MAX || (long)((sx_in + TX - 1) / TX) * ((sy_in + 4 * TY - 1) / (4 * TY)) < 2L * sms)
        return launch(k_downsample_px, grid2d(sx_in, sy_in), dim3(TX, TY), 0, chained, st, flow, U, V, sx, sy, sx_in, sy_in,
                      taps, P, mx, my, nnx, nny);
    return launch(k_downsample, dim3((sx_in + TX - 1) / TX, (sy_in + rows - 1) / rows), dim3(TX, TY), smem, chained, st,
                  flow, U, V, sx, sy, sx_in, sy_in, taps, P, mx, my, nnx, nny, rows);
}

cudaError_t flow_to_planes(const uint32_t* flow, float* U, float* V, size_t n, bool chained, cudaStream_t st)
{
    return launch(k_flow_to_planes, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, chained, st, flow, U, V, n);
}

cudaError_t median_pass(const float* inU, const float* inV, float* outU, float* outV,
                        int dir, int fsize, int sx, int sy, bool chained, cudaStream_t st)
{
    const long n = (long)sx * sy;
    const dim3 g = dir ? dim3((unsigned)((n + 2 * TX * TY - 1) / (2 * TX * TY)), 1, 2)
                       : dim3((sx + TX - 1) / TX, (sy + 2 * TY - 1) / (2 * TY), 2);
#define BM_MED(FSV) return launch(k_median_pass<FSV>, g, dim3(TX, TY), 0, chained, st, inU, inV, outU, outV, dir, fsize, sx, sy)
    if (fsize <= 9) BM_MED(9);
    else if (fsize <= 13) BM_MED(13);
    else if (fsize <= 15) BM_MED(15);
    else if (fsize <= 23) BM_MED(23);
    else if (fsize <= 31) BM_MED(31);
    else if (fsize <= BM_MAX_MEDIAN) BM_MED(BM_MAX_MEDIAN);
#undef BM_MED
    return cudaErrorInvalidValue;
}

// The trilateral kernel's dynamic shared-memory opt-in, raised only when a larger
// window than any before needs it (so launches after the first of a size make no
// attribute call and can be captured in a graph).  The opt-in only ever grows, under
// a lock: contexts created on several host threads never lower it below what another
// thread's launch was checked against.
cudaError_t ensure_trilateral_smem(int s)
{
    static std::mutex mu;
    static int granted[64] = {0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    const int need = (int)tri_smem_bytes(s, 8);
    std::lock_guard<std::mutex> lock(mu);
    if (need <= granted[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(k_trilateral<8, TRI_G>, cudaFuncAttributeMaxDynamicSharedMemorySize, need);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_trilateral<4, TRI_G>, cudaFuncAttributeMaxDynamicSharedMemorySize, need);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_trilateral<2, TRI_G>, cudaFuncAttributeMaxDynamicSharedMemorySize, need);
    if (e == cudaSuccess) granted[dev] = need;
    return e;
}

// Thread rows per block.  A block of 8 (16 warps, an SM's registers) has the smallest
// halo per output and is the fastest wherever the grid is several waves deep; below two
// 32 x 32 tiles per SM the waves' rounding costs more than the halo, and smaller blocks,
// as many per SM as fill it, take over while their tiles fit side by side (584x388:
// 109 -> 101 us with the median, 777x333: 93 -> 88; but 1024x436, 2.9 tiles per SM: 358 -> 369).
static int trilateral_rows(int sx, int sy, int s, int sms)
{
    const size_t per_sm = 224 * 1024;
    if ((long)((sx + TX - 1) / TX) * ((sy + 31) / 32) >= 2L * sms) return 8;
    return 4 * tri_smem_bytes(s, 2) <= per_sm ? 2 : 2 * tri_smem_bytes(s, 4) <= per_sm ? 4 : 8;
}

// Half windows up to TRI_SMALL_S on a grid several waves deep take blocks of four warps
// without the groups' exchange: a window this small is over before the next block's loads
// arrive, so four blocks share an SM (with the medians, 1920x1080, s = 2, 4 and 8: 84, 122 and
// 256 us by blocks of 8 rows, 66, 99 and 228 by these, 66, 103 and 242 with the exponent's
// factor; s = 12: 467 and 439, where the larger block is ahead from s = 16 on smaller frames).
// A half window of 1 needs no tile: four taps a pixel from memory, 42 us instead of 56.
constexpr int TRI_SMALL_S = 8;

cudaError_t trilateral(const float* U, const float* V, const float* Um, const float* Vm,
                       const float* I, float* Uo, float* Vo, int sx, int sy, int s,
                       float sigmaEPE2, float sigmaI2, float sigmaS2, bool chained, cudaStream_t st)
{
    const TriCoef tc = tri_coef(sigmaEPE2, sigmaI2, sigmaS2);
    const float cE = tc.cE, cI = tc.cI, cS = tc.cS;
    if (s > 1 && s <= TRI_MAX_S && tc.scaled) {
        cudaError_t e = ensure_trilateral_smem(s);
        if (e != cudaSuccess) return e;
        auto by_rows = [&](auto kernel, int ty, int groups) {
            dim3 g((sx + TX - 1) / TX, (sy + tri_rows(ty) - 1) / tri_rows(ty));
            return launch(kernel, g, dim3(TX, ty, groups), tri_smem_bytes(s, ty), chained, st, U, V, Um, Vm, I, Uo, Vo, sx,
                          sy, s, tc);
        };
        int sms = 0;
        e = sm_count(&sms);
        if (e != cudaSuccess) return e;
        switch (trilateral_rows(sx, sy, s, sms)) {
        case 2: return by_rows(k_trilateral<2, TRI_G>, 2, TRI_G);
        case 4: return by_rows(k_trilateral<4, TRI_G>, 4, TRI_G);
        default: return s <= TRI_SMALL_S ? by_rows(k_trilateral<4, 1>, 4, 1) : by_rows(k_trilateral<8, TRI_G>, 8, TRI_G);
        }
    }
    return launch(k_trilateral_global, grid2d(sx, sy), dim3(TX, TY), 0, chained, st, U, V, Um, Vm, I, Uo, Vo, sx, sy, s, cE,
                  cI, cS);
}

cudaError_t export_field(const uint32_t* flow, const uint16_t* cost, int16_t* nx, int16_t* ny,
                         float* dist, size_t n, int N, cudaStream_t st)
{
    k_export_field<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(flow, cost, nx, ny, dist, n, N);
    return cudaGetLastError();
}

cudaError_t import_field(const int16_t* nx, const int16_t* ny, const uint16_t* cost_in,
                         uint32_t* flow, uint16_t* cost, size_t n, cudaStream_t st)
{
    k_import_field<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nx, ny, cost_in, flow, cost, n);
    return cudaGetLastError();
}

}  // namespace bmk
