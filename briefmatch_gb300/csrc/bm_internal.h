// bm_internal.h -- engine-private declarations shared by the kernel and API units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "briefmatch_gb300.h"

namespace bmk {

// Sets the text bm_last_error() returns on this thread.
void set_error_text(const char* msg);

// The engine's device allocator (bm_alloc.cpp): cudaMalloc/cudaFree behind the test
// hooks bm_debug_fail_alloc and bm_debug_guard_bands.
cudaError_t device_malloc(void** p, size_t bytes);
// `bytes`, or `least` where the device has no room for more; *got is the one it was.
cudaError_t device_malloc_or(void** p, size_t bytes, size_t least, size_t* got);
void device_free(void* p);

// Random-search stream position for one launch (briefmatch_cuda.cu:237-241).
struct RsArgs {
    int enabled;                 // fuse a random-search candidate into the launch
    int mode;                    // BM_RNG_XORWOW or BM_RNG_PHILOX
    unsigned long long seed;     // Philox key
    unsigned long long call;     // index of this random-search call in the stream
    float dist;                  // search radius, briefmatch.cpp:271
};

// Flow words: low 16 bits nx, high 16 bits ny, both int16.
__host__ __device__ inline uint32_t pack_flow(int nx, int ny)
{
    return (uint32_t)(uint16_t)(int16_t)nx | ((uint32_t)(uint16_t)(int16_t)ny << 16);
}

// Words per descriptor in the engine layout: ceil(N/32) rounded up to 1, 2, 4, 8 or 16.
inline uint32_t feature_stride(uint32_t N)
{
    uint32_t ns = (N + 31) / 32;
    uint32_t s = 1;
    while (s < ns) s <<= 1;
    return s;
}

cudaError_t lanczos_tables(float* w, int* idx, int n_in, int n_out, cudaStream_t st);
cudaError_t upsample_f32(const float* in, float* out, int sxi, int syi, int sxo, int syo,
                         const float* lx, const int* ix, const float* ly, const int* iy, cudaStream_t st);
cudaError_t upsample_u8(const uint8_t* in, float* out, int sxi, int syi, int sxo, int syo,
                        const float* lx, const int* ix, const float* ly, const int* iy, cudaStream_t st);
// Up-sampling into an image with an edge-replicated margin of m pixels on every
// side; `out` is the start of the (sxo + 2m) x (syo + 2m) buffer, row pitch `pitch`.
// `keys`, of the same shape, receives the 16-bit keys the descriptors compare first: per
// word the pixel's key and that of the pixel below it (null: no keys).  `frame`, unless
// null, receives the input frame as float.
cudaError_t upsample_u8_pad(const uint8_t* in, float* frame, float* out, uint32_t* keys, int pitch, int m, int sxi,
                            int syi, int sxo, int syo, const float* lx, const int* ix, const float* ly, const int* iy,
                            cudaStream_t st);
cudaError_t u8_to_f32(const uint8_t* in, float* out, size_t n, cudaStream_t st);

// Linear image offsets (o1, o2) of every BRIEF sample for one image width, padded
// with zeros to a whole number of 32-bit words; passed by value as a kernel
// parameter (4 KB) so that the sample loop reads them as constants.
struct PatternOffsets {
    int2 off[BM_PATCH_MAX / 4];
};

cudaError_t features(const float* up, uint32_t* F, int sx, int sy, int N, int nsp,
                     const int4* pat, int rmax, const PatternOffsets& po, int rev, cudaStream_t st);

// Byte offsets (o1, o2) of every BRIEF sample from a pixel's own position less the
// margin, in an image of one pitch and margin, and per descriptor word the samples
// whose two points differ; passed by value as a kernel parameter.
struct KeyOffsets {
    uint2 off[BM_PATCH_MAX / 4];
    uint32_t differ[BM_PATCH_MAX / 4 / 32];
};
void key_offsets(KeyOffsets& ko, const int4* pat, int N, int m, int pitch);
// Whether every sample stays within 32-bit byte offsets (a margin of tens of thousands of
// pixels does not); the dense image serves the others.
bool key_image_fits(int m, int pitch);
// Whether upsample_u8_pad's rows share most of their windows: where frames are reduced to less
// than a seventh of their rows, every output's window is new, and sliding to it row by row
// loads more than the window (1920x1080 u0.1 and u0.12: 40 and 34 us with the frame's
// conversion, 16 and 16 by the dense image; at u0.15 sliding takes 25 and at u0.2 18).
inline bool rows_slide(int syi, int syo) { return syi < 7 * (long)syo; }

// `chained` in a launcher: the launch before it on the stream is a kernel that either was
// launched unchained or itself waits for its predecessor before it lets the next start
// (the stages of one frame in a row); this one may then start under its last blocks.

// Descriptors from an edge-replicated image and its keys (upsample_u8_pad): both point
// at the start of the margin, which is no narrower than the largest pattern offset.  Without
// keys (null) every pair is compared on the float image.
cudaError_t features_keys(const uint32_t* keys, const float* up, int pitch, uint32_t* F, int sx, int sy, int nsp,
                          const KeyOffsets& ko, int rev, bool chained, cudaStream_t st);

cudaError_t initialize(const uint32_t* F1, const uint32_t* F2, const uint32_t* flow_prev,
                       uint32_t* flow_out, uint16_t* cost, int sx, int sy, int nsp, int first, int rev,
                       bool chained, cudaStream_t st);

cudaError_t seed_field(const uint32_t* F1, const uint32_t* F2, const uint32_t* flow_prev, uint32_t* flow_out,
                       uint16_t* cost, int sx, int sy, int nsp, int first, const float* pred, int w4, int h4,
                       float scale_x, float scale_y, float logit_min, bool chained, cudaStream_t st);

cudaError_t local_step(const uint32_t* F1, const uint32_t* F2, const uint32_t* flow_in, uint32_t* flow_out,
                       uint16_t* cost, int sx, int sy, int nsp, int r, int rev, bool chained, cudaStream_t st);

cudaError_t jump_level(const uint32_t* F1, const uint32_t* F2, const uint32_t* flow_in,
                       uint32_t* flow_out, uint16_t* cost, int sx, int sy, int nsp,
                       int p, int pd, int doubleProp, const RsArgs& rs, int rev, bool chained, cudaStream_t st);

cudaError_t random_search(const uint32_t* F1, const uint32_t* F2, uint32_t* flow, uint16_t* cost,
                          int sx, int sy, int nsp, const RsArgs& rs, cudaStream_t st);

cudaError_t normals(float2* out, int sx, int sy, const RsArgs& rs, cudaStream_t st);

cudaError_t nn_table(unsigned int* idx, int n_up, int n_in, cudaStream_t st);
cudaError_t downsample(const uint32_t* flow, float* U, float* V, int sx, int sy, int sx_in, int sy_in,
                       const float* taps, int P, float mx, float my, const unsigned int* nnx,
                       const unsigned int* nny, bool chained, cudaStream_t st);

cudaError_t flow_to_planes(const uint32_t* flow, float* U, float* V, size_t n, bool chained, cudaStream_t st);

cudaError_t median_pass(const float* inU, const float* inV, float* outU, float* outV,
                        int dir, int fsize, int sx, int sy, bool chained, cudaStream_t st);

// Half window of the cross-trilateral filter, s = ceil(2.5*sqrt(sS^2))
// (briefmatch_cuda.cu:266), for an input frame of w x h pixels.  Returns -1 when a
// sigma is not a finite positive number, -2 when s would exceed the frame's larger
// side (such a window adds only clamped edge samples, and its cost grows as s^2).
inline int trilateral_half_window(float sEPE, float sI, float sS, uint32_t w, uint32_t h)
{
    const float big = 3.0e38f;
    if (!(sEPE > 0 && sEPE < big) || !(sI > 0 && sI < big) || !(sS > 0 && sS < big)) return -1;
    const double s = __builtin_ceil(2.5 * (double)__builtin_sqrtf(sS * sS));
    const uint32_t side = w > h ? w : h;
    if (s > (double)side) return -2;
    return (int)s;
}

cudaError_t ensure_trilateral_smem(int s);
cudaError_t trilateral(const float* U, const float* V, const float* Um, const float* Vm,
                       const float* I, float* Uo, float* Vo, int sx, int sy, int s,
                       float sigmaEPE2, float sigmaI2, float sigmaS2, bool chained, cudaStream_t st);

// Colour coding of a flow field (u, v planes of n floats) into n*3 bytes R G B
// (briefmatch.cpp:373-421, colorcode.cpp:52-74).  max_motion > 0 normalises by it;
// otherwise by the largest known vector length, measured into the device word
// d_word first.
cudaError_t flow_colors(const float* U, const float* V, size_t n, float max_motion, int* d_word, uint8_t* rgb,
                        cudaStream_t st);

cudaError_t export_field(const uint32_t* flow, const uint16_t* cost, int16_t* nx, int16_t* ny,
                         float* dist, size_t n, int N, cudaStream_t st);
cudaError_t import_field(const int16_t* nx, const int16_t* ny, const uint16_t* cost_in,
                         uint32_t* flow, uint16_t* cost, size_t n, cudaStream_t st);

}  // namespace bmk
