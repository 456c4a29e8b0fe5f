// ps_kernels.cu -- the per-frame stitch kernels (sm_103a).
//
// One frame of one or more rigs runs as at most 2L+2 launches over prepared
// work lists:
//   k_remap        level 0: LUT gain + bilinear remap of every covered tile,
//                  written as uchar4 G0 (cudaTransform + cudaReprojectTo16S);
//   k_pyrdown      levels 1..L: masked 5x5 decimation G_j -> G_{j+1}
//                  (pyrDown16SC4To16SC4 with alpha scale); k_pyrdown_pair, two
//                  levels of few tiles at once;
//   k_blend        levels L..0: for every canvas tile, the Laplacian of each
//                  camera whose seam weight touches the tile
//                  (G_j - pyrUp(G_{j+1})), its weighted accumulation, the
//                  normalisation, and the collapse step pyrUp(C_{j+1}) + N_j,
//                  all in registers; level 0 writes the 8-bit output with
//                  the uncovered pixels zeroed;
//   k_blend_rows, k_blend_small  the same for levels of few tiles (row pairs
//                  a warp; half tiles a CTA);
//   k_tail         pyrDown and blend of the smallest levels, one thread-block
//                  cluster a rig.
// The reference runs the same arithmetic as ~35 launches per camera plus
// ~36 per frame over full-canvas int16/int32 images
// (source/CudaAccel/CudaMultibandBlend.cpp:785-823).
#include <algorithm>
#include <cstddef>
#include <cstdlib>

#include "ps_async.cuh"
#include "ps_device.cuh"
#include "ps_internal.h"

namespace ps {


// ---- the checked build ---------------------------------------------------------
// Compiled with -DPS_CHECK_BOUNDS (libpanostitch_checked.so), every global
// access of the stitch kernels is checked against the extent of the buffer
// it belongs to.  An access outside is not made -- a load reads 0, a store is
// dropped -- and the device-wide violation counter goes up
// (ps_debug_bounds_violations).  Nothing traps.  k_blend's units are then all
// staged by checked loads instead of tensor copies (which the hardware
// bounds).  In the normal build every check is a constant true.
#ifdef PS_CHECK_BOUNDS
__device__ unsigned long long g_boundsViolations;
#endif

template <class T>
__device__ __forceinline__ bool inside(const T* p, const void* base, long long bytes)
{
#ifdef PS_CHECK_BOUNDS
    const char* c = reinterpret_cast<const char*>(p);
    const char* b = static_cast<const char*>(base);
    if (!base || c < b || c + sizeof(T) > b + bytes) {
        atomicAdd(&g_boundsViolations, 1ull);
        return false;
    }
#endif
    return true;
}

// [p, p + n) inside [base, base + bytes)
__device__ __forceinline__ bool insideRange(const void* p, long long n, const void* base, long long bytes)
{
#ifdef PS_CHECK_BOUNDS
    const char* c = static_cast<const char*>(p);
    const char* b = static_cast<const char*>(base);
    if (!base || c < b || c + n > b + bytes) {
        atomicAdd(&g_boundsViolations, 1ull);
        return false;
    }
#endif
    return true;
}

template <class T>
__device__ __forceinline__ T ldChecked(const T* p, const void* base, long long bytes)
{
    return inside(p, base, bytes) ? __ldg(p) : T{};
}

// Extents of a rig's buffers.
__device__ __forceinline__ long long gBytes(const RigDev& R, const LevelDev& L) { return (long long)R.n * L.camStride * 4; }
__device__ __forceinline__ long long wBytes(const RigDev& R, const LevelDev& L) { return (long long)R.n * L.camStride * 2; }
__device__ __forceinline__ long long cBytes(const LevelDev& L) { return (long long)L.pitch * L.h * 8; }

// ============================================================================
// Remap of one canvas pixel: cudaTransform (source/CudaAccel/
// CudaGainAdjust.cu:57-101) fused with the bilinear map remap.  The
// arithmetic follows the double-precision CPU bilinear (source/Warp/
// ZReproject.cpp:101-130): weights from the float map coordinates, taps
// (x0,y0) (x1,y0) (x0,y1) (x1,y1) with x1 and y1 clamped to the frame, the
// result rounded half to even.
//
// The fast path is fixed point.  A weight is W = w * 2^24, read out of the
// mantissa of 1 + w, with an error below 2^-23 (one fma rounded at 2^-24,
// and 1 - fx rounded at 2^-25 where the coordinate is below 1); the weight of
// (x0,y0) is 2^24 minus the other three, so constant areas are exact.  A
// channel is then four 32-bit multiply-adds of table bytes by weights, exact in
// 32 bits: no byte-to-float step per tap, and the rounded byte is the top byte
// of the sum, packed by two PRMTs.  The sum's error is below 255 * 4 * 2^-24 =
// 6.1e-5; a sum within 2^-13 of a rounding tie (0.07% of the pixels) goes to
// remapExact.
// ============================================================================
__device__ __forceinline__ uint32_t loadTexel(const uint8_t* row, int x, int fmt, const uint8_t* base, long long bytes)
{
    if (fmt == PS_FMT_BGR32) return ldChecked(reinterpret_cast<const uint32_t*>(row) + x, base, bytes);
    const uint8_t* p = row + 3 * x;
    if (!insideRange(p, 3, base, bytes)) return 0;
    return (uint32_t)__ldg(p) | ((uint32_t)__ldg(p + 1) << 8) | ((uint32_t)__ldg(p + 2) << 16);
}

__device__ __noinline__ int bilinearExact(double x, double y, int x0, int y0, int p00, int p01, int p10, int p11)
{
    const double wx0 = __dsub_rn(x, (double)x0), wx1 = __dsub_rn(1.0, wx0);
    const double wy0 = __dsub_rn(y, (double)y0), wy1 = __dsub_rn(1.0, wy0);
    const double w00 = __dmul_rn(wx1, wy1), w01 = __dmul_rn(wx0, wy1);
    const double w10 = __dmul_rn(wx1, wy0), w11 = __dmul_rn(wx0, wy0);
    double r = __dmul_rn((double)p00, w00);
    r = __dadd_rn(r, __dmul_rn((double)p01, w01));
    r = __dadd_rn(r, __dmul_rn((double)p10, w10));
    r = __dadd_rn(r, __dmul_rn((double)p11, w11));
    const int v = __double2int_rn(r);
    return min(max(v, 0), 255);
}

// Exact float of a byte without a conversion instruction: 2^23 + b has b in
// its low mantissa bits.
__device__ __forceinline__ float byteToFloat(uint32_t b) { return __int_as_float(0x4B000000u | b) - 8388608.f; }

// The camera frame a pixel samples.
struct RemapSrc {
    const uint8_t* base;
    long long pitch;
    int fmt, sw, sh;
};

// The byte the reference's double sequence gives, for a pixel the fast path
// could not decide (its map is valid).  A coordinate of 1 or more has a
// fraction of at most 23 bits, so the weights are integers over 2^46 and the
// sum is exact in 64 bits; the double sequence is within 7 * 2^-46 of it, so
// where the sum is farther than 2^-40 from a tie its rounding is the same.
// The double sequence itself (FP64 runs at 1/64 rate here: 60 such operations
// a pixel were most of the old recompute's cost) is left for the sums nearer
// than that and for coordinates below 1 with a longer fraction.
__device__ __noinline__ uint32_t remapExact(float2 m, RemapSrc src, const uint8_t* lut)
{
    const uint8_t* base = src.base;
    const long long pitch = src.pitch;
    const int fmt = src.fmt, sw = src.sw, sh = src.sh;
    const int x0 = (int)m.x, y0 = (int)m.y;
    const int x1 = min(x0 + 1, sw - 1), y1 = min(y0 + 1, sh - 1);
    const uint8_t* r0 = base + (size_t)y0 * pitch;
    const uint8_t* r1 = base + (size_t)y1 * pitch;
    const long long bytes = pitch * sh;
    const uint32_t t00 = loadTexel(r0, x0, fmt, base, bytes), t01 = loadTexel(r0, x1, fmt, base, bytes);
    const uint32_t t10 = loadTexel(r1, x0, fmt, base, bytes), t11 = loadTexel(r1, x1, fmt, base, bytes);
    const float qx = (m.x - (float)x0) * 8388608.f, qy = (m.y - (float)y0) * 8388608.f;  // both exact
    const uint32_t ix = (uint32_t)qx, iy = (uint32_t)qy;
    const bool fixed = (float)ix == qx && (float)iy == qy;
    const uint64_t one = 8388608u;
    const uint64_t w11 = (uint64_t)ix * iy, w01 = (uint64_t)ix * (one - iy), w10 = (one - ix) * iy;
    const uint64_t w00 = (one - ix) * (one - iy);
    uint32_t out = 0;
#pragma unroll 1
    for (int c = 0; c < 3; c++) {
        const int s = 8 * c;
        const uint8_t* t = lut + c * 256;
        const int p00 = t[(t00 >> s) & 0xFF], p01 = t[(t01 >> s) & 0xFF];
        const int p10 = t[(t10 >> s) & 0xFF], p11 = t[(t11 >> s) & 0xFF];
        const uint64_t sum = p00 * w00 + p01 * w01 + p10 * w10 + p11 * w11 + (1ull << 45);  // + 1/2
        uint32_t v = (uint32_t)(sum >> 46);
        const uint64_t frac = sum & ((1ull << 46) - 1);  // 0 at a tie
        if (!fixed || ((frac + 64) & ((1ull << 46) - 1)) <= 128)
            v = (uint32_t)bilinearExact((double)m.x, (double)m.y, x0, y0, p00, p01, p10, p11);
        out |= v << s;
    }
    return out;
}

// The remap of one pixel: the texel fetch and the LUT + bilinear finish.
struct RemapTap {
    uint32_t t00, t01, t10, t11;  // texels (x0,y0) (x1,y0) (x0,y1) (x1,y1)
    float fx, fy;                 // fractional coordinates
    bool valid;                   // false: the map is invalid here
};

// The texel pair (x, y), (x + 1, y) of a BGR24 row: its six bytes start at any
// alignment, so they are cut out of the two or (offset 3) three aligned words
// that hold them.  Every word read holds at least one of the six bytes.  The
// byte loads this replaced (twelve a pixel) kept L1 at 63% of its rate: the
// remap of 2 x 960x960 to 2048x1024 took 53 us.
__device__ __forceinline__ void loadPair24(const uint8_t* p, uint32_t& a, uint32_t& b, const uint8_t* base,
                                           long long bytes)
{
    a = b = 0;
    if (!insideRange(p, 6, base, bytes)) return;
    const uint32_t o = (uint32_t)reinterpret_cast<uintptr_t>(p) & 3u;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - o);
    const uint32_t w0 = __ldg(q), w1 = __ldg(q + 1), w2 = o == 3 ? __ldg(q + 2) : 0u;
    a = __byte_perm(w0, w1, 0x3210u + 0x1111u * o);
    b = o == 3 ? __byte_perm(w1, w2, 0x5432u) : __byte_perm(w0, w1, 0x0543u + 0x0111u * o);
}

// Integer parts use a float addition at 2^23 scale (round toward zero: the
// floor of a non-negative coordinate, an integer of 2^31 or more for any other
// value), which keeps the conversion unit out of the inner loop.  kFmt fixes
// the format at compile time (see remapSourceFormat) or leaves everything to
// the frame (0).  With kFmt the left tap is clamped to the frame's last but one
// column (row), the fraction then becoming 1, which is the same sample: both
// columns and both rows are then at fixed distances, and an invalid pixel
// fetches some texel of the frame, to be dropped by the finish.
template <int kFmt>
__device__ __forceinline__ void remapFetch(float2 m, const RemapSrc& S, RemapTap& p)
{
    const long long bytes = S.pitch * S.sh;
    if constexpr (kFmt != 0) {
        const uint32_t x = __float_as_uint(__fadd_rz(m.x, 8388608.f)) - 0x4B000000u;
        const uint32_t y = __float_as_uint(__fadd_rz(m.y, 8388608.f)) - 0x4B000000u;
        p.valid = x < (uint32_t)S.sw && y < (uint32_t)S.sh;
        const uint32_t x0 = min(x, (uint32_t)S.sw - 2u), y0 = min(y, (uint32_t)S.sh - 2u);
        p.fx = fminf(m.x - (__uint_as_float(x0 + 0x4B000000u) - 8388608.f), 1.f);  // exact
        p.fy = fminf(m.y - (__uint_as_float(y0 + 0x4B000000u) - 8388608.f), 1.f);
        const uint32_t pitch = (uint32_t)S.pitch;
        const uint8_t* r0 = S.base + (uint64_t)y0 * pitch;
        if constexpr (kFmt == PS_FMT_BGR32) {
            const uint32_t* q0 = reinterpret_cast<const uint32_t*>(r0) + x0;
            const uint32_t* q1 = reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(q0) + pitch);
            p.t00 = ldChecked(q0, S.base, bytes);
            p.t01 = ldChecked(q0 + 1, S.base, bytes);
            p.t10 = ldChecked(q1, S.base, bytes);
            p.t11 = ldChecked(q1 + 1, S.base, bytes);
        } else {
            const uint8_t* q0 = r0 + 3 * x0;
            loadPair24(q0, p.t00, p.t01, S.base, bytes);
            loadPair24(q0 + pitch, p.t10, p.t11, S.base, bytes);
        }
    } else {
        p.valid = m.x >= 0.f && m.y >= 0.f && m.x < (float)S.sw && m.y < (float)S.sh;
        const float mx = p.valid ? m.x : 0.f, my = p.valid ? m.y : 0.f;
        const float tx = __fadd_rz(mx, 8388608.f), ty = __fadd_rz(my, 8388608.f);
        const int x0 = __float_as_int(tx) - 0x4B000000, y0 = __float_as_int(ty) - 0x4B000000;
        const int x1 = min(x0 + 1, S.sw - 1), y1 = min(y0 + 1, S.sh - 1);
        const uint8_t* r0 = S.base + (size_t)y0 * S.pitch;
        const uint8_t* r1 = S.base + (size_t)y1 * S.pitch;
        p.t00 = loadTexel(r0, x0, S.fmt, S.base, bytes);
        p.t01 = loadTexel(r0, x1, S.fmt, S.base, bytes);
        p.t10 = loadTexel(r1, x0, S.fmt, S.base, bytes);
        p.t11 = loadTexel(r1, x1, S.fmt, S.base, bytes);
        p.fx = mx - (tx - 8388608.f);
        p.fy = my - (ty - 8388608.f);
    }
}

// w * 2^24 of a weight in [0, 1]: 1 + w has w * 2^23 in its mantissa.
__device__ __forceinline__ uint32_t fixedWeight(float a, float b)
{
    return 2u * __float_as_uint(fmaf(a, b, 1.f)) - 0x7F000000u;
}

// A LUT in shared memory on a 256-byte boundary, so that one PRMT puts a
// texel's byte c into the low byte of the table's address.
__device__ __forceinline__ uint32_t lutEntry(uint32_t lutAddr, uint32_t texel, int c)
{
    return static_cast<const uint8_t*>(__cvta_shared_to_generic(__byte_perm(texel, lutAddr, 0x7650u + c)))[c * 256];
}

// Returns B | G << 8 | R << 16 (0 where the map is invalid); nearTie: the
// pixel needs remapExact.  lutAddr: the camera's LUT (lutEntry).
__device__ __forceinline__ uint32_t remapFinish(const RemapTap& p, uint32_t lutAddr, bool& nearTie)
{
    const float gx = 1.f - p.fx, gy = 1.f - p.fy;
    const uint32_t w01 = fixedWeight(p.fx, gy), w10 = fixedWeight(gx, p.fy), w11 = fixedWeight(p.fx, p.fy);
    const uint32_t w00 = 0x1000000u - (w01 + w10 + w11);
    uint32_t r[3];
    nearTie = false;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const uint32_t p00 = lutEntry(lutAddr, p.t00, c), p01 = lutEntry(lutAddr, p.t01, c);
        const uint32_t p10 = lutEntry(lutAddr, p.t10, c), p11 = lutEntry(lutAddr, p.t11, c);
        r[c] = p00 * w00 + p01 * w01 + p10 * w10 + p11 * w11 + 0x800000u;  // + 1/2
        // the fraction (24 bits, moved to the top) within 2^-13 of zero
        nearTie |= (r[c] << 8) + (2048u << 8) < (4096u << 8);
    }
    nearTie = nearTie && p.valid;
    // the top bytes of the three sums
    return __byte_perm(__byte_perm(r[0], r[1], 0x0073), r[2], 0x0710) & (p.valid ? 0x00FFFFFFu : 0u);
}

// Map-free remap: the source coordinate of canvas pixel (cx, cy) in fp32,
// the steps of Remap::remapImage (source/Warp/Remap.cpp:356-514) as the
// reference's dstToSrc takes them (source/CudaAccel/CudaReproject.cu:81-264),
// which keeps them in double.  Within about 1e-3 px of the FP64 maps; the
// caller clamps the result into the frame, coverage comes from the FP64
// geometry of prepare.
__device__ __forceinline__ float2 remapPointF(const RemapParamF& m, float cx, float cy)
{
    constexpr float kPiF = 3.14159265358979323846f;
    const float xs = cx - (m.srcTX - 0.5f), ys = cy - (m.srcTY - 0.5f);
    float xd = xs + m.rot1;
    while (xd < -m.rot0) xd += 2.f * m.rot0;
    while (xd > m.rot0) xd -= 2.f * m.rot0;
    float phi = xd / m.distance;
    float theta = -ys / m.distance + kPiF / 2.f;
    if (theta < 0.f) { theta = -theta; phi += kPiF; }
    if (theta > kPiF) { theta = kPiF - (theta - kPiF); phi += kPiF; }
    float st, ct, sp, cp;
    sincosf(theta, &st, &ct);
    sincosf(phi, &sp, &cp);
    const float u0 = st * sp, u1 = ct, u2 = st * cp;
    const float v0 = m.mt[0] * u0 + m.mt[3] * u1 + m.mt[6] * u2;
    const float v1 = m.mt[1] * u0 + m.mt[4] * u1 + m.mt[7] * u2;
    const float v2 = m.mt[2] * u0 + m.mt[5] * u1 + m.mt[8] * u2;
    const float r = sqrtf(v0 * v0 + v1 * v1);
    const float th0 = r == 0.f ? 0.f : m.distance * atan2f(r, v2) / r;
    float x = th0 * v0, y = th0 * v1;
    if (m.type == 0) {
        const float rr = sqrtf(x * x + y * y);
        const float th = rr / m.distance;
        const float rho = th >= kPiF / 2.f ? 1.6e16f : (th == 0.f ? 1.f : tanf(th) / th);
        x *= rho;
        y *= rho;
    }
    x *= m.scale0;
    y *= m.scale1;
    const float rt = sqrtf(x * x + y * y) / m.rad[4];
    const float sc = rt < m.rad[5] ? ((m.rad[3] * rt + m.rad[2]) * rt + m.rad[1]) * rt + m.rad[0] : 1000.f;
    x *= sc;
    y *= sc;
    y += m.vertical;
    x += m.horizontal;
    const float xo = x + m.shear0 * y, yo = y + m.shear1 * x;
    return make_float2(xo + (m.destTX - 0.5f), yo + (m.destTY - 0.5f));
}

// The map value of a map-free pixel: -1 where the camera does not cover it,
// else the fp32 coordinate clamped into the frame.
__device__ __forceinline__ float2 mapFreeValue(const RemapParamF& m, uint32_t covWord, int lx, int cx, int cy, int sw,
                                               int sh)
{
    if (!((covWord >> lx) & 1u)) return make_float2(-1.f, -1.f);
    const float2 v = remapPointF(m, (float)cx, (float)cy);
    return make_float2(fminf(fmaxf(v.x, 0.f), __int_as_float(__float_as_int((float)sw) - 1)),
                       fminf(fmaxf(v.y, 0.f), __int_as_float(__float_as_int((float)sh) - 1)));
}

// The map value of pixel i of a remap tile (mapTileX, mapTileY): from the
// resident map at `map`, or, map-free, from the tile's coverage words there
// (the FP64 coverage of prepare) and the fp32 geometry.
template <bool kMaps>
__device__ __forceinline__ float2 remapMapValue(const void* map, const RigDev& R, const RemapItem& itm, int i)
{
    const long long tiles = R.numRemapItems;
    if (kMaps || R.maps)
        return ldChecked(static_cast<const float2*>(map) + i, R.maps,
                         tiles * kRemapTW * kRemapTH * (long long)sizeof(float2));
    const int lx = mapTileX(i), ly = mapTileY(i);
    const uint32_t bits = ldChecked(static_cast<const uint32_t*>(map) + ly, R.covTiles, tiles * kRemapTH * 4);
    return mapFreeValue(R.camsF[itm.cam], bits, lx, itm.tx * kRemapTW + lx, itm.ty * kRemapTH + ly, R.srcW, R.srcH);
}

// Level-0 remap over the covered 32x16 tiles of every camera.  The launch is
// bound by L1's rate on the gathers (four texels and twelve table bytes a
// pixel: its data pipe is 66% busy, its tags more) and by their latency, so
// everything is arranged for warps that never wait for each other: a consumer
// warp takes 16x2 blocks of a chunk's tiles, one pixel a lane, and all it needs
// besides its map values lies in shared memory or registers.  (A warp's taps
// fall on 4.3 - 8.3 lines of the frame with 16x2 blocks, 5.6 - 13 with 32x1
// rows.)  A producer warp hands the tiles out: it takes a run of tiles from the
// launch's counter and resolves them to chunks (one camera's tiles, its frame,
// its LUT) in a ring that it fills ahead of the consumers.  Runs shrink
// towards the end of the launch (a share of what is left), so the CTAs finish
// together.
// The rare pixels near a rounding tie are only marked (a ballot kept by the
// lane of the block's number) and recomputed by remapExact after the chunk: a
// call or a second code path inside the loop costs every pixel its registers.
// Measured (events around the launch): 6 x 1920x1080 to 4096x2048 57.5 us, and
// 69 + 14 us before (float sums, whole CTAs per tile, the near-tie pixels in a
// second launch); 8 x 3840x2160 to 7680x3840 197 us, before 263 + 19 us; one
// 1920x960 BGR24 frame to 2048x1024 29 us, before 54 + 14 us.  Four CTAs of 56
// registers: more warps spill (9 consumers: 62 us, 11 at 40 registers: 68 us),
// texels fetched one block ahead cost registers too (73 us).
constexpr int kRemapWarps = 8;                         // consumer warps
constexpr int kRemapThreads = (kRemapWarps + 1) * 32;  // + the producer warp
constexpr int kRemapRun = 8;                           // most tiles of a chunk
constexpr int kRemapCtas = 4;                          // CTAs per SM: 36 warps of 56 registers
constexpr int kRemapRing = 4;                          // chunks
constexpr int kRemapBlocks = kRemapTW * kRemapTH / 32;  // 16x2 blocks of a tile
static_assert((kRemapRun * kRemapBlocks + kRemapWarps - 1) / kRemapWarps <= 32, "a lane per block of a warp's chunk");

// A tile of a chunk, resolved: its map (map-free: its coverage words), its
// first pixel in the camera's level-0 plane (a 128-byte boundary) and, in that
// address's low bits, the number of its rows inside the canvas.
struct alignas(16) RemapTile {
    const void* map;
    uint64_t g;
};
__device__ __forceinline__ uint32_t* remapPixelAt(const RemapTile& t, uint32_t off)
{
    return reinterpret_cast<uint32_t*>(t.g & ~31ull) + off;
}

struct RemapChunk {
    RemapSrc src;
    const RigDev* R;
    int n, gpitch;        // n: tiles, 0 ends the launch
    RemapTile tile[kRemapRun];
    RemapItem item[kRemapRun];
    alignas(256) uint8_t lut[3 * 256];
};

// The producer warp's state: the run of tiles it has taken.  The first run is
// the CTA's by its number, the counter hands out what lies behind all of them:
// a frame starts with nothing to hide an atomic's trip to L2 behind.
struct RemapRun {
    int it, end, pos, seg;
    int first;  // tiles of all first runs; 0 before this CTA's
};

// The next chunk (all lanes of the producer warp); false after the last one.
__device__ __forceinline__ bool remapProduce(RemapRun& r, RemapChunk& c, const Segment* segs, int nsegs, int total,
                                             int* counter)
{
    const int lane = threadIdx.x & 31;
    if (r.it >= r.end) {  // a new run: a quarter of a CTA's share of what is left
        const int want = max(1, min(kRemapRun, (total - r.pos) / (4 * (int)gridDim.x)));
        if (r.first == 0) {
            r.it = r.pos = blockIdx.x * want;
            r.first = gridDim.x * want;
        } else {
            int v = 0;
            if (lane == 0) v = atomicAdd(counter, want);
            r.it = r.pos = r.first + __shfl_sync(0xffffffffu, v, 0);
        }
        r.end = min(r.it + want, total);
    }
    if (r.it >= total) {
        if (lane == 0) c.n = 0;
        return false;
    }
    r.seg = findSegment(segs, nsegs, r.it, r.seg);
    const Segment& sg = segs[r.seg];
    const int last = min(r.end, sg.prefix + sg.count);  // the run's tiles in this segment
    RemapItem item{};
    if (r.it + lane < last) item = static_cast<const RemapItem*>(sg.items)[r.it - sg.prefix + lane];
    // what does not depend on the item is on its way with it
    const FrameDev& F = *sg.frame;
    const RigDev& R = *sg.rig;
    const LevelDev L = R.lv[0];
    const float2* const maps = R.maps;
    const uint32_t* const covTiles = R.covTiles;
    const uint8_t* const luts = F.luts;
    const int H = R.H, srcW = R.srcW, srcH = R.srcH, srcFmt = F.srcFmt;
    const int cam = __shfl_sync(0xffffffffu, (int)item.cam, 0);
    const uint32_t other = __ballot_sync(0xffffffffu, r.it + lane >= last || item.cam != cam);
    const int n = other ? __ffs(other) - 1 : 32;  // the leading tiles of that camera
    if (lane < n) {
        c.item[lane] = item;
        c.tile[lane] = {maps ? static_cast<const void*>(maps + (size_t)item.mapTile * (kRemapTW * kRemapTH))
                             : static_cast<const void*>(covTiles + (size_t)item.mapTile * kRemapTH),
                        reinterpret_cast<uint64_t>(reinterpret_cast<uint32_t*>(L.G) + (size_t)cam * L.camStride +
                                                   (size_t)item.ty * kRemapTH * L.pitch + item.tx * kRemapTW) +
                            (uint32_t)min(kRemapTH, H - item.ty * kRemapTH)};
    }
    const uint4* t = reinterpret_cast<const uint4*>(luts + cam * 768);
    for (int k = lane; k < 48; k += 32) reinterpret_cast<uint4*>(c.lut)[k] = __ldg(t + k);
    if (lane == 0) {
        c.src = {F.src[cam], F.srcPitch[cam], srcFmt, srcW, srcH};
        c.R = &R;
        c.n = n;
        c.gpitch = L.pitch;
    }
    r.it += n;
    return true;
}

// A wait of the launch ran out: every frame of it is flagged (bit: kStatusBlend
// or kStatusRemap).
__device__ __forceinline__ void flagTimeout(const Segment* segs, int nsegs, int bit)
{
    for (int k = 0; k < nsegs; k++)
        if (segs[k].frame->status) atomicOr(segs[k].frame->status, bit);
}

// probePolls: as k_blend's.
template <int kFmt, bool kMaps>
__global__ void __launch_bounds__(kRemapThreads, kRemapCtas) k_remap(const Segment* __restrict__ segs, int nsegs,
                                                                        int total, int* __restrict__ counter,
                                                                        int probePolls)
{
    __shared__ RemapChunk s_chunk[kRemapRing];
    __shared__ uint64_t full[kRemapRing], empty[kRemapRing], never;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int k = 0; k < kRemapRing; k++) {
            mbarInit(&full[k], 1);
            mbarInit(&empty[k], kRemapWarps);
        }
        mbarInit(&never, 1);
    }
    __syncthreads();
    if (threadIdx.x >= kRemapWarps * 32) {
        // The hand-out counter, items, descriptors and LUTs are written before
        // the launch sequence, not by a kernel: the first chunks are resolved
        // while the previous kernel finishes.
        RemapRun r{0, 0, 0, 0, 0};
        bool more = true;
        for (int k = 0; more; k++) {
            const int s = k % kRemapRing;
            if (k >= kRemapRing && !mbarWait(&empty[s], (k / kRemapRing - 1) & 1)) {
                if (lane == 0) flagTimeout(segs, nsegs, kStatusRemap);
                break;
            }
            more = remapProduce(r, s_chunk[s], segs, nsegs, total, counter);
            __syncwarp();
            if (lane == 0) mbarArrive(&full[s]);
        }
        waitPrevGrid();
        allowNextGrid();
        return;
    }
    const int warp = threadIdx.x >> 5;
    if (probePolls > 0 && threadIdx.x == 0 && !mbarWait(&never, 0, probePolls)) flagTimeout(segs, nsegs, kStatusRemap);
    bool waited = false;
    for (int k = 0;; k++) {
        const int s = k % kRemapRing;
        if (!mbarWait(&full[s], (k / kRemapRing) & 1)) {
            if (lane == 0) flagTimeout(segs, nsegs, kStatusRemap);
            break;
        }
        const RemapChunk& c = s_chunk[s];
        const int blocks = c.n * kRemapBlocks;
        if (blocks == 0) break;
        // registers for what every block of the chunk needs: the compiler
        // would read shared memory again after each store
        const RemapSrc src = c.src;
        const int gpitch = c.gpitch;
        const RigDev* const R = c.R;
        const uint32_t lutAddr = smemAddr(c.lut);
        auto mapAt = [&](int b) {
            return remapMapValue<kMaps>(c.tile[b / kRemapBlocks].map, *R, c.item[b / kRemapBlocks],
                                        b % kRemapBlocks * 32 + lane);
        };
        int b = warp;
        float2 m{};
        if (b < blocks) m = mapAt(b);
        if (!waited) {
            waitPrevGrid();
            allowNextGrid();
            waited = true;
        }
        uint32_t ties = 0;  // lane q: the near-tie pixels of the warp's q-th block
        for (int q = 0; b < blocks; q++) {
            float2 nm = m;
            if (b + kRemapWarps < blocks) nm = mapAt(b + kRemapWarps);
            RemapTap p;
            remapFetch<kFmt>(m, src, p);
            bool tie;
            const uint32_t v = remapFinish(p, lutAddr, tie);
            // pixels beyond the canvas are invalid in the map: the columns
            // inside the plane's row pitch keep their zeros
            const int i = b % kRemapBlocks * 32 + lane;
            const RemapTile t = c.tile[b / kRemapBlocks];
            uint32_t* g = remapPixelAt(t, (uint32_t)(mapTileY(i) * gpitch + mapTileX(i)));
            if (mapTileY(i) < (int)(t.g & 31u) && inside(g, R->lv[0].G, gBytes(*R, R->lv[0]))) *g = v;
            const uint32_t near = __ballot_sync(0xffffffffu, tie);
            if (lane == q) ties = near;
            b += kRemapWarps;
            m = nm;
        }
        for (uint32_t any = __ballot_sync(0xffffffffu, ties != 0); any; any &= any - 1) {
            const int q = __ffs(any) - 1;
            if (__shfl_sync(0xffffffffu, ties, q) >> lane & 1u) {
                const int e = warp + q * kRemapWarps, i = e % kRemapBlocks * 32 + lane;
                const RemapTile te = c.tile[e / kRemapBlocks];
                uint32_t* g = remapPixelAt(te, (uint32_t)(mapTileY(i) * gpitch + mapTileX(i)));
                const float2 me = remapMapValue<kMaps>(te.map, *R, c.item[e / kRemapBlocks], i);
                const uint32_t v = remapExact(me, c.src, c.lut);
                if (inside(g, R->lv[0].G, gBytes(*R, R->lv[0]))) *g = v;
            }
            __syncwarp();
        }
        __syncwarp();
        if (lane == 0) mbarArrive(&empty[s]);  // this warp is done with the chunk
    }
    if (!waited) {
        waitPrevGrid();
        allowNextGrid();
    }
}

// ============================================================================
// k_linear: the linear-blend render (highQualityBlend == 0, CudaPanoramaRender2::
// render, source/Task/RicohUtil.cpp:1269-1286): per canvas pixel
//   accum = sum over cameras, in index order, of remap_i * w_i
// in fp32 with one rounded product and one rounded sum per camera
// (reprojectWeightedAccumulateTo32F, source/Warp/ZReproject.cpp:606-633),
// then convertTo(CV_8U): round half to even, saturate.  One 32x16 canvas
// tile per item (all tiles are items, so uncovered tiles are written 0).  The
// LUTs of all cameras of the current rig are staged in shared memory.
// ============================================================================
__device__ __forceinline__ void storeBgr(const FrameDev& F, int x, int y, int H, uint32_t v)
{
    uint8_t* row = F.out + (size_t)y * F.outPitch;
    if (!insideRange(row + (F.outFmt == PS_FMT_BGR32 ? 4 : 3) * x, F.outFmt == PS_FMT_BGR32 ? 4 : 3, F.out,
                     F.outPitch * H))
        return;
    if (F.outFmt == PS_FMT_BGR32) {
        reinterpret_cast<uint32_t*>(row)[x] = v;
    } else {
        row[3 * x] = v & 0xFF;
        row[3 * x + 1] = (v >> 8) & 0xFF;
        row[3 * x + 2] = (v >> 16) & 0xFF;
    }
}

__device__ __forceinline__ uint32_t roundSaturate3(const float* a)
{
    uint32_t v = 0;
#pragma unroll
    for (int c = 0; c < 3; c++) v |= (uint32_t)min(max(__float2int_rn(a[c]), 0), 255) << (8 * c);
    return v;
}

// A warp takes four 16x2 blocks of a tile through all of its cameras: the
// descriptors of a (tile, camera) pair are read once for 128 pixels, and its
// four map values and weights are in flight together.  A pixel at a time, 23
// of the 35 wavefronts a block and camera took in L1 were descriptors' and
// tables': 6 x 1920x1080 to 4096x2048 took 89.1 us a frame (109 us the launch
// before 16x2 blocks and fixed point), 76.4 us now.  Two blocks a warp: 94 us;
// eight: 88; two CTAs of 512 threads: 84.4, four of 256: 85.2.
constexpr int kLinearThreads = 384;
constexpr int kLinearCtas = 3;    // CTAs per SM: 36 warps of 56 registers
constexpr int kLinearBlocks = 4;  // blocks of a warp
constexpr int kLinearRun = kLinearThreads / 32 * kLinearBlocks / kRemapBlocks;  // tiles of a CTA's step
static_assert(kLinearRun >= 1 && kRemapBlocks % kLinearBlocks == 0, "a tile is whole warps");

template <int kFmt>
__global__ void __launch_bounds__(kLinearThreads, kLinearCtas) k_linear(const Segment* __restrict__ segs, int nsegs,
                                                                            int total)
{
    extern __shared__ __align__(256) uint8_t luts[];  // 768 bytes per camera of the current rig
    constexpr int kWarps = kRemapBlocks / kLinearBlocks;  // of a tile
    const int warp = threadIdx.x >> 5;
    const int first = warp % kWarps * kLinearBlocks * 32 + (threadIdx.x & 31);  // the lane's first pixel of the tile
    int s = 0, loaded = -1;
    waitPrevGrid();
    allowNextGrid();
    for (int run = blockIdx.x * kLinearRun; run < total; run += gridDim.x * kLinearRun) {
        for (int it = run, end; it < min(run + kLinearRun, total); it = end) {  // the run's tiles, segment by segment
            s = findSegment(segs, nsegs, it, s);
            const Segment& sg = segs[s];
            end = min(min(run + kLinearRun, total), sg.prefix + sg.count);
            const RigDev& R = *sg.rig;
            const FrameDev& F = *sg.frame;
            if (s != loaded) {
                __syncthreads();
                for (int k = threadIdx.x; k < R.n * 768; k += kLinearThreads) luts[k] = __ldg(F.luts + k);
                __syncthreads();
                loaded = s;
            }
            if (it + warp / kWarps >= end) continue;
            const uint32_t lutAddr = smemAddr(luts);
            const LinearItem item = static_cast<const LinearItem*>(sg.items)[it - sg.prefix + warp / kWarps];
            const long long tilePx = (long long)R.numRemapItems * kRemapTW * kRemapTH;
            auto add = [&](float* a, uint32_t v, float wv) {
#pragma unroll
                for (int c = 0; c < 3; c++) a[c] = __fadd_rn(a[c], __fmul_rn(byteToFloat((v >> (8 * c)) & 0xFF), wv));
            };
            auto store = [&](int q, const float* a) {
                const int x = item.tx * kRemapTW + mapTileX(first + 32 * q), y = item.ty * kRemapTH + mapTileY(first + 32 * q);
                if (x < R.W && y < R.H) storeBgr(F, x, y, R.H, roundSaturate3(a));
            };
            float a[kLinearBlocks][3];
#pragma unroll
            for (int q = 0; q < kLinearBlocks; q++) a[q][0] = a[q][1] = a[q][2] = 0.f;
            uint32_t ties = 0;
            for (uint32_t e = item.first; e < item.first + item.count; e++) {
                // a remap item's tile number is its index
                const float2* mp = R.maps + (size_t)e * (kRemapTW * kRemapTH) + first;
                const float* wp = R.linWeights + (size_t)e * (kRemapTW * kRemapTH) + first;
                const int cam = R.remapItems[e].cam;
                float2 m[kLinearBlocks];
                float w[kLinearBlocks];
#pragma unroll
                for (int q = 0; q < kLinearBlocks; q++) {
                    m[q] = ldChecked(mp + 32 * q, R.maps, tilePx * 8);
                    w[q] = ldChecked(wp + 32 * q, R.linWeights, tilePx * 4);
                }
                const RemapSrc src{F.src[cam], F.srcPitch[cam], F.srcFmt, R.srcW, R.srcH};
#pragma unroll
                for (int q = 0; q < kLinearBlocks; q++) {
                    RemapTap p;
                    remapFetch<kFmt>(m[q], src, p);
                    bool tie;
                    const uint32_t v = remapFinish(p, lutAddr + cam * 768, tie);
                    if (tie) ties |= 1u << q;
                    add(a[q], v, w[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < kLinearBlocks; q++) store(q, a[q]);
#pragma unroll 1
            for (; ties; ties &= ties - 1) {  // near a rounding tie in some camera: the pixel again, exactly
                const int q = __ffs(ties) - 1;
                float x[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
                for (uint32_t e = item.first; e < item.first + item.count; e++) {
                    const size_t at = (size_t)e * (kRemapTW * kRemapTH) + first + 32 * q;
                    const float2 m = ldChecked(R.maps + at, R.maps, tilePx * 8);
                    const float w = ldChecked(R.linWeights + at, R.linWeights, tilePx * 4);
                    const int cam = R.remapItems[e].cam;
                    const RemapSrc src{F.src[cam], F.srcPitch[cam], F.srcFmt, R.srcW, R.srcH};
                    const bool valid = m.x >= 0.f && m.y >= 0.f && m.x < (float)src.sw && m.y < (float)src.sh;
                    add(x, valid ? remapExact(m, src, luts + cam * 768) : 0u, w);
                }
                store(q, x);
            }
        }
    }
}

// Standalone cudaReprojectTo16S with an optional LUT: full-canvas maps,
// int16x4 output (B, G, R, 0).  A CTA takes a 64x16 tile, a warp four 16x2
// blocks of it whose map values are all loaded first, so that one round trip to
// memory serves 128 pixels; a block no pixel of which is valid (most of a
// canvas, for one camera) fetches nothing.  Near-tie pixels are recomputed at
// the end, which keeps the call out of the blocks' code.  4096x2048 from
// 1920x1080: 53.8 us before (one pixel a thread, FP64 behind a
// test per channel), 27.1 us now.
constexpr int kReprojectBlocks = 4;
// Canvases of this many CTAs take the build of five CTAs a SM: 3872 of them
// (2800x1400) are as fast either way, 5000 (3200x1600) 14.6 us against 16.4,
// 8192 (4096x2048) 27.1 against 29.2, 28800 (7680x3840) 80 against 88; 2048
// (2048x1024) 8.9 against 8.5.
constexpr unsigned kReprojectMany = 3500;

template <int kFmt, int kCtas>  // kCtas: CTAs per SM
__global__ void __launch_bounds__(kThreads, kCtas) k_reproject16s(RemapSrc src, const float* __restrict__ xmap,
                                                           const float* __restrict__ ymap, long long mapPitch,
                                                           int W, int H, const uint8_t* __restrict__ glut,
                                                           short4* dst, long long dstPitch)
{
    __shared__ __align__(256) uint8_t lut[3 * 256];
    const int lane = threadIdx.x & 31;
    const int x = blockIdx.x * 16 * kReprojectBlocks + (lane & 15), y = blockIdx.y * 16 + (threadIdx.x >> 5) * 2 + (lane >> 4);
    float2 m[kReprojectBlocks];
    if (y < H) {
        const float* xr = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(xmap) + (size_t)y * mapPitch);
        const float* yr = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(ymap) + (size_t)y * mapPitch);
#pragma unroll
        for (int k = 0; k < kReprojectBlocks; k++)
            m[k] = x + 16 * k < W ? make_float2(__ldg(xr + x + 16 * k), __ldg(yr + x + 16 * k)) : make_float2(-1.f, -1.f);
    }
    for (int k = threadIdx.x; k < 768; k += kThreads) lut[k] = glut ? glut[k] : (uint8_t)(k & 255);
    __syncthreads();
    const uint32_t lanes = __ballot_sync(0xffffffffu, y < H);  // the warp's lanes inside the canvas
    if (y >= H) return;
    short4* row = reinterpret_cast<short4*>(reinterpret_cast<uint8_t*>(dst) + (size_t)y * dstPitch) + x;
    auto store = [&](int k, uint32_t v) {
        row[16 * k] = make_short4((short)(v & 0xFF), (short)((v >> 8) & 0xFF), (short)((v >> 16) & 0xFF), 0);
    };
    uint32_t ties = 0;
#pragma unroll
    for (int k = 0; k < kReprojectBlocks; k++) {
        uint32_t v = 0;
        if (__any_sync(lanes, m[k].x >= 0.f)) {
            RemapTap p;
            bool tie;
            remapFetch<kFmt>(m[k], src, p);
            v = remapFinish(p, smemAddr(lut), tie);
            if (tie) ties |= 1u << k;
        }
        if (x + 16 * k < W) store(k, v);
    }
#pragma unroll 1
    for (; ties; ties &= ties - 1) {
        const int k = __ffs(ties) - 1;
        const float* xr = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(xmap) + (size_t)y * mapPitch);
        const float* yr = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(ymap) + (size_t)y * mapPitch);
        store(k, remapExact(make_float2(xr[x + 16 * k], yr[x + 16 * k]), src, lut));
    }
}

// ============================================================================
// k_pyrdown: pyrDown16SC4To16SC4 with alpha scale
// (source/CudaAccel/CudaPyramid2.cu:436-542): per output pixel
//   S = sum_{5x5} [1 4 6 4 1]^2 * G_j(2y+dy, 2x+dx), rows reflect-101,
//   columns wrap;  G_{j+1} = alpha ? (S << 8) / alpha : 0.
// With alpha = 256*m this is floor(S / m), evaluated exactly as
// (S * ceil(2^24 / m)) >> 24 (exact for S < 65793; S <= 65280 here).
// One CTA produces a 32x16 output tile of one camera from its 67x35 input
// tile; warp w owns output rows 4w .. 4w + 3, i.e. input rows 8w .. 8w + 10.
// Lane l loads input columns 2l and 2l + 1 of those rows, all before the first
// is used, and forms the four output rows' vertical sums in registers, B and R
// in one word a column, G of both columns in another; lanes 0..11 form those of
// the three columns beyond.  They go to the warp through its own rows of shared
// memory, and lane l filters output columns 2(l % 16) and 2(l % 16) + 1 of two
// output rows.  No step waits for another warp.  Tiles whose every alpha is 256
// (DownItem::whole, nearly all) read no divisors: S / 256 is a byte of S.
// Two output rows a warp, four words a column pair and a division for every
// pixel were 274 instructions a warp for 64 pixels, 60% of the issue slots.  Now
// level 1 of 6 x 1920x1080 to 4096x2048 takes 11.7 us (17.3 before), of 8 x
// 3840x2160 to 7680x3840 41 us (71), where memory alone would take about 10 and
// 38 us.  The item's level descriptions wait in shared memory, a level of few
// tiles is one trip to L2 long: 2.3 us against 3.2 us with them read from L2.
// ============================================================================
constexpr int kDInW = 2 * kDownTW + 3;   // 67 input columns
constexpr int kDVP = kDInW + 1;          // 68: row stride of the vertical sums
constexpr int kDownThreads = 128;
constexpr int kDWarps = kDownThreads / 32;
constexpr int kDOut = kDownTH / kDWarps;  // 4 output rows of a warp
constexpr int kDRows = 2 * kDOut + 3;     // 11 input rows
constexpr int kDHalo = kDInW - 64;        // 3 input columns beyond the lanes' pairs
static_assert(kDownTW == 32 && kDOut % 2 == 0 && kDHalo * kDOut <= 32, "the lanes' columns, rows and halo sums");

struct alignas(16) DownSmem {
    uint32_t br[kDWarps][kDOut][kDVP];  // vertical sums, B | R << 16
    uint16_t g[kDWarps][kDOut][kDVP];   // G
    uint32_t magic[257];
    alignas(16) LevelDev lv[kDWarps][2];  // the item's input and output level, a copy a warp
};
static_assert(sizeof(LevelDev) % 4 == 0 && 2 * sizeof(LevelDev) / 4 <= 32, "a word a lane");
static_assert(kDVP * 4 % 16 == 0 && kDVP * 2 % 8 == 0, "16- and 8-byte loads of rows");

__device__ __forceinline__ void initMagic(uint32_t* magic)
{
    for (int m = threadIdx.x; m < 257; m += blockDim.x) magic[m] = m ? (uint32_t)((16777216u + m - 1) / m) : 0u;
}

// [1 4 6 4 1] over five 16-bit-lane words (sums of up to 16 * 4080 stay in
// the lanes).
__device__ __forceinline__ uint32_t k5(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3, uint32_t p4)
{
    return p0 + p4 + 4 * (p1 + p3) + 6 * p2;
}

// floor(S / m) of the B, G, R sums (lo = B | R << 16, hi = G | X << 16):
// floor(S / m) = floor(S * ceil(2^24 / m) / 2^24) = umulhi(S << 8, ceil(2^24 / m)).
__device__ __forceinline__ uint32_t downDivide(uint32_t lo, uint32_t hi, uint32_t m, const uint32_t* magic)
{
    if (!m) return 0;
    const uint32_t mg = magic[m];
    const uint32_t b = __umulhi((lo & 0xFFFFu) << 8, mg);
    const uint32_t r = __umulhi((lo >> 16) << 8, mg);
    const uint32_t gg = __umulhi((hi & 0xFFFFu) << 8, mg);
    return b | (gg << 8) | (r << 16);
}

// The warp's four output rows of one tile.
__device__ __forceinline__ void downRows(const RigDev& R, const DownItem& item, DownSmem& sm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const LevelDev &Ls = sm.lv[w][0], &Ld = sm.lv[w][1];
    const int ox0 = item.tx * kDownTW, oy0 = item.ty * kDownTH + kDOut * w;
    if (oy0 >= Ld.h) return;
    const int ix0 = 2 * ox0 - 2, iy0 = 2 * oy0 - 2;  // the warp's first input pixel
    const uint32_t* G = reinterpret_cast<const uint32_t*>(Ls.G) + (size_t)item.cam * Ls.camStride;
    const long long ext = gBytes(R, Ls);
    // the lane's halo sum: column 64 + hc of output row hr
    const bool halo = lane < kDHalo * kDOut;
    const int hc = lane % kDHalo, hr = lane / kDHalo;
    uint32_t a[kDRows], b[kDRows], h[5];
    // Tiles inside the level read whole rows (8-byte loads: the first input
    // column is even and rows are 256-byte aligned); where the input crosses the
    // border every row and column is mapped by the reference's rules.
    if (ix0 >= 0 && iy0 >= 0 && ix0 + kDInW <= Ls.w && iy0 + kDRows <= Ls.h) {
        const uint32_t* row = G + (size_t)iy0 * Ls.pitch + ix0;
        const uint2* q = reinterpret_cast<const uint2*>(row) + lane;
        const uint32_t* p = row + 2 * hr * Ls.pitch + 64 + hc;
#pragma unroll
        for (int r = 0; r < kDRows; r++, q += Ls.pitch / 2) {
            const uint2 v = inside(q, Ls.G, ext) ? __ldg(q) : make_uint2(0, 0);
            a[r] = v.x;
            b[r] = v.y;
        }
#pragma unroll
        for (int r = 0; r < 5; r++, p += Ls.pitch) h[r] = halo && inside(p, Ls.G, ext) ? __ldg(p) : 0u;
    } else {
        const int c0 = colMap(ix0 + 2 * lane, Ls.w), c1 = colMap(ix0 + 2 * lane + 1, Ls.w);
        const int c2 = colMap(ix0 + 64 + hc, Ls.w);
#pragma unroll
        for (int r = 0; r < kDRows; r++) {
            const uint32_t* row = G + (size_t)rowMap(iy0 + r, Ls.h) * Ls.pitch;
            a[r] = inside(row + c0, Ls.G, ext) ? __ldg(row + c0) : 0u;
            b[r] = inside(row + c1, Ls.G, ext) ? __ldg(row + c1) : 0u;
        }
#pragma unroll
        for (int r = 0; r < 5; r++) {
            const uint32_t* p = G + (size_t)rowMap(iy0 + 2 * hr + r, Ls.h) * Ls.pitch + c2;
            h[r] = halo && inside(p, Ls.G, ext) ? __ldg(p) : 0u;
        }
    }
    // the lane's outputs (X, y), (X + 1, y) for y = oy0 + rsel and two below: X
    // is even, so both divisors are one aligned 4-byte load (X + 1 stays inside
    // the row pitch)
    const int k = lane & 15, rsel = lane >> 4;
    const int X = ox0 + 2 * k;
    const size_t at = (size_t)item.cam * Ld.camStride + (size_t)(oy0 + rsel) * Ld.pitch + X;
    uint32_t m[kDOut / 2];
    if (!item.whole) {
#pragma unroll
        for (int i = 0; i < kDOut / 2; i++)
            m[i] = X < Ld.w && oy0 + rsel + 2 * i < Ld.h
                       ? ldChecked(reinterpret_cast<const uint32_t*>(Ld.Am + at + 2 * i * Ld.pitch), Ld.Am, wBytes(R, Ld))
                       : 0u;
    }
    uint32_t ba[kDRows], bb[kDRows], gg[kDRows];  // B | R << 16 of either column, G of both (the fourth byte is 0)
#pragma unroll
    for (int r = 0; r < kDRows; r++) {
        ba[r] = a[r] & 0x00FF00FFu;
        bb[r] = b[r] & 0x00FF00FFu;
        gg[r] = __byte_perm(a[r], b[r], 0x7531);
    }
    __syncwarp();  // the warp's reads of its previous tile are done
#pragma unroll
    for (int o = 0; o < kDOut; o++) {
        const int r = 2 * o;
        *reinterpret_cast<uint2*>(&sm.br[w][o][2 * lane]) =
            make_uint2(k5(ba[r], ba[r + 1], ba[r + 2], ba[r + 3], ba[r + 4]),
                       k5(bb[r], bb[r + 1], bb[r + 2], bb[r + 3], bb[r + 4]));
        *reinterpret_cast<uint32_t*>(&sm.g[w][o][2 * lane]) = k5(gg[r], gg[r + 1], gg[r + 2], gg[r + 3], gg[r + 4]);
    }
    if (halo) {
        uint2 u[5];
#pragma unroll
        for (int r = 0; r < 5; r++) u[r] = unpackBytes(h[r]);
        sm.br[w][hr][64 + hc] = k5(u[0].x, u[1].x, u[2].x, u[3].x, u[4].x);
        sm.g[w][hr][64 + hc] = (uint16_t)k5(u[0].y, u[1].y, u[2].y, u[3].y, u[4].y);
    }
    __syncwarp();
    uint32_t* dst = reinterpret_cast<uint32_t*>(Ld.G) + at;
    const long long oext = gBytes(R, Ld);
#pragma unroll
    for (int i = 0; i < kDOut / 2; i++, dst += 2 * Ld.pitch) {
        // output columns 2k and 2k + 1 read vertical sums 4k .. 4k + 4 and 4k + 2 .. 4k + 6
        const uint32_t* vb = &sm.br[w][rsel + 2 * i][4 * k];
        const uint16_t* vg = &sm.g[w][rsel + 2 * i][4 * k];
        const uint4 p = *reinterpret_cast<const uint4*>(vb), q = *reinterpret_cast<const uint4*>(vb + 4);
        const uint2 gp = *reinterpret_cast<const uint2*>(vg), gq = *reinterpret_cast<const uint2*>(vg + 4);
        const uint32_t br0 = k5(p.x, p.y, p.z, p.w, q.x), br1 = k5(p.z, p.w, q.x, q.y, q.z);
        const uint32_t g0 = __dp2a_lo(gp.x, 0x0401u, __dp2a_lo(gp.y, 0x0406u, gq.x & 0xFFFFu));
        const uint32_t g1 = __dp2a_lo(gp.y, 0x0401u, __dp2a_lo(gq.x, 0x0406u, gq.y & 0xFFFFu));
        uint32_t out0, out1;
        if (item.whole) {
            out0 = __byte_perm(br0, g0, 0x7351);
            out1 = __byte_perm(br1, g1, 0x7351);
        } else {
            out0 = downDivide(br0, g0, m[i] & 0xFFFFu, sm.magic);
            out1 = downDivide(br1, g1, m[i] >> 16, sm.magic);
        }
        if (X >= Ld.w || oy0 + rsel + 2 * i >= Ld.h) continue;
        if (X + 1 < Ld.w) {
            if (inside(reinterpret_cast<uint2*>(dst), Ld.G, oext)) *reinterpret_cast<uint2*>(dst) = make_uint2(out0, out1);
        } else if (inside(dst, Ld.G, oext)) {
            dst[0] = out0;
        }
    }
}

// The levels of an item into the warp's copy.
__device__ __forceinline__ void downLevels(const RigDev& R, int level, DownSmem& sm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncwarp();
    if (lane < 2 * (int)sizeof(LevelDev) / 4)
        reinterpret_cast<uint32_t*>(sm.lv[w])[lane] = __ldg(reinterpret_cast<const uint32_t*>(&R.lv[level - 1]) + lane);
    __syncwarp();
}

// One CTA walks a contiguous run of tiles, each warp for itself.
__global__ void __launch_bounds__(kDownThreads, 8) k_pyrdown(const Segment* __restrict__ segs, int nsegs, int total)
{
    __shared__ DownSmem sm;
    initMagic(sm.magic);
    int s = 0, begin, end;
    itemRange(total, begin, end);
    // Items and descriptors are written before the launch sequence, not by
    // a kernel: the first tile's are read while the previous kernel finishes.
    DownItem item{};
    if (begin < end) {
        s = findSegment(segs, nsegs, begin, s);
        item = static_cast<const DownItem*>(segs[s].items)[begin - segs[s].prefix];
        downLevels(*segs[s].rig, item.level, sm);
    }
    __syncthreads();  // the magic table
    waitPrevGrid();
    allowNextGrid();
    for (int it = begin; it < end;) {
        const DownItem now = item;
        const int sn = s;
        if (++it < end) {
            s = findSegment(segs, nsegs, it, s);
            item = static_cast<const DownItem*>(segs[s].items)[it - segs[s].prefix];
        }
        downRows(*segs[sn].rig, now, sm);
        if (s != sn) downLevels(*segs[s].rig, item.level, sm);
    }
}

// ============================================================================
// k_pyrdown_pair: two levels J and J + 1 of few tiles in one launch.  A level of
// few tiles is a chain of latencies (its release, a trip to L2, the arithmetic,
// the stores), 3 us whatever it holds.  A CTA takes a 32x16 tile of level J and
// the 16x8 pixels of level J + 1 under it: it stages the 73x41 input pixels,
// makes the 35x19 pixels of level J that its part of level J + 1 reads (the
// halo a second time: each belongs to a neighbour's tile) and filters those.
// Columns wrap as the input does, which is the reference's rule as long as the
// input is twice level J wide (Rig::preparePyramids lists only such); rows beyond the level are mapped
// when level J + 1 reads them.
// 512 threads: with 256 a launch is 3.8 us, with 704 no shorter.  256x128: 31.2 us
// a frame, 33.5 with a launch a level; 2048x1024: 78.8 against 80.3; 6 x
// 1920x1080 to 4096x2048: 161.2 against 163.5.
// ============================================================================
constexpr int kPairThreads = 512;
constexpr int kPairInW = 74, kPairInH = 41;    // staged input (an even number of columns)
constexpr int kPairInP = 76;
constexpr int kPairMidW = 35, kPairMidH = 19;  // staged level J
constexpr int kPairMidP = 36;

struct alignas(16) PairSmem {
    uint32_t in[kPairInH][kPairInP];
    uint32_t mid[kPairMidH][kPairMidP];
    uint32_t magic[257];
    alignas(16) LevelDev lv[3];  // J - 1, J, J + 1
};

// The 5x5 filter on five rows from their first tap.
__device__ __forceinline__ uint32_t pairFilter(const uint32_t* const (&rows)[5], uint32_t m, const uint32_t* magic)
{
    uint32_t lo[5], hi[5];
#pragma unroll
    for (int r = 0; r < 5; r++) {
        uint2 u[5];
#pragma unroll
        for (int i = 0; i < 5; i++) u[i] = unpackBytes(rows[r][i]);
        lo[r] = k5(u[0].x, u[1].x, u[2].x, u[3].x, u[4].x);
        hi[r] = k5(u[0].y, u[1].y, u[2].y, u[3].y, u[4].y);
    }
    return downDivide(k5(lo[0], lo[1], lo[2], lo[3], lo[4]), k5(hi[0], hi[1], hi[2], hi[3], hi[4]), m, magic);
}

__device__ __forceinline__ void pairStore(const RigDev& R, const LevelDev& L, int cam, int x, int y, uint32_t v)
{
    uint32_t* d = reinterpret_cast<uint32_t*>(L.G) + (size_t)cam * L.camStride + (size_t)y * L.pitch + x;
    if (inside(d, L.G, gBytes(R, L))) *d = v;
}

__device__ __forceinline__ uint32_t pairAlpha(const RigDev& R, const LevelDev& L, int cam, int x, int y)
{
    return ldChecked(L.Am + (size_t)cam * L.camStride + (size_t)y * L.pitch + x, L.Am, wBytes(R, L));
}

__device__ __forceinline__ void pairTile(const RigDev& R, const DownItem& item, PairSmem& sm)
{
    const LevelDev &Li = sm.lv[0], &Lm = sm.lv[1], &Lo = sm.lv[2];
    const int t = threadIdx.x, cam = item.cam;
    const int mx0 = item.tx * kDownTW - 2, my0 = item.ty * kDownTH - 2;  // first pixel of mid
    const int ix0 = 2 * mx0 - 2, iy0 = 2 * my0 - 2;                      // of in
    const uint32_t* G = reinterpret_cast<const uint32_t*>(Li.G) + (size_t)cam * Li.camStride;
    const long long ext = gBytes(R, Li);
    // every load before any store
    constexpr int kPieces = kPairInH * (kPairInW / 2), kIn = (kPieces + kPairThreads - 1) / kPairThreads;
    constexpr int kMid = (kPairMidH * kPairMidP + kPairThreads - 1) / kPairThreads;
    const bool whole = ix0 >= 0 && iy0 >= 0 && ix0 + kPairInW <= Li.w && iy0 + kPairInH <= Li.h;
    uint2 v[kIn];
#pragma unroll
    for (int k = 0; k < kIn; k++) {
        const int e = t + k * kPairThreads, r = e / (kPairInW / 2), c = 2 * (e % (kPairInW / 2));
        v[k] = make_uint2(0, 0);
        if (e >= kPieces) continue;
        if (whole) {
            const uint2* p = reinterpret_cast<const uint2*>(G + (size_t)(iy0 + r) * Li.pitch + ix0 + c);
            if (inside(p, Li.G, ext)) v[k] = __ldg(p);
        } else {
            const uint32_t* row = G + (size_t)rowMap(iy0 + r, Li.h) * Li.pitch;
            const uint32_t *p = row + colMap(ix0 + c, Li.w), *q = row + colMap(ix0 + c + 1, Li.w);
            v[k] = make_uint2(inside(p, Li.G, ext) ? __ldg(p) : 0u, inside(q, Li.G, ext) ? __ldg(q) : 0u);
        }
    }
    uint32_t m[kMid];
    int mx[kMid];
#pragma unroll
    for (int k = 0; k < kMid; k++) {
        const int e = t + k * kPairThreads, r = e / kPairMidP, c = e % kPairMidP;
        mx[k] = -1;
        m[k] = 0;
        if (r < kPairMidH && c < kPairMidW && my0 + r >= 0 && my0 + r < Lm.h) {
            mx[k] = colMap(mx0 + c, Lm.w);
            m[k] = pairAlpha(R, Lm, cam, mx[k], my0 + r);
        }
    }
    const int ox = item.tx * (kDownTW / 2) + (t & 15), oy = item.ty * (kDownTH / 2) + (t >> 4);
    const bool out = t < 128 && ox < Lo.w && oy < Lo.h;
    const uint32_t mo = out ? pairAlpha(R, Lo, cam, ox, oy) : 0u;
    __syncthreads();  // readers of the tile before are done
#pragma unroll
    for (int k = 0; k < kIn; k++) {
        const int e = t + k * kPairThreads, r = e / (kPairInW / 2), c = 2 * (e % (kPairInW / 2));
        if (e < kPieces) *reinterpret_cast<uint2*>(&sm.in[r][c]) = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kMid; k++) {
        if (mx[k] < 0) continue;
        const int e = t + k * kPairThreads, r = e / kPairMidP, c = e % kPairMidP;
        const uint32_t* p = &sm.in[2 * r][2 * c];
        const uint32_t* const rows[5] = {p, p + kPairInP, p + 2 * kPairInP, p + 3 * kPairInP, p + 4 * kPairInP};
        const uint32_t o = pairFilter(rows, m[k], sm.magic);
        sm.mid[r][c] = o;
        // the tile's own pixels
        if (r >= 2 && r < 2 + kDownTH && c >= 2 && c < 2 + kDownTW && mx0 + c < Lm.w) pairStore(R, Lm, cam, mx[k], my0 + r, o);
    }
    __syncthreads();
    if (out) {
        const uint32_t* rows[5];
#pragma unroll
        for (int r = 0; r < 5; r++) rows[r] = &sm.mid[rowMap(2 * oy - 2 + r, Lm.h) - my0][2 * (t & 15)];
        pairStore(R, Lo, cam, ox, oy, pairFilter(rows, mo, sm.magic));
    }
}

__global__ void __launch_bounds__(kPairThreads) k_pyrdown_pair(const Segment* __restrict__ segs, int nsegs, int total)
{
    __shared__ PairSmem sm;
    initMagic(sm.magic);
    int s = -1;
    for (int it = blockIdx.x; it < total; it += gridDim.x) {
        const int sn = findSegment(segs, nsegs, it, max(s, 0));
        const DownItem item = static_cast<const DownItem*>(segs[sn].items)[it - segs[sn].prefix];
        const RigDev& R = *segs[sn].rig;
        if (sn != s) {  // the first one's while the previous kernel finishes
            __syncthreads();
            if (threadIdx.x < 3 * sizeof(LevelDev) / 4)
                reinterpret_cast<uint32_t*>(sm.lv)[threadIdx.x] =
                    __ldg(reinterpret_cast<const uint32_t*>(&R.lv[item.level - 1]) + threadIdx.x);
            __syncthreads();
            if (s < 0) {
                waitPrevGrid();
                allowNextGrid();
            }
            s = sn;
        }
        pairTile(R, item, sm);
    }
    if (s < 0) {
        waitPrevGrid();
        allowNextGrid();
    }
}

// ============================================================================
// k_blend: one canvas level of the blend, all cameras at once.
//   For each camera i whose weight touches the tile:
//     U = pyrUp(G_{i,j+1})            pyrUp16SC4To16SC4, CudaPyramid2.cu:628-710
//     L = G_{i,j} - U  (L_L = G_L)    subtract16SC4, :836-845
//     R += w_ij * L, W += w_ij        accumulate16SC4To32SC4, :759-773
//   N = full ? (R + 128) >> 8 : R / max(W, 1)     normalize32SC4, :749-791
//   C_j = N + pyrUp32(C_{j+1})        restoreImageFromLaplacePyramid,
//                                     CudaMultibandBlend.cpp:220-231
//   level 0: out = clamp(C_0, 0, 255), 0 where no camera covers
//   (convertTo(CV_8U) + setTo(0, maskNot), CudaMultibandBlend.cpp:820-822).
// A tile whose only camera has weight 256 on every pixel has N = L exactly
// (R = 256 L, W = 256; (256 L + 128) >> 8 = L), so it skips the weights.
//
// A tile is 64x16 canvas pixels; consumer thread t (of 256) owns the 2x2
// block at (2*(t%32), 2*(t/32)), so the zero-inserted upsample's three
// footprint rows serve both of its rows and the YUV chroma of the block is
// its own.  Work flows through a 2-stage shared-memory ring of "units" (a
// tile and up to two of its cameras).  A dedicated producer warp stages each
// unit with bulk tensor copies -- per camera the G_j tile, its weights (not
// for uniform tiles) and its G_{j+1} footprint, and with a tile's last unit
// the C_{j+1} footprint -- completing on the stage's "full" mbarrier; the
// eight consumer warps compute from shared memory and release the stage on its
// "empty" mbarrier.  Tiles whose footprints cross the canvas border
// (horizontal wrap, vertical reflect-101) are staged by the consumers with the
// reference's index mapping.
//
// Level 0 of 6 x 1920x1080 to 4096x2048 in a running frame: 30 us from its
// release, 37.5 before the uniform tiles' packed path and the runs (24.3 M instead
// of 32.0 M warp instructions); of 8 x 3840x2160 to 7680x3840: 77 us, 101 before.
// Left: a unit's arithmetic (2300 cycles of eight warps a scheduler) and the
// staging of the next take turns waiting for each other; a 4-stage ring, a
// 3-stage one, one lane doing the producer's work, and copies issued ahead of
// everything else in the producer's step measured no shorter.
// ============================================================================
constexpr int kFW = kBlendTW / 2 + 2;  // 34: footprint columns fx0 .. fx0+33
constexpr int kFH = kBlendTH / 2 + 2;  // 10: footprint rows    fy0 .. fy0+9
constexpr int kBStages = 2;
constexpr int kCamsPerUnit = 2;
constexpr int kFpW = 40;   // staged footprint row: columns fx0-3 .. fx0+36 (16-byte aligned start)
constexpr int kCfW = 36;   // staged collapse footprint row: columns fx0-1 .. fx0+34
constexpr int kMaxSmemSegs = 64;
constexpr int kConsumers = kThreads;          // 8 warps
// Tiles the producer takes at a time: a kBlendShare'th of a CTA's part of what
// is left, at most kBlendRun.  One at a time, the atomic's round trip and the
// descriptor's load per tile held the consumers up (7680x3840 level 0: 94 us,
// 84 with runs of 4); larger shares leave CTAs unequal at the end.
constexpr int kBlendRun = 4, kBlendShare = 4;
constexpr int kYuvThreads = 128;  // of the eight-pixel conversions
constexpr int kBlendThreads = kConsumers + 32;  // + the producer warp

// One unit's shared-memory stage: NC cameras of one tile (k_blend stages
// two cameras per unit in a ring; the kernels of the few-tile levels stage up
// to eight at once, of a half tile).
// Every camera's part starts on a 128-byte boundary, as the bulk tensor
// copies into it require: the footprint of a camera is kFH rows of kFpW
// words (a dense box), padded to kFpCam words.
// ROWS: the rows of the tile it holds, all or one half's.
template <int NC, int ROWS = kBlendTH>
struct alignas(128) BlendStageT {
    static constexpr int kCams = NC, kRows = ROWS, kFpRows = ROWS / 2 + 2;
    static constexpr int kFpCam = (kFpRows * kFpW + 31) / 32 * 32;
    uint32_t gj[NC][ROWS][kBlendTW];  // G_j, uchar4
    uint16_t w[NC][ROWS][kBlendTW];   // weights
    uint32_t fpw[NC][kFpCam];         // G_{j+1} footprint: row r, column c at [r * kFpW + c]
    uint2 cf[kFpRows][kCfW];          // C_{j+1} footprint (short4 bits)
};
using BlendStage = BlendStageT<kCamsPerUnit>;
static_assert(offsetof(BlendStage, w) % 128 == 0 && offsetof(BlendStage, fpw) % 128 == 0 &&
                  offsetof(BlendStage, cf) % 128 == 0 && sizeof(BlendStage::gj[0]) % 128 == 0 &&
                  sizeof(BlendStage::w[0]) % 128 == 0 && sizeof(BlendStage::fpw[0]) % 128 == 0,
              "every bulk tensor copy destination starts on a 128-byte boundary");
constexpr int kHalfRows = kBlendTH / 2;
using HalfStage = BlendStageT<8, kHalfRows>;  // half tiles of the few-tile levels

// What the consumers need of a unit besides its stage: the level geometry
// and the frame's output, resolved once per unit (in k_blend by the
// producer warp, so the consumers read it from shared memory).
struct UnitGeo {
    int w, h, pitch, full, hasUp, outFmt;
    short4* C;              // collapsed result of the unit's level (j >= 1)
    const uint8_t* um;      // union mask (level 0, partially covered tiles)
    uint8_t* out;           // BGR canvas or Y plane
    uint8_t* outU;          // U (YUV420P) or UV (NV12) plane
    uint8_t* outV;          // V plane (YUV420P)
    long long outPitch, outCPitch, outVPitch;
};

__device__ __forceinline__ void fillGeo(UnitGeo& g, const RigDev& R, const FrameDev& F, int j)
{
    const LevelDev& Lj = R.lv[j];
    g.w = Lj.w;
    g.h = Lj.h;
    g.pitch = Lj.pitch;
    g.full = R.full;
    g.hasUp = j < R.L;
    g.C = Lj.C;
    if (j > 0) return;  // the frame's output is level 0's
    g.outFmt = F.outFmt;
    g.um = R.unionMask;
    g.out = F.out;
    g.outU = F.outU;
    g.outV = F.outV;
    g.outPitch = F.outPitch;
    g.outCPitch = F.outCPitch;
    g.outVPitch = F.outVPitch;
}

struct UnitInfo {
    uint4 raw;
    int chunk, valid, staged;  // staged: copies issued by the producer
    int seg;                   // the segment geo was filled in for
    UnitGeo geo;
};

// ---- BT.601 studio-range conversion (cvtBGRToYUV2x2Block,
// ImageProc.cu:44-95): 20-bit fixed point, Y = 16 + ..., chroma = 128 + ...
// These are the standard BT.601 coefficients scaled by 2^20; the chroma of
// a 2x2 block is the mean of its left column's two pixels.
constexpr int kYR = 269484, kYG = 528482, kYB = 102760;
constexpr int kUR = -155188, kUG = -305135, kUB = 460324;
constexpr int kVR = 460324, kVG = -385875, kVB = -74448;
constexpr int kYuvShift = 20;
constexpr int kYuvHalf = 1 << (kYuvShift - 1);
constexpr int kYOff = (16 << kYuvShift) + kYuvHalf;
constexpr int kCOff = (128 << kYuvShift) + kYuvHalf;

__device__ __forceinline__ int clamp255(int v) { return min(max(v, 0), 255); }

// B | G << 8 | R << 16 with each channel saturated to 0..255: two
// cvt.pack.sat.u8.s32.b32 (PTX: d = sat(b) | sat(a) << 8 | c[15:0] << 16)
// instead of six min / max and the shifts.
__device__ __forceinline__ uint32_t packSatBgr(int b, int g, int r)
{
    uint32_t hi, out;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(0), "r"(r), "r"(0));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(g), "r"(b), "r"(hi));
    return out;
}

// Luma before saturation; yuvLuma saturates it.
__device__ __forceinline__ int yuvLumaRaw(uint32_t bgr)
{
    const int b = bgr & 0xFF, g = (bgr >> 8) & 0xFF, r = (bgr >> 16) & 0xFF;
    return (kYR * r + kYG * g + kYB * b + kYOff) >> kYuvShift;
}

__device__ __forceinline__ uint32_t yuvLuma(uint32_t bgr) { return (uint32_t)clamp255(yuvLumaRaw(bgr)); }

// sat(lo) | sat(hi) << 8, each saturated to 0..255 (one cvt.pack.sat)
__device__ __forceinline__ uint32_t packSat2(int lo, int hi)
{
    uint32_t out;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(hi), "r"(lo), "r"(0));
    return out;
}

// Unshifted chroma sums of one pixel (both are non-negative).
__device__ __forceinline__ int2 yuvChromaSums(uint32_t bgr)
{
    const int b = bgr & 0xFF, g = (bgr >> 8) & 0xFF, r = (bgr >> 16) & 0xFF;
    return make_int2(kUR * r + kUG * g + kUB * b + kCOff, kVR * r + kVG * g + kVB * b + kCOff);
}

// Level-0 store of a consumer thread's 2x2 block as four Y samples and the
// block's U and V (from its left column, as cvtBGRToYUV2x2Block computes
// them).  o[0] o[1] are the top pixels, o[2] o[3] the bottom ones.
__device__ __forceinline__ void storeYuv(const UnitGeo& G, int x, int y, const uint32_t* o)
{
#pragma unroll
    for (int r = 0; r < 2; r++) {
        uint8_t* yrow = G.out + (size_t)(y + r) * G.outPitch + x;
        const uint32_t yy = packSat2(yuvLumaRaw(o[2 * r]), yuvLumaRaw(o[2 * r + 1]));
        if (!insideRange(yrow, 2, G.out, G.outPitch * G.h)) continue;
        if ((reinterpret_cast<uintptr_t>(yrow) & 1) == 0) {
            *reinterpret_cast<uint16_t*>(yrow) = (uint16_t)yy;
        } else {
            yrow[0] = (uint8_t)yy;
            yrow[1] = (uint8_t)(yy >> 8);
        }
    }
    const int2 c = yuvChromaSums(o[0]), d = yuvChromaSums(o[2]);
    const uint32_t uv = packSat2((c.x + d.x) >> (kYuvShift + 1), (c.y + d.y) >> (kYuvShift + 1));
    const uint8_t u = (uint8_t)uv, v = (uint8_t)(uv >> 8);
    const size_t cy = (size_t)(y >> 1);
    const long long cext = G.outCPitch * (G.h / 2);
    if (G.outFmt == PS_FMT_NV12) {
        uint8_t* p = G.outU + cy * G.outCPitch + x;
        if (!insideRange(p, 2, G.outU, cext)) return;
        if ((reinterpret_cast<uintptr_t>(p) & 1) == 0) {
            *reinterpret_cast<uint16_t*>(p) = (uint16_t)uv;
        } else {
            p[0] = u;
            p[1] = v;
        }
    } else {
        if (inside(G.outU + cy * G.outCPitch + (x >> 1), G.outU, cext)) G.outU[cy * G.outCPitch + (x >> 1)] = u;
        if (inside(G.outV + cy * G.outVPitch + (x >> 1), G.outV, G.outVPitch * (G.h / 2)))
            G.outV[cy * G.outVPitch + (x >> 1)] = v;
    }
}

// q-th camera of a blend tile (raw 16-byte descriptor)
__device__ __forceinline__ int tileCam(const uint4& raw, const uint8_t* camLists, int q)
{
    if (((raw.x >> 16) & 0xFF) > kInlineCams) return __ldg(camLists + raw.z + q);
    const uint32_t w = q < 4 ? raw.z : raw.w;
    return (int)((w >> (8 * (q & 3))) & 0xFF);
}

template <int NC = kCamsPerUnit>
__device__ __forceinline__ int unitChunks(const uint4& raw)
{
    const int cnt = (raw.x >> 16) & 0xFF;
    return cnt <= NC ? 1 : (cnt + NC - 1) / NC;
}

// Accumulators of a thread's 2x2 block: pixel p = 2 * row + column.
struct BlendAcc {
    int r[4][3];
    int wsum[4];
};

// Stage one unit with index-mapped loads (border tiles).  Threads 0..kConsumers-1; the caller synchronises.
// fRow / fCol: footprint index tables (kFH / kFW ints) filled here; sync is
// the barrier over the calling threads.
template <class Stage, class Sync>
__device__ __forceinline__ void stageUnitDirect(Stage& S, const RigDev& R, const uint4& raw, int chunk, int* fRow,
                                                int* fCol, Sync sync)
{
    const int lx = (threadIdx.x & 31) * 2, ly = (threadIdx.x >> 5) * 2;
    const int j = raw.x & 0xFF, camCnt = (raw.x >> 16) & 0xFF;
    const int tx = raw.y & 0xFFFF, ty = raw.y >> 16;
    const LevelDev& Lj = R.lv[j];
    const bool hasUp = j < R.L;
    const LevelDev& Lu = R.lv[hasUp ? j + 1 : j];
    const int x = tx * kBlendTW + lx, y = ty * kBlendTH + ly;
    constexpr int NC = Stage::kCams;
    const int c0 = chunk * NC;
    const int nc = max(0, min(NC, camCnt - c0));
    const bool last = chunk == unitChunks<NC>(raw) - 1;
    const int fx0 = tx * (kBlendTW / 2) - 1, fy0 = ty * (kBlendTH / 2) - 1;
    for (int q = 0; q < nc; q++) {
        const int cam = tileCam(raw, R.camLists, c0 + q);
        for (int r = 0; r < 2; r++) {
            uint2 g = make_uint2(0, 0);
            uint32_t w = 0;
            if (y + r < Lj.h) {  // columns up to the pitch are allocated (and zero beyond the width)
                const size_t o = (size_t)cam * Lj.camStride + (size_t)(y + r) * Lj.pitch + x;
                const uint2* gp = reinterpret_cast<const uint2*>(Lj.G + o);
                const uint32_t* wp = reinterpret_cast<const uint32_t*>(Lj.Wt + o);
                if (inside(gp, Lj.G, gBytes(R, Lj))) g = __ldg(gp);
                if (inside(wp, Lj.Wt, wBytes(R, Lj))) w = __ldg(wp);
            }
            *reinterpret_cast<uint2*>(&S.gj[q][ly + r][lx]) = g;
            *reinterpret_cast<uint32_t*>(&S.w[q][ly + r][lx]) = w;
        }
    }
    if (hasUp) {
        if (threadIdx.x < kFH) fRow[threadIdx.x] = rowMap(fy0 + (int)threadIdx.x, Lu.h);
        else if (threadIdx.x < kFH + kFW) fCol[threadIdx.x - kFH] = colMap(fx0 + (int)threadIdx.x - kFH, Lu.w);
        sync();
        constexpr int elems = kFH * kFW;
        for (int k = threadIdx.x; k < nc * elems; k += kConsumers) {
            const int q = k / elems, e = k - q * elems;
            const int r = e / kFW, c = e % kFW;
            const int cam = tileCam(raw, R.camLists, c0 + q);
            const uint32_t* gp = reinterpret_cast<const uint32_t*>(Lu.G) + (size_t)cam * Lu.camStride +
                                 (size_t)fRow[r] * Lu.pitch + fCol[c];
            S.fpw[q][r * kFpW + c + 3] = inside(gp, Lu.G, gBytes(R, Lu)) ? __ldg(gp) : 0u;
        }
        if (last)
            for (int k = threadIdx.x; k < elems; k += kConsumers) {
                const int r = k / kFW, c = k % kFW;
                const uint2* cp = reinterpret_cast<const uint2*>(Lu.C + (size_t)fRow[r] * Lu.pitch + fCol[c]);
                S.cf[r][c + 1] = inside(cp, Lu.C, cBytes(Lu)) ? __ldg(cp) : make_uint2(0, 0);
            }
    }
}

// The half-tile staging of the few-tile levels, where one unit's staging is
// most of a level's critical path: 16-byte loads of whole rows, the footprint
// element by element with the reference's index mapping, in little code (a level's kernel runs its code once, so every
// line of it is fetched from L2).  A unit is eight rows (8 * half ..) of a tile
// and up to eight of its cameras.  Threads 0..kConsumers-1; the caller
// synchronises before the stage is read.
//
// stageHalfG: of the cameras' G_j rows, weights and G_{j+1} footprints the
// parts asked for, through L2 (what another launch wrote while this one began).
static_assert(HalfStage::kFpRows * kFW <= kConsumers, "a footprint element a thread");
constexpr int kPartW = 1, kPartG = 2, kPartUp = 4, kPartsAll = 7;

// Element (r, c) of a half tile's footprint in a plane of level Lu.  Elements
// that no pixel of level Lj needs (the tile reaches beyond the level) map to 0.
__device__ __forceinline__ size_t halfFpOffset(const LevelDev& Lu, const LevelDev& Lj, int tx, int ty, int half, int r,
                                               int c)
{
    const int x = tx * kBlendTW, y = ty * kBlendTH + kHalfRows * half;
    if (c > (Lj.w - x + 1) / 2 + 1 || r > (Lj.h - y + 1) / 2 + 1) return 0;
    return (size_t)rowMap(y / 2 - 1 + r, Lu.h) * Lu.pitch + colMap(x / 2 - 1 + c, Lu.w);
}

__device__ __forceinline__ void stageHalfG(HalfStage& S, const RigDev& R, const uint4& raw, int chunk, int half,
                                           int parts)
{
    constexpr int NC = HalfStage::kCams;
    const int j = raw.x & 0xFF, camCnt = (raw.x >> 16) & 0xFF;
    const int tx = raw.y & 0xFFFF, ty = raw.y >> 16;
    const LevelDev& Lj = R.lv[j];
    const int c0 = chunk * NC, nc = max(0, min(NC, camCnt - c0));
    const int t = threadIdx.x;
    auto camAt = [&](int q) { return (size_t)tileCam(raw, R.camLists, c0 + q); };
    // every load of the unit before any store: G_j rows (two cameras a pass),
    // weights (four cameras a pass; columns up to the pitch are allocated, and
    // zero beyond the width), and one footprint element of every camera, whose
    // index mapping is thus worked out once
    uint4 g[NC / 2], w[NC / 4];
    uint32_t f[NC];
    const int gc = (t & 15) * 4, gr = t >> 4 & 7, gy = ty * kBlendTH + kHalfRows * half + gr;
    const int wc = (t & 7) * 8, wr = t >> 3 & 7, wy = ty * kBlendTH + kHalfRows * half + wr;
    const int fr = t / kFW, fc = t % kFW;
    const bool hasF = (parts & kPartUp) && j < R.L && fr < HalfStage::kFpRows;
    const LevelDev& Lu = R.lv[j < R.L ? j + 1 : j];
    const size_t fo = hasF ? halfFpOffset(Lu, Lj, tx, ty, half, fr, fc) : 0;
#pragma unroll
    for (int q = 0; q < NC; q++) {
        f[q] = 0;
        if (q < nc && hasF) {
            const uint32_t* p = reinterpret_cast<const uint32_t*>(Lu.G) + camAt(q) * Lu.camStride + fo;
            if (inside(p, Lu.G, gBytes(R, Lu))) f[q] = __ldcg(p);
        }
    }
#pragma unroll
    for (int i = 0; i < NC / 2; i++) {
        const int q = (t >> 7) + 2 * i;
        g[i] = make_uint4(0, 0, 0, 0);
        if ((parts & kPartG) && q < nc && gy < Lj.h) {
            const uint4* p = reinterpret_cast<const uint4*>(Lj.G + camAt(q) * Lj.camStride + (size_t)gy * Lj.pitch +
                                                            tx * kBlendTW + gc);
            if (inside(p, Lj.G, gBytes(R, Lj))) g[i] = __ldcg(p);
        }
    }
#pragma unroll
    for (int i = 0; i < NC / 4; i++) {
        const int q = (t >> 6) + 4 * i;
        w[i] = make_uint4(0, 0, 0, 0);
        if ((parts & kPartW) && q < nc && wy < Lj.h) {
            const uint4* p = reinterpret_cast<const uint4*>(Lj.Wt + camAt(q) * Lj.camStride + (size_t)wy * Lj.pitch +
                                                            tx * kBlendTW + wc);
            if (inside(p, Lj.Wt, wBytes(R, Lj))) w[i] = __ldg(p);
        }
    }
#pragma unroll
    for (int q = 0; q < NC; q++)
        if (q < nc && hasF) S.fpw[q][fr * kFpW + fc + 3] = f[q];
#pragma unroll
    for (int i = 0; i < NC / 2; i++)
        if ((parts & kPartG) && (t >> 7) + 2 * i < nc) *reinterpret_cast<uint4*>(&S.gj[(t >> 7) + 2 * i][gr][gc]) = g[i];
#pragma unroll
    for (int i = 0; i < NC / 4; i++)
        if ((parts & kPartW) && (t >> 6) + 4 * i < nc) *reinterpret_cast<uint4*>(&S.w[(t >> 6) + 4 * i][wr][wc]) = w[i];
}

// ---- the zero-inserted upsample of a 2x2 block ----------------------------------
// Thread (lane, warp) owns rows ly = 2*warp, ly + 1 and columns lx = 2*lane,
// lx + 1 of the tile.  The upsample (weights 1 6 1 for an even output row or
// column, 4 4 for an odd one, over 64) reads footprint rows warp .. warp+2
// (even row: all three; odd row: the last two) and columns lane .. lane+2 the
// same way.  Words hold two channels in 16-bit lanes.  The common factors 4
// and 16 of the odd rows and columns are left out and taken off the final
// shift: (4x + 32) >> 6 = (x + 8) >> 4, (16x + 32) >> 6 = (x + 2) >> 2.
struct ColumnSums {
    uint32_t e, o;  // even row: a + 6 b + c; odd row: b + c
};
__device__ __forceinline__ ColumnSums columnSums(uint32_t a, uint32_t b, uint32_t c) { return {a + 6 * b + c, b + c}; }

// The block's four values, rounded and shifted; one: a 1 in every lane in use.
// Lane sums are at most 64 * 1023 + 32, so nothing carries between lanes; the
// shifts move bits from the upper lane into the lower, which the caller masks.
__device__ __forceinline__ void upsampleBlock(const ColumnSums* s, uint32_t one, uint32_t* out)
{
    out[0] = (s[0].e + s[2].e + 32 * one + 6 * s[1].e) >> 6;
    out[1] = (s[1].e + s[2].e + 8 * one) >> 4;
    out[2] = (s[0].o + s[2].o + 8 * one + 6 * s[1].o) >> 4;
    out[3] = (s[1].o + s[2].o + 2 * one) >> 2;
}

// U = pyrUp(G_{j+1}) of the block from three columns of three footprint rows:
// B | R << 16 in lo, G in hi, 0..255 each.
__device__ __forceinline__ void upsampleG(const uint32_t* a, const uint32_t* b, const uint32_t* c, uint32_t* lo,
                                          uint32_t* hi)
{
    ColumnSums sl[3], sh[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        sl[k] = columnSums(__byte_perm(a[k], 0, 0x4240), __byte_perm(b[k], 0, 0x4240), __byte_perm(c[k], 0, 0x4240));
        sh[k] = columnSums(__byte_perm(a[k], 0, 0x4341), __byte_perm(b[k], 0, 0x4341), __byte_perm(c[k], 0, 0x4341));
    }
    upsampleBlock(sl, 0x00010001u, lo);
    upsampleBlock(sh, 1u, hi);  // the fourth channel is 0
#pragma unroll
    for (int p = 0; p < 4; p++) lo[p] &= 0x00FF00FFu;
}
// The same from a staged footprint (row pitch kFpW).
__device__ __forceinline__ void upsampleG(const uint32_t* g, uint32_t* lo, uint32_t* hi)
{
    upsampleG(g, g + kFpW, g + 2 * kFpW, lo, hi);
}

// ---- the collapsed levels C_j ---------------------------------------------------
// A pixel is two words, B | R << 16 and G, each lane the value + kCBias.  |C| <
// 8700 (see ps_device.cuh), so a lane is a signed 16-bit number; nearly always
// C lies in -256 .. 767, where the lanes are 0..1023 and the upsample runs two
// channels per word (cInRange).
__device__ __forceinline__ uint2 packC(int b, int g, int r)
{
    return make_uint2((uint32_t)(uint16_t)(b + kCBias) | ((uint32_t)(uint16_t)(r + kCBias) << 16),
                      (uint32_t)(uint16_t)(g + kCBias));
}

// The thread's nine footprint pixels of C_{j+1}.
struct CFootprint {
    uint2 v[3][3];  // [row][column]
};
__device__ __forceinline__ CFootprint loadC(const uint2* cf)
{
    CFootprint f;
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int k = 0; k < 3; k++) f.v[r][k] = cf[r * kCfW + k];
    return f;
}
__device__ __forceinline__ bool cInRange(const CFootprint& f)
{
    uint32_t any = 0;
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int k = 0; k < 3; k++) any |= f.v[r][k].x | f.v[r][k].y;
    return (any & 0xFC00FC00u) == 0;
}
// pyrUp(C_{j+1}) of the block, biased by kCBias: B | R << 16 in lo, G in hi.
__device__ __forceinline__ void upsampleC(const CFootprint& f, uint32_t* lo, uint32_t* hi)
{
    ColumnSums sl[3], sh[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        sl[k] = columnSums(f.v[0][k].x, f.v[1][k].x, f.v[2][k].x);
        sh[k] = columnSums(f.v[0][k].y, f.v[1][k].y, f.v[2][k].y);
    }
    upsampleBlock(sl, 0x00010001u, lo);
    upsampleBlock(sh, 1u, hi);
#pragma unroll
    for (int p = 0; p < 4; p++) lo[p] &= 0x03FF03FFu;
}
// The same for any values, added to n[p] = (B, G, R).
__device__ __forceinline__ void addUpsampledC(const CFootprint& f, int (*n)[3])
{
#pragma unroll
    for (int ch = 0; ch < 3; ch++) {
        int e[3], o[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            int v[3];
#pragma unroll
            for (int r = 0; r < 3; r++)
                v[r] = ch == 0 ? (int)(short)f.v[r][k].x : (ch == 2 ? (int)f.v[r][k].x >> 16 : (int)(short)f.v[r][k].y);
            e[k] = v[0] + 6 * v[1] + v[2];
            o[k] = v[1] + v[2];
        }
        n[0][ch] += ((e[0] + 6 * e[1] + e[2] + 32) >> 6) - kCBias;
        n[1][ch] += ((e[1] + e[2] + 8) >> 4) - kCBias;
        n[2][ch] += ((o[0] + 6 * o[1] + o[2] + 8) >> 4) - kCBias;
        n[3][ch] += ((o[1] + o[2] + 2) >> 2) - kCBias;
    }
}

// The block's collapsed level (j >= 1) from its four pixels' words.
__device__ __forceinline__ void storeC(const UnitGeo& G, int x, int y, const uint2* v)
{
    const long long cext = (long long)G.pitch * G.h * 8;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (y + r >= G.h) break;
        uint2* Cj = reinterpret_cast<uint2*>(G.C) + (size_t)(y + r) * G.pitch + x;
        if (x + 1 < G.w) {
            if (inside(reinterpret_cast<uint4*>(Cj), G.C, cext))
                *reinterpret_cast<uint4*>(Cj) = make_uint4(v[2 * r].x, v[2 * r].y, v[2 * r + 1].x, v[2 * r + 1].y);
        } else if (x < G.w && inside(Cj, G.C, cext)) {
            Cj[0] = v[2 * r];
        }
    }
}

// The block's output pixels (level 0), o[2 * row + column] = B | G << 8 | R << 16;
// the render's canvas is even in both directions, the blender's need not be.
__device__ __forceinline__ void storeOut(const UnitGeo& G, int x, int y, const uint32_t* o)
{
    const int rows = y + 1 < G.h ? 2 : 1, cols = x + 1 < G.w ? 2 : 1;
    if (G.outFmt == PS_FMT_YUV420P || G.outFmt == PS_FMT_NV12) {  // even sizes only (checked at the API)
        storeYuv(G, x, y, o);
        return;
    }
    const long long oext = G.outPitch * G.h;
    for (int r = 0; r < rows; r++) {
        uint8_t* orow = G.out + (size_t)(y + r) * G.outPitch;
        if (G.outFmt == PS_FMT_BGR32) {
            if (cols == 2 && (reinterpret_cast<uintptr_t>(orow) & 7) == 0) {
                if (inside(reinterpret_cast<uint2*>(orow) + x / 2, G.out, oext))
                    reinterpret_cast<uint2*>(orow)[x / 2] = make_uint2(o[2 * r], o[2 * r + 1]);
            } else {
                if (inside(reinterpret_cast<uint32_t*>(orow) + x, G.out, oext))
                    reinterpret_cast<uint32_t*>(orow)[x] = o[2 * r];
                if (cols == 2 && inside(reinterpret_cast<uint32_t*>(orow) + x + 1, G.out, oext))
                    reinterpret_cast<uint32_t*>(orow)[x + 1] = o[2 * r + 1];
            }
        } else {
            for (int i = 0; i < cols; i++) {
                const uint32_t v = o[2 * r + i];
                if (!insideRange(orow + 3 * (x + i), 3, G.out, oext)) continue;
                orow[3 * (x + i)] = v & 0xFF;
                orow[3 * (x + i) + 1] = (v >> 8) & 0xFF;
                orow[3 * (x + i) + 2] = (v >> 16) & 0xFF;
            }
        }
    }
}

// The Laplacian L = G - U of one pixel, B and R in the two 16-bit lanes of one
// word, each biased by 256 so that neither the lane sums nor the subtraction
// carry or borrow across lanes (one PRMT puts a byte and the 1 of the bias into
// a lane).
__device__ __forceinline__ uint32_t biasedBR(uint32_t px) { return __byte_perm(px, 0x01010101u, 0x4240); }
__device__ __forceinline__ uint32_t biasedG(uint32_t px) { return __byte_perm(px, 0x01010101u, 0x4341); }

// A 2x2 block of a uniform tile (one camera, weight 256 everywhere: 80% of
// level 0 of the six-camera rig) is G - U + pyrUp(C), both upsamples, the sum
// and the saturation two channels per word: half the instructions of the
// general path, which such a block takes only where C leaves the packed range.
// px: the block's pixels of G; ulo .. chi: upsampleG's and upsampleC's.
__device__ __forceinline__ void finishUniform(const UnitGeo& G, int j, int x, int y, const uint32_t* px, const uint32_t* ulo,
                                              const uint32_t* uhi, const uint32_t* clo, const uint32_t* chi)
{
    // lanes: (256 + G - U) + (256 + C), at least 1
    uint32_t br[4], gg[4];
#pragma unroll
    for (int p = 0; p < 4; p++) {
        br[p] = biasedBR(px[p]) - ulo[p] + clo[p];
        gg[p] = biasedG(px[p]) - uhi[p] + chi[p];
    }
    if (j > 0) {
        uint2 v[4];
#pragma unroll
        for (int p = 0; p < 4; p++)  // back to one bias, as signed lanes (the fourth channel 0)
            v[p] = make_uint2(__viaddmax_s16x2(br[p], 0xFF00FF00u, 0x80008000u),
                              __viaddmax_s16x2(gg[p], 0xFF00FF00u, 0x80008000u));
        storeC(G, x, y, v);
        return;
    }
    if (y >= G.h || x >= G.w) return;
    uint32_t o[4];
#pragma unroll
    for (int p = 0; p < 4; p++)  // min(max(lane - 512, 0), 255)
        o[p] = __viaddmin_s16x2_relu(br[p], 0xFE00FE00u, 0x00FF00FFu) +
               (__viaddmin_s16x2_relu(gg[p], 0xFE00FE00u, 0x00FF00FFu) << 8);
    storeOut(G, x, y, o);
}

// One camera's part of the general path: w * L, and w.
__device__ __forceinline__ void accumulateBlock(BlendAcc& acc, const uint32_t* px, const uint32_t* ulo, const uint32_t* uhi,
                                                const uint32_t* wq)
{
#pragma unroll
    for (int p = 0; p < 4; p++) {
        // w * (256 + L); the 256 * sum(w) comes off at normalisation
        const uint32_t br = biasedBR(px[p]) - ulo[p];
        const int g = (int)(biasedG(px[p]) & 0xFFFFu) - (int)uhi[p];
        const int w = (int)((wq[p >> 1] >> (16 * (p & 1))) & 0xFFFFu);
        acc.r[p][0] += w * (int)(br & 0xFFFFu);
        acc.r[p][1] += w * g;
        acc.r[p][2] += w * (int)(br >> 16);
        acc.wsum[p] += w;
    }
}

// Normalise, collapse (loadUp: the C_{j+1} footprint, called where there is one)
// and store.
template <class LoadUp>
__device__ __forceinline__ void finishBlock(const UnitGeo& G, int j, int cls, int x, int y, BlendAcc& acc, LoadUp loadUp)
{
    int n[4][3];
#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
        for (int c = 0; c < 3; c++) acc.r[p][c] -= acc.wsum[p] << 8;
    if (G.full) {
#pragma unroll
        for (int p = 0; p < 4; p++)
#pragma unroll
            for (int c = 0; c < 3; c++) n[p][c] = (acc.r[p][c] + 128) >> 8;
    } else if (j == 0 && __all_sync(0xffffffffu, ((acc.wsum[0] | acc.wsum[1] | acc.wsum[2] | acc.wsum[3]) & ~256) == 0)) {
        // Level-0 weights are the 0/256 seam masks.  Where each pixel's sum is 0 or 256 (one camera at
        // most: always, unless custom masks overlap), R = 256 L exactly, and R / W truncated is the shift.
#pragma unroll
        for (int p = 0; p < 4; p++)
#pragma unroll
            for (int c = 0; c < 3; c++) n[p][c] = acc.r[p][c] >> 8;
    } else {
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int d = acc.wsum[p] ? acc.wsum[p] : 1;
            const float inv = __frcp_rn((float)d);
#pragma unroll
            for (int c = 0; c < 3; c++) n[p][c] = divTrunc(acc.r[p][c], d, inv);
        }
    }
    // collapse: + pyrUp32(C_{j+1})
    if (G.hasUp != 0 && !(j == 0 && cls == 0)) addUpsampledC(loadUp(), n);
    if (j > 0) {
        uint2 v[4];
#pragma unroll
        for (int p = 0; p < 4; p++) v[p] = packC(n[p][0], n[p][1], n[p][2]);
        storeC(G, x, y, v);
        return;
    }
    if (y >= G.h || x >= G.w) return;
    uint32_t o[4] = {0, 0, 0, 0};
    if (cls != 0) {
#pragma unroll
        for (int p = 0; p < 4; p++)
            o[p] = packSatBgr(n[p][0], n[p][1], n[p][2]);
        if (cls == 2) {
            const long long uext = (long long)G.pitch * G.h;
            const int rows = y + 1 < G.h ? 2 : 1, cols = x + 1 < G.w ? 2 : 1;
            for (int r = 0; r < rows; r++) {
                const uint8_t* um = G.um + (size_t)(y + r) * G.pitch + x;
                if (!(inside(um, G.um, uext) ? um[0] : 0)) o[2 * r] = 0;
                if (cols == 2 && !(inside(um + 1, G.um, uext) ? um[1] : 0)) o[2 * r + 1] = 0;
            }
        }
    }
    storeOut(G, x, y, o);
}

// Accumulate one unit from its stage; at a tile's last unit normalise,
// collapse and store.  Threads 0..kConsumers-1.
template <class Stage>
__device__ __forceinline__ void computeUnit(const Stage& S, const UnitGeo& G, const uint4& raw, int chunk, BlendAcc& acc)
{
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int lx = 2 * lane, ly = 2 * wp;
    const int j = raw.x & 0xFF, cls = (raw.x >> 8) & 0xFF, camCnt = (raw.x >> 16) & 0xFF;
    const bool uni = ((raw.x >> 24) & kTileUniform) != 0;  // weights are not read
    const int tx = raw.y & 0xFFFF, ty = raw.y >> 16;
    const bool hasUp = G.hasUp != 0;
    const int x = tx * kBlendTW + lx, y = ty * kBlendTH + ly;
    constexpr int NC = Stage::kCams;
    const int nc = max(0, min(NC, camCnt - chunk * NC));
    auto pixels = [&](int q, uint32_t* px) {
        const uint2 gt = *reinterpret_cast<const uint2*>(&S.gj[q][ly][lx]);
        const uint2 gb = *reinterpret_cast<const uint2*>(&S.gj[q][ly + 1][lx]);
        px[0] = gt.x;
        px[1] = gt.y;
        px[2] = gb.x;
        px[3] = gb.y;
    };
    if (uni && hasUp) {
        const CFootprint cf = loadC(&S.cf[wp][1 + lane]);
        if (__all_sync(0xffffffffu, cInRange(cf))) {
            uint32_t ulo[4], uhi[4], clo[4], chi[4], px[4];
            upsampleG(&S.fpw[0][wp * kFpW + 3 + lane], ulo, uhi);
            upsampleC(cf, clo, chi);
            pixels(0, px);
            finishUniform(G, j, x, y, px, ulo, uhi, clo, chi);
            return;
        }
    }
    if (chunk == 0) acc = BlendAcc{};
    if (!(j == 0 && cls == 0)) {
        for (int q = 0; q < nc; q++) {
            uint32_t ulo[4] = {0, 0, 0, 0}, uhi[4] = {0, 0, 0, 0}, px[4];
            if (hasUp) upsampleG(&S.fpw[q][wp * kFpW + 3 + lane], ulo, uhi);
            pixels(q, px);
            uint32_t wq[2] = {0x01000100u, 0x01000100u};
            if (!uni) {
                wq[0] = *reinterpret_cast<const uint32_t*>(&S.w[q][ly][lx]);
                wq[1] = *reinterpret_cast<const uint32_t*>(&S.w[q][ly + 1][lx]);
            }
            accumulateBlock(acc, px, ulo, uhi, wq);
        }
    }
    if (chunk == unitChunks<NC>(raw) - 1) finishBlock(G, j, cls, x, y, acc, [&] { return loadC(&S.cf[wp][1 + lane]); });
}

// The Laplacian of one pixel in half tiles: U unrounded, scaled by 64.
struct Lap {
    uint32_t br;  // (256 + L_B) | (256 + L_R) << 16
    int g;        // L_G
};

__device__ __forceinline__ Lap laplacian(uint32_t gpx, uint32_t ulo, uint32_t uhi)
{
    const uint32_t ubr = ((ulo + 0x00200020u) >> 6) & 0x03FF03FFu;  // round(U) of B and R, per lane
    Lap l;
    l.br = biasedBR(gpx) - ubr;
    l.g = (int)__byte_perm(gpx, 0, 0x4441) - (int)(((uhi & 0xFFFFu) + 32u) >> 6);
    return l;
}

// k_blend_small's variant, for levels above 0: one 64x8 half of a tile
// (rows 8*half ..), consumer thread t owning pixels (2*(t%32), t/32) and the
// one to its right, so all eight warps share the few tiles of these levels.
// Same arithmetic as computeUnit; output is the collapsed level C_j.
struct PairAcc {
    int r0[3], r1[3];
    int wsum0, wsum1;
};

// The thread's element of the C_{j+1} footprint.
__device__ __forceinline__ size_t halfCOffset(const RigDev& R, const uint4& raw, int half)
{
    const int j = raw.x & 0xFF, r = threadIdx.x / kFW, c = threadIdx.x % kFW;
    if (j >= R.L || r >= HalfStage::kFpRows) return 0;
    return halfFpOffset(R.lv[j + 1], R.lv[j], raw.y & 0xFFFF, raw.y >> 16, half, r, c);
}
__device__ __forceinline__ void stageHalfC(HalfStage& S, const RigDev& R, int j, size_t offset)
{
    const int r = threadIdx.x / kFW, c = threadIdx.x % kFW;
    if (j >= R.L || r >= HalfStage::kFpRows) return;
    const LevelDev& Lu = R.lv[j + 1];
    const uint2* p = reinterpret_cast<const uint2*>(Lu.C + offset);
    S.cf[r][c + 1] = inside(p, Lu.C, cBytes(Lu)) ? __ldg(p) : make_uint2(0, 0);
}

// Accumulate one unit's cameras.
__device__ __forceinline__ void accumulateRows(const HalfStage& S, const UnitGeo& G, const uint4& raw, int chunk,
                                               PairAcc& acc)
{
    const int lx = (threadIdx.x & 31) * 2, ly = threadIdx.x >> 5;  // row in the half tile
    // vertical taps: even rows footprint rows ly/2 .. ly/2+2 (1 6 1), odd rows
    // (ly+1)/2 .. (ly+1)/2+1 (4 4); footprint columns lx/2 .. lx/2+2 as in computeUnit
    const bool evenRow = (ly & 1) == 0;
    const int vr0 = evenRow ? ly / 2 : (ly + 1) / 2;
    const int fc = lx / 2;
    const int camCnt = (raw.x >> 16) & 0xFF;
    const bool hasUp = G.hasUp != 0;
    constexpr int NC = HalfStage::kCams;
    const int nc = max(0, min(NC, camCnt - chunk * NC));
    if (chunk == 0) acc = PairAcc{};
#pragma unroll 2
    for (int q = 0; q < nc; q++) {
        uint32_t u0lo = 0, u0hi = 0, u1lo = 0, u1hi = 0;
        if (hasUp) {
            const uint32_t* g = &S.fpw[q][0] + 3;
            uint32_t vlo[3], vhi[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const uint2 a = unpackBytes(g[vr0 * kFpW + fc + k]);
                const uint2 b = unpackBytes(g[(vr0 + 1) * kFpW + fc + k]);
                if (evenRow) {
                    const uint2 c = unpackBytes(g[(vr0 + 2) * kFpW + fc + k]);
                    vlo[k] = a.x + 6 * b.x + c.x;
                    vhi[k] = a.y + 6 * b.y + c.y;
                } else {
                    vlo[k] = 4 * (a.x + b.x);
                    vhi[k] = 4 * (a.y + b.y);
                }
            }
            u0lo = vlo[0] + 6 * vlo[1] + vlo[2];
            u0hi = vhi[0] + 6 * vhi[1] + vhi[2];
            u1lo = 4 * (vlo[1] + vlo[2]);
            u1hi = 4 * (vhi[1] + vhi[2]);
        }
        const uint2 gq = *reinterpret_cast<const uint2*>(&S.gj[q][ly][lx]);
        const uint32_t wq = *reinterpret_cast<const uint32_t*>(&S.w[q][ly][lx]);
        const int w0 = (int)(wq & 0xFFFFu), w1 = (int)(wq >> 16);
        // B and R accumulate w * (256 + L); the 256 * sum(w) comes off below
        const Lap l0 = laplacian(gq.x, u0lo, u0hi), l1 = laplacian(gq.y, u1lo, u1hi);
        acc.r0[0] += w0 * (int)(l0.br & 0xFFFFu);
        acc.r0[1] += w0 * l0.g;
        acc.r0[2] += w0 * (int)(l0.br >> 16);
        acc.r1[0] += w1 * (int)(l1.br & 0xFFFFu);
        acc.r1[1] += w1 * l1.g;
        acc.r1[2] += w1 * (int)(l1.br >> 16);
        acc.wsum0 += w0;
        acc.wsum1 += w1;
    }
}

// The two pixels' normalised values.
__device__ __forceinline__ void normaliseRows(const UnitGeo& G, PairAcc& acc, int* n0, int* n1)
{
    acc.r0[0] -= acc.wsum0 << 8;
    acc.r0[2] -= acc.wsum0 << 8;
    acc.r1[0] -= acc.wsum1 << 8;
    acc.r1[2] -= acc.wsum1 << 8;
    if (G.full) {
#pragma unroll
        for (int c = 0; c < 3; c++) { n0[c] = (acc.r0[c] + 128) >> 8; n1[c] = (acc.r1[c] + 128) >> 8; }
    } else {
        const int d0 = acc.wsum0 ? acc.wsum0 : 1, d1 = acc.wsum1 ? acc.wsum1 : 1;
        const float i0 = __frcp_rn((float)d0), i1 = __frcp_rn((float)d1);
#pragma unroll
        for (int c = 0; c < 3; c++) { n0[c] = divTrunc(acc.r0[c], d0, i0); n1[c] = divTrunc(acc.r1[c], d1, i1); }
    }
}

// Collapse (the staged C_{j+1} footprint) and store.
__device__ __forceinline__ void collapseRows(const HalfStage& S, const UnitGeo& G, int x, int y, int* n0, int* n1)
{
    if (G.hasUp) {
        const int ly = threadIdx.x >> 5, fc = threadIdx.x & 31;
        const bool evenRow = (ly & 1) == 0;
        const int vr0 = evenRow ? ly / 2 : (ly + 1) / 2;
        const uint2* cf = &S.cf[0][0] + 1;
        int v[3][3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const uint2 a = cf[vr0 * kCfW + fc + k], b = cf[(vr0 + 1) * kCfW + fc + k];
            const int ax = (short)a.x, ay = (short)a.y, az = (int)a.x >> 16;  // B, G, R
            const int bx = (short)b.x, by = (short)b.y, bz = (int)b.x >> 16;
            if (evenRow) {
                const uint2 c = cf[(vr0 + 2) * kCfW + fc + k];
                v[k][0] = ax + 6 * bx + (short)c.x;
                v[k][1] = ay + 6 * by + (short)c.y;
                v[k][2] = az + 6 * bz + ((int)c.x >> 16);
            } else {
                v[k][0] = 4 * (ax + bx);
                v[k][1] = 4 * (ay + by);
                v[k][2] = 4 * (az + bz);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            n0[c] += ((v[0][c] + 6 * v[1][c] + v[2][c] + 32) >> 6) - kCBias;
            n1[c] += ((4 * (v[1][c] + v[2][c]) + 32) >> 6) - kCBias;
        }
    }
    uint2* Cj = reinterpret_cast<uint2*>(G.C) + (size_t)y * G.pitch + x;
    const long long cext = (long long)G.pitch * G.h * 8;
    const uint2 c0 = packC(n0[0], n0[1], n0[2]), c1 = packC(n1[0], n1[1], n1[2]);
    if (x + 1 < G.w) {
        if (inside(reinterpret_cast<uint4*>(Cj), G.C, cext))
            *reinterpret_cast<uint4*>(Cj) = make_uint4(c0.x, c0.y, c1.x, c1.y);
    } else if (x < G.w && inside(Cj, G.C, cext)) {
        Cj[0] = c0;
    }
}

// Tiles are handed out in runs of up to kBlendRun through `counter` (zero at
// launch), so a CTA that starts late, behind other frames' kernels, simply takes
// fewer.
//
// probePolls > 0 is the failure-path test of the bounded waits: consumer
// thread 0 first waits that many polls on an mbarrier that nothing arrives
// on, so the wait runs out, and the timeout is reported as any other
// (kStatusBlend in every frame of the launch).
__global__ void __launch_bounds__(kBlendThreads, 4) k_blend(const Segment* __restrict__ gsegs, int nsegs, int total,
                                                            int* __restrict__ counter, int probePolls, int early)
{
    __shared__ BlendStage st[kBStages];
    __shared__ UnitInfo info[kBStages];
    __shared__ uint64_t full[kBStages], empty[kBStages], never;
    __shared__ Segment s_segs[kMaxSmemSegs];
    __shared__ int s_timeout;
    __shared__ int fRow[kFH], fCol[kFW];
    const Segment* segs = gsegs;
    if (nsegs <= kMaxSmemSegs) {
        for (int k = threadIdx.x; k < nsegs; k += kBlendThreads) s_segs[k] = gsegs[k];
        segs = s_segs;
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < kBStages; k++) {
            mbarInit(&full[k], 1);
            mbarInit(&empty[k], kConsumers / 32);
        }
        mbarInit(&never, 1);
        s_timeout = 0;
    }
    if (threadIdx.x < kBStages) {
        info[threadIdx.x].valid = 0;  // a stage read after a wait ran out ends the loop
        info[threadIdx.x].seg = -1;   // its geometry is not filled in
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;

    if (threadIdx.x >= kConsumers) {
        // ---------------- producer warp ----------------
        // The hand-out counter, items and descriptors are written before the
        // launch sequence, not by a kernel: the first unit is worked out
        // while the previous kernel finishes, and the wait comes before its
        // first copy of level data -- or, with early set (every blend step
        // after the first, where the launch before this one wrote only C
        // levels), before its first copy of C_{j+1}: its G_j, weights and
        // G_{j+1} footprint, written by launches that have completed, are
        // copied (through L2, by the tensor copies) while it finishes.
        bool waited = false;
        // Tiles are taken in runs, a lane holding a tile's descriptor; the next
        // run is fetched once the first unit of the one in use is on its way.
        int seg = -1, chunk = 0;
        uint4 raw = make_uint4(0, 0, 0, 0);
        bool valid = false;
        uint4 laneRaw = raw, nextRaw = raw;
        int laneSeg = 0, nextSeg = 0, len = 0, nextLen = 0, at = 0, pos = 0;
        bool ahead = false;  // the next run is fetched
        auto fetchRun = [&] {
            const int want = max(1, min(kBlendRun, (total - pos) / (kBlendShare * (int)gridDim.x)));
            int it = 0;
            if (lane == 0) it = atomicAdd(counter, want);
            it = pos = __shfl_sync(0xffffffffu, it, 0);
            nextLen = max(0, min(want, total - it));
            if (lane < nextLen) {
                nextSeg = findSegment(segs, nsegs, it + lane, nextSeg);
                nextRaw = __ldg(static_cast<const uint4*>(segs[nextSeg].items) + (it + lane - segs[nextSeg].prefix));
            }
            ahead = true;
        };
        // of the segment (one level of one rig)
        int h = 0, uw = 0, uh = 0;
        bool hasUp = false;
        const uint8_t *tmJ = nullptr, *tmU = nullptr;  // tensor maps of the level and of the one above
        const uint8_t* camLists = nullptr;
        auto takeNext = [&] {
            if (at == len) {
                laneRaw = nextRaw;
                laneSeg = nextSeg;
                len = nextLen;
                at = 0;
                ahead = false;
            }
            valid = len > 0;
            if (!valid) return;
            raw.x = __shfl_sync(0xffffffffu, laneRaw.x, at);
            raw.y = __shfl_sync(0xffffffffu, laneRaw.y, at);
            raw.z = __shfl_sync(0xffffffffu, laneRaw.z, at);
            raw.w = __shfl_sync(0xffffffffu, laneRaw.w, at);
            const int s = __shfl_sync(0xffffffffu, laneSeg, at);
            at++;
            if (s != seg) {
                seg = s;
                const RigDev& R = *segs[seg].rig;
                const int j = raw.x & 0xFF;
                hasUp = j < R.L;
                h = R.lv[j].h;
                uw = R.lv[hasUp ? j + 1 : j].w;
                uh = R.lv[hasUp ? j + 1 : j].h;
                tmJ = R.tmaps ? static_cast<const uint8_t*>(R.tmaps) + (size_t)j * kTmapsPerLevel * 128 : nullptr;
                tmU = tmJ + kTmapsPerLevel * 128;
                camLists = R.camLists;
            }
        };
        fetchRun();
        takeNext();
        for (int u = 0;; u++) {
            const int stg = u % kBStages;
            if (u >= kBStages && !mbarWait(&empty[stg], ((u / kBStages) - 1) & 1)) s_timeout = 1;
            const int tx = raw.y & 0xFFFF, ty = raw.y >> 16;
            const int fx0 = tx * (kBlendTW / 2) - 1, fy0 = ty * (kBlendTH / 2) - 1;
            const int nc = max(0, min(kCamsPerUnit, (int)((raw.x >> 16) & 0xFF) - chunk * kCamsPerUnit));
            const bool last = chunk == unitChunks(raw) - 1, uni = ((raw.x >> 24) & kTileUniform) != 0;
            bool staged = false;  // by tensor copies; else the consumers stage the unit
#ifndef PS_CHECK_BOUNDS
            staged = valid && tmJ && !((raw.x & 0xFFFF) == 0) && (ty + 1) * kBlendTH <= h && (nc > 0 || (hasUp && last)) &&
                     (!hasUp || (fx0 - 3 >= 0 && fx0 - 3 + kFpW <= uw && fy0 >= 0 && fy0 + kFH <= uh));
#endif
            fenceProxyAsync();
            if (lane == 0) {
                UnitInfo& I = info[stg];
                I.raw = raw;
                I.chunk = chunk;
                I.valid = valid;
                I.staged = staged;
                if (valid && I.seg != seg) {
                    I.seg = seg;
                    fillGeo(I.geo, *segs[seg].rig, *segs[seg].frame, raw.x & 0xFF);
                }
            }
            if (!waited && !(early && staged)) {
                waitPrevGrid();
                allowNextGrid();
                waited = true;
            }
            if (staged) {
                // one bulk tensor copy per camera and array: the G_j tile,
                // its weights, its G_{j+1} footprint; then the C_{j+1} footprint
                if (lane == 0) {
                    mbarArriveExpectTx(&full[stg], nc * (kBlendTH * kBlendTW * 4 + (uni ? 0 : kBlendTH * kBlendTW * 2) +
                                                         (hasUp ? kFH * kFpW * 4 : 0)) +
                                                       (hasUp && last ? kFH * kCfW * 8 : 0));
                    for (int q = 0; q < nc; q++) {
                        const int cam = tileCam(raw, camLists, chunk * kCamsPerUnit + q);
                        tmaLoad3d(&st[stg].gj[q][0][0], tmJ + kTmG * 128, tx * kBlendTW, ty * kBlendTH, cam, &full[stg]);
                        if (!uni)
                            tmaLoad3d(&st[stg].w[q][0][0], tmJ + kTmW * 128, tx * kBlendTW, ty * kBlendTH, cam, &full[stg]);
                        if (hasUp) tmaLoad3d(&st[stg].fpw[q][0], tmU + kTmGfp * 128, fx0 - 3, fy0, cam, &full[stg]);
                    }
                }
                if (!waited) {  // C_{j+1} is the previous launch's output
                    __syncwarp();
                    waitPrevGrid();
                    allowNextGrid();
                    waited = true;
                }
                if (lane == 0 && hasUp && last) tmaLoad2d(&st[stg].cf[0][0], tmU + kTmC * 128, fx0 - 1, fy0, &full[stg]);
            } else if (lane == 0) {
                mbarArrive(&full[stg]);
            }
            if (!valid) break;  // the terminal unit is out
            if (!ahead) fetchRun();
            if (chunk + 1 < unitChunks(raw)) {
                chunk++;
            } else {
                chunk = 0;
                takeNext();
            }
            __syncwarp();
        }
        return;
    }

    // ---------------- consumer warps ----------------
    waitPrevGrid();
    allowNextGrid();
    if (probePolls > 0 && threadIdx.x == 0 && !mbarWait(&never, 0, probePolls)) s_timeout = 1;
    BlendAcc acc;
    for (int u = 0;; u++) {
        const int stg = u % kBStages;
        if (!mbarWait(&full[stg], (u / kBStages) & 1)) s_timeout = 1;
        const UnitInfo& ui = info[stg];  // rewritten only after this warp releases the stage
        const uint4 raw = ui.raw;
        if (!ui.valid) break;
        const int chunk = ui.chunk;
        const bool staged = ui.staged != 0;
        const bool active = !((raw.x & 0xFF) == 0 && ((raw.x >> 8) & 0xFF) == 0);
        if (active && !staged) {
            stageUnitDirect(st[stg], *segs[ui.seg].rig, raw, chunk, fRow, fCol,
                                   [] { namedBarrier(1, kConsumers); });
            namedBarrier(1, kConsumers);
        }
        computeUnit(st[stg], ui.geo, raw, chunk, acc);
        if (active && !staged) fenceProxyAsync();  // our stage writes precede later bulk copies into it
        __syncwarp();
        if (lane == 0) mbarArrive(&empty[stg]);  // this warp is done with the stage
    }
    // The producer's timeouts precede its terminal arrive, which every
    // consumer has waited on; the consumers' own meet here.  A desynchronised
    // ring can have corrupted any unit, so every frame of the launch is flagged.
    namedBarrier(1, kConsumers);
    if (s_timeout && threadIdx.x == 0) flagTimeout(segs, nsegs, kStatusBlend);
}

// ============================================================================
// k_blend_rows: k_blend's levels of few tiles (kRowsWork), without the ring: a
// warp takes kPairs row pairs of a tile and loads what they need straight into
// registers.  A uniform tile's footprint rows go from one pair to the next.  The
// ring's warm-up (a producer's trips before the first copy, the copies, a CTA's
// eight warps on one tile) is what a launch of few tiles consists of; on larger
// levels the ring's bulk copies move more (level 0 of 4096x2048: 45 us by rows,
// 40 us by the ring; of 7680x3840: 107 and 83 us).  256x128: 28.5 us a frame,
// 31.0 with the ring; 2048x1024: 74.0 against 78.4; 4096x2048: 158.4 against 160.0.
// ============================================================================
// The line between the two: the tiles' cameras, counted over the level's tiles.
// 2048 mostly uniform tiles (level 0 of 2048x1024) are 4.3 us shorter here, 1800
// tiles of two cameras (level 2 of the 8K ring) as long, 2048 tiles and 2500
// cameras (level 1 of 6 x 1920x1080 to 4096x2048) 0.8 us longer, eight frames
// in flight 8 us.
constexpr int kRowsWork = 2200;
constexpr int kRowsCtas = 3;  // CTAs per SM: 80 registers (64 spill, 2 us more)

// The levels of a unit's segment and its output, a copy a warp.
struct RowsGeo {
    LevelDev j, u;
    UnitGeo g;
    const uint8_t* camLists;
    int n;
};
static_assert(sizeof(LevelDev) / 4 <= 16, "two descriptions a warp, a word a lane");

__device__ __forceinline__ void fillRowsGeo(RowsGeo& b, const RigDev& R, const FrameDev& F, int j)
{
    const int lane = threadIdx.x & 31, k = lane & 15;
    __syncwarp();
    if (k < (int)sizeof(LevelDev) / 4)
        reinterpret_cast<uint32_t*>(lane < 16 ? &b.j : &b.u)[k] =
            __ldg(reinterpret_cast<const uint32_t*>(&R.lv[lane < 16 ? j : min(j + 1, R.L)]) + k);
    if (lane == 0) {
        fillGeo(b.g, R, F, j);
        b.camLists = R.camLists;
        b.n = R.n;
    }
    __syncwarp();
}

// Pixel (x, y) of camera cam at the unit's level, rows y and y + 1.
__device__ __forceinline__ void rowsPixels(const RowsGeo& B, int cam, int x, int y, uint32_t* px)
{
    const uint2* p = reinterpret_cast<const uint2*>(B.j.G + (size_t)cam * B.j.camStride + (size_t)y * B.j.pitch + x);
    const uint2* q = p + B.j.pitch / 2;
    const long long ext = (long long)B.n * B.j.camStride * 4;
    const uint2 t = inside(p, B.j.G, ext) ? __ldg(p) : make_uint2(0, 0);
    const uint2 b = y + 1 < B.j.h && inside(q, B.j.G, ext) ? __ldg(q) : make_uint2(0, 0);
    px[0] = t.x;
    px[1] = t.y;
    px[2] = b.x;
    px[3] = b.y;
}
// Three columns of a row of the level above: a camera's G, and C.
__device__ __forceinline__ void rowsFootprint(const RowsGeo& B, const uint32_t* row, const int* col, uint32_t* f)
{
#pragma unroll
    for (int k = 0; k < 3; k++)
        f[k] = inside(row + col[k], B.u.G, (long long)B.n * B.u.camStride * 4) ? __ldg(row + col[k]) : 0u;
}
__device__ __forceinline__ void rowsFootprint(const RowsGeo& B, const uint2* row, const int* col, uint2* f)
{
#pragma unroll
    for (int k = 0; k < 3; k++) f[k] = inside(row + col[k], B.u.C, cBytes(B.u)) ? __ldg(row + col[k]) : make_uint2(0, 0);
}
__device__ __forceinline__ int rowsOffset(const RowsGeo& B, int y, int r)
{
    return rowMap(y / 2 - 1 + r, B.u.h) * B.u.pitch;
}

// One row pair, any cameras, any values.
__device__ __forceinline__ void rowsPair(const RowsGeo& B, const uint4& raw, int x, int y, const int* col)
{
    const int j = raw.x & 0xFF, cls = (raw.x >> 8) & 0xFF, camCnt = (raw.x >> 16) & 0xFF;
    const bool uni = ((raw.x >> 24) & kTileUniform) != 0, hasUp = B.g.hasUp != 0;
    BlendAcc acc{};
    if (!(j == 0 && cls == 0)) {
        for (int q = 0; q < camCnt; q++) {
            const int cam = tileCam(raw, B.camLists, q);
            uint32_t ulo[4] = {0, 0, 0, 0}, uhi[4] = {0, 0, 0, 0}, px[4], f[3][3];
            rowsPixels(B, cam, x, y, px);
            uint32_t wq[2] = {0x01000100u, 0x01000100u};
            if (!uni) {
                const uint32_t* p =
                    reinterpret_cast<const uint32_t*>(B.j.Wt + (size_t)cam * B.j.camStride + (size_t)y * B.j.pitch + x);
                const uint32_t* p1 = p + B.j.pitch / 2;
                const long long ext = (long long)B.n * B.j.camStride * 2;
                wq[0] = inside(p, B.j.Wt, ext) ? __ldg(p) : 0u;
                wq[1] = y + 1 < B.j.h && inside(p1, B.j.Wt, ext) ? __ldg(p1) : 0u;
            }
            if (hasUp) {
                const uint32_t* U = reinterpret_cast<const uint32_t*>(B.u.G) + (size_t)cam * B.u.camStride;
#pragma unroll
                for (int r = 0; r < 3; r++) rowsFootprint(B, U + rowsOffset(B, y, r), col, f[r]);
                upsampleG(f[0], f[1], f[2], ulo, uhi);
            }
            accumulateBlock(acc, px, ulo, uhi, wq);
        }
    }
    finishBlock(B.g, j, cls, x, y, acc, [&] {
        CFootprint c;
#pragma unroll
        for (int r = 0; r < 3; r++)
            rowsFootprint(B, reinterpret_cast<const uint2*>(B.u.C) + rowsOffset(B, y, r), col, c.v[r]);
        return c;
    });
}

template <int kPairs>
__global__ void __launch_bounds__(kThreads, kRowsCtas) k_blend_rows(const Segment* __restrict__ segs, int nsegs, int total,
                                                                    int probePolls)
{
    __shared__ RowsGeo s_geo[kThreads / 32];
    __shared__ uint64_t never;
    constexpr int kParts = kBlendTH / 2 / kPairs;  // units of a tile
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) mbarInit(&never, 1);
    __syncthreads();
    RowsGeo& B = s_geo[warp];
    const int units = total * kParts, first = blockIdx.x * (kThreads / 32) + warp;
    int seg = 0, filled = -1;
    for (int u = first; u < units; u += gridDim.x * (kThreads / 32)) {
        seg = findSegment(segs, nsegs, u / kParts, seg);
        const uint4 raw = __ldg(static_cast<const uint4*>(segs[seg].items) + (u / kParts - segs[seg].prefix));
        const int j = raw.x & 0xFF;
        if (seg != filled) fillRowsGeo(B, *segs[seg].rig, *segs[seg].frame, j);
        if (filled < 0) {  // items and descriptors are written before the launch sequence, not by a kernel
            waitPrevGrid();
            allowNextGrid();
            if (probePolls > 0 && threadIdx.x == 0 && !mbarWait(&never, 0, probePolls))
                flagTimeout(segs, nsegs, kStatusBlend);
        }
        filled = seg;
        const int tx = raw.y & 0xFFFF, ty = raw.y >> 16;
        const int x = tx * kBlendTW + 2 * lane, y0 = ty * kBlendTH + u % kParts * (2 * kPairs);
        const int rows = (B.g.h - y0 + 1) / 2;                     // row pairs inside the level
        int todo = rows <= 0 ? 0 : (1 << min(kPairs, rows)) - 1;  // left for the general path
        int col[3] = {0, 0, 0};
        if (B.g.hasUp) {
#pragma unroll
            for (int k = 0; k < 3; k++) col[k] = colMap(tx * (kBlendTW / 2) - 1 + lane + k, B.u.w);
        }
        if ((raw.x >> 24 & kTileUniform) && B.g.hasUp && rows >= kPairs) {
            const int cam = tileCam(raw, B.camLists, 0);
            const uint32_t* U = reinterpret_cast<const uint32_t*>(B.u.G) + (size_t)cam * B.u.camStride;
            const uint2* C = reinterpret_cast<const uint2*>(B.u.C);
            uint32_t f[kPairs + 2][3], px[kPairs][4];
            uint2 c[kPairs + 2][3];
#pragma unroll
            for (int r = 0; r < kPairs + 2; r++) {
                const int o = rowsOffset(B, y0, r);
                rowsFootprint(B, U + o, col, f[r]);
                rowsFootprint(B, C + o, col, c[r]);
            }
#pragma unroll
            for (int p = 0; p < kPairs; p++) rowsPixels(B, cam, x, y0 + 2 * p, px[p]);
            todo = 0;
#pragma unroll
            for (int p = 0; p < kPairs; p++) {
                CFootprint cf;
#pragma unroll
                for (int r = 0; r < 3; r++)
#pragma unroll
                    for (int k = 0; k < 3; k++) cf.v[r][k] = c[p + r][k];
                if (!__all_sync(0xffffffffu, cInRange(cf))) {
                    todo |= 1 << p;
                    continue;
                }
                uint32_t ulo[4], uhi[4], clo[4], chi[4];
                upsampleG(f[p], f[p + 1], f[p + 2], ulo, uhi);
                upsampleC(cf, clo, chi);
                finishUniform(B.g, j, x, y0 + 2 * p, px[p], ulo, uhi, clo, chi);
            }
        }
        for (; todo; todo &= todo - 1) rowsPair(B, raw, x, y0 + 2 * (__ffs(todo) - 1), col);
    }
    if (filled < 0) {
        waitPrevGrid();
        allowNextGrid();
    }
}

// ============================================================================
// k_tail: the levels of at most 32x16 pixels (one pyrDown tile a camera, one
// blend tile) of rigs of up to 16 cameras in one launch.  A launch a level is
// 3 us of release, loads and stores around some hundred nanoseconds of
// arithmetic.  Here a cluster owns a rig.  The levels' pyrDown needs no other
// camera, so a CTA takes a camera (two in small clusters) down all of them in
// its own shared memory and pushes every level into that of the cluster's last
// CTA, which blends them all from there: between two levels lie a CTA's barrier
// and a few shared loads, and one cluster barrier is left.  What does not
// depend on the frame (alpha divisors, weights, index maps with the reference's
// borders) is fetched while the launch before finishes.  The levels' buffers in
// memory are written as everywhere, for the levels below and the state export.
// A tail that also took the levels of up to 16 tiles, each spread over 16 CTAs
// with a cluster barrier between levels, cost as much as a launch a level did.
// The two levels of 6 x 1920x1080 to 4096x2048 (8 levels): 6.1 us from its
// release, and a frame of 172.5 us when it came (177.5 with a launch a level,
// 183.8 with that wider tail); 256x128: 33.7 us a frame against 40.6 and 42.4.
// ============================================================================
constexpr int kTailThreads = 512;     // a pixel of the largest level each
// of all levels of a plane: 512 + 128 + 32 + 8 + 2 + 1 + 1 ...
constexpr int kTailPx = 704;
static_assert(kTailThreads == kTailW * kTailH && kTailW == 32 && kTailH == 16, "tailLevel and tailPixel");
static_assert(PS_MAX_LEVELS <= 24, "levels of one pixel fit behind the others");

__device__ __forceinline__ void clusterArrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void clusterWait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// The address of a shared variable of this CTA in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t clusterAddr(const void* p, int rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void clusterStore(uint32_t addr, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void clusterStore(uint32_t addr, uint16_t v)
{
    asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(addr), "h"(v) : "memory");
}

struct TailSmem {
    RigDev rig;
    alignas(16) uint32_t in[2 * kTailH][2 * kTailW];  // the camera's level above the first
    uint32_t plane[kTailPx];              // the camera's levels
    uint16_t am[kTailPx];                 // their alpha divisors
    uint32_t magic[257];
    // the pixels that the borders' rules give a filter's columns and rows:
    // pyrDown column 2X - 2 + i at [2X + i], upsample column x / 2 - 1 + i at
    // [x / 2 + i], rows the same
    uint8_t downCol[PS_MAX_LEVELS + 1][72], downRow[PS_MAX_LEVELS + 1][40];
    uint8_t upCol[PS_MAX_LEVELS + 1][20], upRow[PS_MAX_LEVELS + 1][12];
    uint2 c[kTailPx];  // the collapsed levels (the last CTA's)
    // behind it in the last CTA: every camera's levels, then their weights
};
constexpr int kTailTables = 72 + 40 + 20 + 12;
size_t tailSmemBytes(int cams) { return sizeof(TailSmem) + (size_t)cams * kTailPx * 6; }

// Level k of the tail in a plane of kTailPx pixels: its row pitch is the least
// power of two that fits any such level, its place what lies before it.
struct TailLevel {
    int shift, rows, off;
};
__device__ __forceinline__ TailLevel tailLevel(int k)
{
    if (k < 5) return {5 - k, max(1, kTailH >> k), (2048 - (2048 >> 2 * k)) / 3};
    return {0, 1, 682 + k - 5};
}
// Pixel i of a plane; false where no level has it.
__device__ __forceinline__ bool tailPixel(const RigDev& R, int i, int& j, int& x, int& y)
{
    const int k = i < 512 ? 0 : (i < 640 ? 1 : (i < 672 ? 2 : (i < 680 ? 3 : (i < 682 ? 4 : i - 677))));
    const TailLevel t = tailLevel(k);
    j = R.tailStart + k;
    x = (i - t.off) & ((1 << t.shift) - 1);
    y = (i - t.off) >> t.shift;
    return j <= R.L && x < R.lv[j].w && y < R.lv[j].h;
}

// The alpha divisors or the weights of a camera, a value at a time through f(pixel, value).
template <class F>
__device__ __forceinline__ void tailConstants(const RigDev& R, bool weights, int cam, F f)
{
    uint16_t v[2];
    bool ok[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int i = threadIdx.x + q * kTailThreads;
        int j, x, y;
        ok[q] = i < kTailPx && tailPixel(R, i, j, x, y);
        if (!ok[q]) continue;
        const LevelDev& lv = R.lv[j];
        const uint16_t* base = weights ? lv.Wt : lv.Am;
        v[q] = ldChecked(base + cam * lv.camStride + (size_t)y * lv.pitch + x, base, wBytes(R, lv));
    }
#pragma unroll
    for (int q = 0; q < 2; q++)
        if (ok[q]) f((int)threadIdx.x + q * kTailThreads, v[q]);
}

// A camera through its pyrDown levels; to: its levels in the last CTA.
__device__ __forceinline__ void tailDown(TailSmem& S, int cam, uint32_t to)
{
    const RigDev& R = S.rig;
    const uint32_t* src = &S.in[0][0];
    int pitch = 2 * kTailW;
    for (int j = R.tailStart; j <= R.L; j++) {
        __syncthreads();
        const TailLevel t = tailLevel(j - R.tailStart);
        const LevelDev& Ld = R.lv[j];
        const int p = threadIdx.x, X = p & ((1 << t.shift) - 1), Y = p >> t.shift;
        if (p < t.rows << t.shift && X < Ld.w && Y < Ld.h) {
            uint32_t v = 0;
            if (R.tailCams[j] >> cam & 1) {
                const uint8_t *cols = &S.downCol[j][2 * X], *rows = &S.downRow[j][2 * Y];
                int col[5];
                uint32_t lo[5], hi[5];
#pragma unroll
                for (int i = 0; i < 5; i++) col[i] = cols[i];
#pragma unroll
                for (int r = 0; r < 5; r++) {
                    const uint32_t* row = src + rows[r] * pitch;
                    uint2 u[5];
#pragma unroll
                    for (int i = 0; i < 5; i++) u[i] = unpackBytes(row[col[i]]);
                    lo[r] = k5(u[0].x, u[1].x, u[2].x, u[3].x, u[4].x);
                    hi[r] = k5(u[0].y, u[1].y, u[2].y, u[3].y, u[4].y);
                }
                v = downDivide(k5(lo[0], lo[1], lo[2], lo[3], lo[4]), k5(hi[0], hi[1], hi[2], hi[3], hi[4]),
                               S.am[t.off + p], S.magic);
                uint32_t* d = reinterpret_cast<uint32_t*>(Ld.G) + cam * Ld.camStride + (size_t)Y * Ld.pitch + X;
                if (inside(d, Ld.G, gBytes(R, Ld))) *d = v;
            }
            S.plane[t.off + p] = v;
            clusterStore(to + 4 * (t.off + p), v);
        }
        src = S.plane + t.off;
        pitch = 1 << t.shift;
    }
}

// Blend levels L .. tailStart from the shared memory of this CTA: the cameras'
// levels g and weights w.  A level of few pixels has its cameras spread over
// lanes of a pixel.
__device__ __forceinline__ void tailBlend(TailSmem& S, const uint32_t* g, const uint16_t* w)
{
    const RigDev& R = S.rig;
    const int most = R.n <= 1 ? 1 : 1 << (32 - __clz(R.n - 1));  // lanes with a camera of their own
    for (int j = R.L; j >= R.tailStart; j--) {
        const TailLevel t = tailLevel(j - R.tailStart), tu = tailLevel(j - R.tailStart + 1);
        const LevelDev& Lj = R.lv[j];
        const bool hasUp = j < R.L;
        const int slots = t.rows << t.shift;
        const int lanes = min(most, kTailThreads / slots);
        const int p = threadIdx.x / lanes, sub = threadIdx.x & (lanes - 1);
        if (((int)threadIdx.x & ~31) < slots * lanes) {  // whole warps
            const int x = p & ((1 << t.shift) - 1), y = p >> t.shift;
            const bool in = p < slots && x < Lj.w && y < Lj.h;
            int at[3][3], wt[3][3];
            if (in && hasUp) {
                const int wx[3] = {x & 1 ? 0 : 1, x & 1 ? 4 : 6, x & 1 ? 4 : 1};
                const int wy[3] = {y & 1 ? 0 : 1, y & 1 ? 4 : 6, y & 1 ? 4 : 1};
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    const int row = tu.off + (S.upRow[j][(y >> 1) + r] << tu.shift);
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        at[r][i] = row + S.upCol[j][(x >> 1) + i];
                        wt[r][i] = wy[r] * wx[i];
                    }
                }
            }
            int acc[4] = {0, 0, 0, 0};  // weighted B, G, R and the weights
            for (int cam = sub; in && cam < R.n; cam += lanes) {
                const int wq = w[cam * kTailPx + t.off + p];
                if (!wq) continue;
                const uint32_t* gc = g + cam * kTailPx;
                uint32_t lo = 0, hi = 0;
                if (hasUp) {
#pragma unroll
                    for (int r = 0; r < 3; r++)
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            const uint2 u = unpackBytes(gc[at[r][i]]);
                            lo += wt[r][i] * u.x;
                            hi += wt[r][i] * u.y;
                        }
                }
                const Lap l = laplacian(gc[t.off + p], lo, hi);
                acc[0] += wq * ((int)(l.br & 0xFFFFu) - 256);
                acc[1] += wq * l.g;
                acc[2] += wq * ((int)(l.br >> 16) - 256);
                acc[3] += wq;
            }
            for (int o = lanes / 2; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
            if (in && !sub) {
                int n[3];
                const int d = acc[3] ? acc[3] : 1;
                const float rcp = __frcp_rn((float)d);
#pragma unroll
                for (int c = 0; c < 3; c++) n[c] = R.full ? (acc[c] + 128) >> 8 : divTrunc(acc[c], d, rcp);
                if (hasUp) {
                    int v[3] = {32, 32, 32};
#pragma unroll
                    for (int r = 0; r < 3; r++)
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            const uint2 q = S.c[at[r][i]];
                            v[0] += wt[r][i] * (short)q.x;
                            v[1] += wt[r][i] * (short)q.y;
                            v[2] += wt[r][i] * ((int)q.x >> 16);
                        }
#pragma unroll
                    for (int c = 0; c < 3; c++) n[c] += (v[c] >> 6) - kCBias;
                }
                const uint2 out = packC(n[0], n[1], n[2]);
                S.c[t.off + p] = out;
                uint2* q = reinterpret_cast<uint2*>(Lj.C) + (size_t)y * Lj.pitch + x;
                if (inside(q, Lj.C, cBytes(Lj))) *q = out;
            }
        }
        __syncthreads();
    }
}

// cluster CTAs a segment; cams: the most cameras of any
__global__ void __launch_bounds__(kTailThreads) k_tail(const Segment* __restrict__ segs, int cluster, int cams)
{
    extern __shared__ __align__(128) uint8_t tailSmem[];
    TailSmem& S = *reinterpret_cast<TailSmem*>(tailSmem);
    uint32_t* g = reinterpret_cast<uint32_t*>(tailSmem + sizeof(TailSmem));
    uint16_t* w = reinterpret_cast<uint16_t*>(g + cams * kTailPx);
    const int rank = blockIdx.x % cluster, last = cluster - 1;
    clusterArrive();  // every CTA has started before any writes another's shared memory
    const uint32_t* desc = reinterpret_cast<const uint32_t*>(segs[blockIdx.x / cluster].rig);
    for (int k = threadIdx.x; k < (int)sizeof(RigDev) / 4; k += kTailThreads)
        reinterpret_cast<uint32_t*>(&S.rig)[k] = __ldg(desc + k);
    initMagic(S.magic);
    __syncthreads();
    const RigDev& R = S.rig;
    const int T = R.tailStart;
    if (rank < R.n) tailConstants(R, false, rank, [&](int i, uint16_t v) { S.am[i] = v; });
    for (int k = threadIdx.x; k < (R.L - T + 1) * kTailTables; k += kTailThreads) {
        const int j = T + k / kTailTables, e = k % kTailTables;
        const LevelDev &Ls = R.lv[j - 1], &Ld = R.lv[j], &Lu = R.lv[min(j + 1, R.L)];
        if (e < 72) {
            if (e < 2 * Ld.w + 3) S.downCol[j][e] = (uint8_t)colMap(e - 2, Ls.w);
        } else if (e < 112) {
            if (e - 72 < 2 * Ld.h + 3) S.downRow[j][e - 72] = (uint8_t)rowMap(e - 74, Ls.h);
        } else if (e < 132) {
            if (e - 112 < Ld.w / 2 + 3) S.upCol[j][e - 112] = (uint8_t)colMap(e - 113, Lu.w);
        } else if (e - 132 < Ld.h / 2 + 3) {
            S.upRow[j][e - 132] = (uint8_t)rowMap(e - 133, Lu.h);
        }
    }
    clusterWait();
    for (int cam = rank; cam < R.n; cam += cluster) {
        const uint32_t to = clusterAddr(w + cam * kTailPx, last);
        tailConstants(R, true, cam, [&](int i, uint16_t v) { clusterStore(to + 2 * i, v); });
    }
    waitPrevGrid();
    allowNextGrid();
    const LevelDev& Li = R.lv[T - 1];
    for (int cam = rank; cam < R.n; cam += cluster) {
        if (cam != rank) {
            __syncthreads();  // readers of the camera before are done
            tailConstants(R, false, cam, [&](int i, uint16_t v) { S.am[i] = v; });
        }
        // at most 64x32; its rows are 64 pixels at least
        const int x = threadIdx.x % (kTailW / 2) * 4, y = threadIdx.x / (kTailW / 2);
        if (y < Li.h) {
            const uint4* p = reinterpret_cast<const uint4*>(Li.G + cam * Li.camStride + (size_t)y * Li.pitch + x);
            *reinterpret_cast<uint4*>(&S.in[y][x]) = inside(p, Li.G, gBytes(R, Li)) ? __ldg(p) : make_uint4(0, 0, 0, 0);
        }
        tailDown(S, cam, clusterAddr(g + cam * kTailPx, last));
    }
    clusterArrive();
    clusterWait();
    if (rank == last) tailBlend(S, g, w);
}

// ============================================================================
// k_blend_small: blend levels above 0 with few tiles, below the tail, on a
// plain grid: one 64x8 half tile per work
// item (items 2t and 2t + 1 are the halves of tile t), up to eight cameras
// staged per unit.  In k_blend a CTA walks a tile's cameras two at a time,
// a chain of load-and-compute rounds that these levels cannot hide behind
// other tiles; here each CTA has one short chain and all its warps busy.
// ============================================================================
__global__ void __launch_bounds__(kThreads, 4) k_blend_small(const Segment* __restrict__ segs, int nsegs, int total,
                                                          int early)
{
    __shared__ HalfStage st;

    // Items, descriptors and weights are written before the launch sequence,
    // not by a kernel: the first item's are fetched while the previous kernel
    // finishes.  So are its G_j rows where that kernel is the tail (kEarlyG: the
    // level was complete before the tail began) and its G_{j+1} footprints where
    // it wrote only C levels (kEarlyUp: every blend step after the first); only
    // the C_{j+1} footprint waits.  A launch that begins with the one before it
    // (kEarlyBegin) has the time to normalise its first item ahead of the wait
    // too.  It may: all G levels were complete before the first blend step let
    // its successor begin.
    const int pre = kPartW | (early & kEarlyG ? kPartG : 0) | (early & kEarlyUp ? kPartUp : 0);
    const bool begun = (early & kEarlyBegin) != 0;
    if (early & kEarlyNext) allowNextGrid();
    bool waited = false;
    auto wait = [&] {
        waitPrevGrid();
        if (!(early & kEarlyNext)) allowNextGrid();
        waited = true;
    };
    int s = 0, filled = -1;
    UnitGeo geo;
    PairAcc acc;
    for (int it = blockIdx.x; it < total; it += gridDim.x) {
        s = findSegment(segs, nsegs, it, s);
        const Segment& sg = segs[s];
        const RigDev& R = *sg.rig;
        const uint4 raw = __ldg(static_cast<const uint4*>(sg.items) + ((it - sg.prefix) >> 1));
        if (s != filled) fillGeo(geo, R, *sg.frame, raw.x & 0xFF);
        filled = s;
        const int half = (it - sg.prefix) & 1;
        const size_t up = halfCOffset(R, raw, half);
        const int chunks = unitChunks<HalfStage::kCams>(raw);
        bool staged = false;  // the C_{j+1} footprint
        for (int chunk = 0; chunk < chunks; chunk++) {
            __syncthreads();  // readers of the previous unit are done
            int parts = kPartsAll;
            if (!waited && !begun) {
                stageHalfG(st, R, raw, chunk, half, pre);
                wait();
                parts &= ~pre;
            }
            if (parts) stageHalfG(st, R, raw, chunk, half, parts);
            if (waited && chunk == chunks - 1) {
                stageHalfC(st, R, raw.x & 0xFF, up);
                staged = true;
            }
            __syncthreads();
            accumulateRows(st, geo, raw, chunk, acc);
        }
        int n0[3], n1[3];
        normaliseRows(geo, acc, n0, n1);
        if (!staged) {
            wait();
            stageHalfC(st, R, raw.x & 0xFF, up);
            __syncthreads();
        }
        const int x = (int)(raw.y & 0xFFFF) * kBlendTW + (threadIdx.x & 31) * 2;
        const int y = (int)(raw.y >> 16) * kBlendTH + kHalfRows * half + (threadIdx.x >> 5);
        if (y < geo.h) collapseRows(st, geo, x, y, n0, n1);
    }
    if (!waited) wait();
}

// ============================================================================
// k_cvt_yuv: standalone BGR32 -> YUV420P / NV12 of a device image
// (cvtBGR32ToYUV420P / cvtBGR32ToNV12, ImageProc.cu:97-160).  Where the image
// and its planes allow 16- and 8-byte accesses (cvtVector), a thread converts
// eight pixels of a row pair: four 16-byte loads, 8-byte luma stores, the four
// blocks' chroma in one store (YUV420P: two of 4 bytes).  Otherwise one thread
// per 2x2 block, byte by byte.  4096x2048 NV12: 14.4 us before (byte stores
// for every image), 10.7 us now.
// ============================================================================
__device__ __forceinline__ uint32_t packBytes(uint32_t lo, uint32_t hi) { return lo | (hi << 16); }

__global__ void __launch_bounds__(kYuvThreads) k_cvt_yuv8(const uint8_t* __restrict__ src, long long srcPitch, int w,
                                                          int h, int fmt, uint8_t* __restrict__ py, long long yPitch,
                                                          uint8_t* __restrict__ pu, long long uPitch,
                                                          uint8_t* __restrict__ pv, long long vPitch)
{
    const int x = 8 * (blockIdx.x * kYuvThreads + threadIdx.x);
    if (x >= w) return;
    for (int by = blockIdx.y; by < h / 2; by += gridDim.y) {
        uint4 q[2][2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint4* p = reinterpret_cast<const uint4*>(src + (size_t)(2 * by + r) * srcPitch) + x / 4;
            q[r][0] = __ldg(p);
            q[r][1] = __ldg(p + 1);
        }
        uint32_t us = 0, vs = 0;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint32_t* o = &q[r][0].x;
            uint32_t y4[4];
#pragma unroll
            for (int k = 0; k < 4; k++) y4[k] = packSat2(yuvLumaRaw(o[2 * k]), yuvLumaRaw(o[2 * k + 1]));
            *reinterpret_cast<uint2*>(py + (size_t)(2 * by + r) * yPitch + x) =
                make_uint2(packBytes(y4[0], y4[1]), packBytes(y4[2], y4[3]));
        }
        uint32_t uv[4];  // U | V << 8 of the four blocks, from their left columns
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int2 c = yuvChromaSums((&q[0][0].x)[2 * k]), d = yuvChromaSums((&q[1][0].x)[2 * k]);
            uv[k] = packSat2((c.x + d.x) >> (kYuvShift + 1), (c.y + d.y) >> (kYuvShift + 1));
        }
        if (fmt == PS_FMT_NV12) {
            *reinterpret_cast<uint2*>(pu + (size_t)by * uPitch + x) =
                make_uint2(packBytes(uv[0], uv[1]), packBytes(uv[2], uv[3]));
        } else {
            us = __byte_perm(packBytes(uv[0], uv[1]), packBytes(uv[2], uv[3]), 0x6420);
            vs = __byte_perm(packBytes(uv[0], uv[1]), packBytes(uv[2], uv[3]), 0x7531);
            *reinterpret_cast<uint32_t*>(pu + (size_t)by * uPitch + x / 2) = us;
            *reinterpret_cast<uint32_t*>(pv + (size_t)by * vPitch + x / 2) = vs;
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_cvt_yuv(const uint8_t* __restrict__ src, long long srcPitch, int w,
                                                      int h, int fmt, uint8_t* __restrict__ py, long long yPitch,
                                                      uint8_t* __restrict__ pu, long long uPitch,
                                                      uint8_t* __restrict__ pv, long long vPitch)
{
    const int bw = w >> 1, bh = h >> 1;
    const long long total = (long long)bw * bh;
    for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < total;
         b += (long long)gridDim.x * blockDim.x) {
        const int by = (int)(b / bw), bx = (int)(b - (long long)by * bw);
        const int x = bx * 2, y = by * 2;
        const uint32_t* r0 = reinterpret_cast<const uint32_t*>(src + (size_t)y * srcPitch) + x;
        const uint32_t* r1 = reinterpret_cast<const uint32_t*>(src + (size_t)(y + 1) * srcPitch) + x;
        const uint32_t p00 = r0[0], p01 = r0[1], p10 = r1[0], p11 = r1[1];
        uint8_t* y0 = py + (size_t)y * yPitch + x;
        uint8_t* y1 = y0 + yPitch;
        y0[0] = (uint8_t)yuvLuma(p00);
        y0[1] = (uint8_t)yuvLuma(p01);
        y1[0] = (uint8_t)yuvLuma(p10);
        y1[1] = (uint8_t)yuvLuma(p11);
        const int2 c0 = yuvChromaSums(p00), c1 = yuvChromaSums(p10);
        const uint8_t u = (uint8_t)clamp255((c0.x + c1.x) >> (kYuvShift + 1));
        const uint8_t v = (uint8_t)clamp255((c0.y + c1.y) >> (kYuvShift + 1));
        if (fmt == PS_FMT_NV12) {
            pu[(size_t)by * uPitch + x] = u;
            pu[(size_t)by * uPitch + x + 1] = v;
        } else {
            pu[(size_t)by * uPitch + bx] = u;
            pv[(size_t)by * vPitch + bx] = v;
        }
    }
}

// ============================================================================
// k_yuv_to_bgr32: decoder frames YUV420P / NV12 -> BGR32 (cvtYUV420PToBGR32
// / cvtNV12ToBGR32, ImageProc.cu:165-259): per 2x2 block, with u = U - 128,
// v = V - 128 and y' = max(Y - 16, 0) * CY,
//   R = clamp((y' + 2^19 + CVR v) >> 20), G = clamp((y' + 2^19 + CVG v + CUG u) >> 20),
//   B = clamp((y' + 2^19 + CUB u) >> 20)
// (the standard BT.601 studio-range coefficients scaled by 2^20; the shift
// of a negative sum rounds toward minus infinity).  The fourth byte is
// written 0.  One thread per 2x2 block; blockIdx.y is the frame.
// ============================================================================
constexpr int kInvCY = 1220542, kInvCUB = 2116026, kInvCUG = -409993, kInvCVG = -852492, kInvCVR = 1673527;

__device__ __forceinline__ uint32_t yuvPixel(int yv, int ruv, int guv, int buv)
{
    const int yy = max(yv - 16, 0) * kInvCY;
    return packSatBgr((yy + buv) >> kYuvShift, (yy + guv) >> kYuvShift, (yy + ruv) >> kYuvShift);
}

// Eight pixels of a row pair (four 2x2 blocks) per thread: 8-byte luma
// loads, the blocks' chroma in one load, 16-byte stores.

struct YuvChunk {
    uint2 yt, yb;     // luma of the top and bottom rows
    uint32_t us, vs;  // the four blocks' U and V, one byte each
};

__device__ __forceinline__ YuvChunk yuvLoad(const YuvFrame& F, int cx, int by)
{
    const int x = 8 * cx, y = 2 * by;
    YuvChunk c;
    c.yt = *reinterpret_cast<const uint2*>(F.y + (size_t)y * F.yPitch + x);
    c.yb = *reinterpret_cast<const uint2*>(F.y + (size_t)(y + 1) * F.yPitch + x);
    if (F.fmt == PS_FMT_NV12) {
        const uint2 uv = *reinterpret_cast<const uint2*>(F.u + (size_t)by * F.uPitch + x);
        c.us = __byte_perm(uv.x, uv.y, 0x6420);
        c.vs = __byte_perm(uv.x, uv.y, 0x7531);
    } else {
        c.us = *reinterpret_cast<const uint32_t*>(F.u + (size_t)by * F.uPitch + (x >> 1));
        c.vs = *reinterpret_cast<const uint32_t*>(F.v + (size_t)by * F.vPitch + (x >> 1));
    }
    return c;
}

__device__ __forceinline__ void yuvStore(const YuvFrame& F, int cx, int by, const YuvChunk& c)
{
    const int half = 1 << (kYuvShift - 1);
    uint32_t ot[8], ob[8];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int u = (int)((c.us >> (8 * k)) & 0xFF) - 128, v = (int)((c.vs >> (8 * k)) & 0xFF) - 128;
        const int ruv = half + kInvCVR * v, guv = half + kInvCVG * v + kInvCUG * u, buv = half + kInvCUB * u;
        const uint32_t wt = k < 2 ? c.yt.x : c.yt.y, wb = k < 2 ? c.yb.x : c.yb.y;
        const int s = 16 * (k & 1);
        ot[2 * k] = yuvPixel((wt >> s) & 0xFF, ruv, guv, buv);
        ot[2 * k + 1] = yuvPixel((wt >> (s + 8)) & 0xFF, ruv, guv, buv);
        ob[2 * k] = yuvPixel((wb >> s) & 0xFF, ruv, guv, buv);
        ob[2 * k + 1] = yuvPixel((wb >> (s + 8)) & 0xFF, ruv, guv, buv);
    }
    const int y = 2 * by;
    uint4* t = reinterpret_cast<uint4*>(F.dst + (size_t)y * F.dstPitch) + 2 * cx;
    uint4* b = reinterpret_cast<uint4*>(F.dst + (size_t)(y + 1) * F.dstPitch) + 2 * cx;
    t[0] = make_uint4(ot[0], ot[1], ot[2], ot[3]);
    t[1] = make_uint4(ot[4], ot[5], ot[6], ot[7]);
    b[0] = make_uint4(ob[0], ob[1], ob[2], ob[3]);
    b[1] = make_uint4(ob[4], ob[5], ob[6], ob[7]);
}

// The frames the vector path takes (all of them, or none): a thread has one
// chunk of eight pixels by two rows, blockIdx.y being the row pair and blockIdx.z
// the frame, so that no index needs a division and every load is in flight at
// once; two or four chunks a thread measured slower.  4096x2048 NV12: 13.8 us
// before (a grid of one wave), 12.7 us now; 6 x 1920x1080 22.3 and 19.1 us.
__global__ void __launch_bounds__(kYuvThreads, 8) k_yuv_to_bgr32_8(YuvFrames f)
{
    const int cx = blockIdx.x * kYuvThreads + threadIdx.x;
    if (8 * cx >= f.w) return;
    const YuvFrame& F = f.frame[blockIdx.z];
    for (int by = blockIdx.y; by < f.h >> 1; by += gridDim.y) yuvStore(F, cx, by, yuvLoad(F, cx, by));
}

__global__ void __launch_bounds__(kThreads) k_yuv_to_bgr32(YuvFrames f)
{
    const int cam = blockIdx.y;
    const int bw = f.w >> 1, bh = f.h >> 1;
    const YuvFrame& F = f.frame[cam];
    // the launcher takes frames below 2^32 pixels, so 32-bit indices cover the work
    const unsigned total = (unsigned)bw * (unsigned)bh;
    for (unsigned b = blockIdx.x * blockDim.x + threadIdx.x; b < total; b += gridDim.x * blockDim.x) {
        const int by = (int)(b / (unsigned)bw), bx = (int)(b - (unsigned)by * (unsigned)bw);
        const int x = 2 * bx, y = 2 * by;
        const uint8_t* y0 = F.y + (size_t)y * F.yPitch + x;
        const uint8_t* y1 = y0 + F.yPitch;
        int u, v;
        if (F.fmt == PS_FMT_NV12) {
            const uint8_t* c = F.u + (size_t)by * F.uPitch + x;
            u = c[0];
            v = c[1];
        } else {
            u = F.u[(size_t)by * F.uPitch + bx];
            v = F.v[(size_t)by * F.vPitch + bx];
        }
        u -= 128;
        v -= 128;
        const int half = 1 << (kYuvShift - 1);
        const int ruv = half + kInvCVR * v, guv = half + kInvCVG * v + kInvCUG * u, buv = half + kInvCUB * u;
        uint32_t* o0 = reinterpret_cast<uint32_t*>(F.dst + (size_t)y * F.dstPitch) + x;
        uint32_t* o1 = reinterpret_cast<uint32_t*>(F.dst + (size_t)(y + 1) * F.dstPitch) + x;
        const uint32_t p00 = yuvPixel(y0[0], ruv, guv, buv), p01 = yuvPixel(y0[1], ruv, guv, buv);
        const uint32_t p10 = yuvPixel(y1[0], ruv, guv, buv), p11 = yuvPixel(y1[1], ruv, guv, buv);
        if (((reinterpret_cast<uintptr_t>(o0) | reinterpret_cast<uintptr_t>(o1)) & 7) == 0) {  // images are 4-byte aligned
            *reinterpret_cast<uint2*>(o0) = make_uint2(p00, p01);
            *reinterpret_cast<uint2*>(o1) = make_uint2(p10, p11);
        } else {
            o0[0] = p00;
            o0[1] = p01;
            o1[0] = p10;
            o1[1] = p11;
        }
    }
}

// ---- launch helpers ---------------------------------------------------------
// The lazily computed launch facts below are function-local statics, so
// their first computation is thread-safe (renders may launch from several
// threads).
static int smCount()
{
    static const int sms = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 1;
    }();
    return sms;
}

// One wave of `perSm` CTAs per SM, capped by `want` (> 0) and by the work.
static int gridFor(int total, int perSm, int want = 0)
{
    if (want > 0 && want < perSm) perSm = want;
    const int cap = smCount() * perSm;
    return total < cap ? total : cap;
}

// CTAs of `kernel` that fit on one SM (registers, shared memory, threads),
// so a grid of residentPerSm * SMs runs in a single wave; cached per kernel.
template <auto Kernel>
static int residentPerSm(int threads, size_t dynSmem = 0)
{
    static const int cached = [threads, dynSmem] {  // one per kernel
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, Kernel, threads, dynSmem) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = 1;
        }
        return n;
    }();
    return cached;
}

// Every per-frame kernel is launched with programmatic stream serialisation,
// so its prologue overlaps the previous kernel's tail (see waitPrevGrid).
template <class... Args>
static cudaError_t launchPdl(void (*kernel)(Args...), int grid, int block, cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

int residentCtasPerSm(int kind)
{
    switch (kind) {
    case 0:
        return std::min({residentPerSm<k_remap<0, true>>(kRemapThreads), residentPerSm<k_remap<PS_FMT_BGR24, true>>(kRemapThreads),
                         residentPerSm<k_remap<PS_FMT_BGR32, true>>(kRemapThreads)});
    case 1: return residentPerSm<k_pyrdown>(kDownThreads);
    case 2: return residentPerSm<k_blend>(kBlendThreads);
    default: return 1;
    }
}

int remapSourceFormat(int fmt, int sw, int sh, long long pitch)
{
    constexpr int kMost = 1 << 22;
    return sw >= 2 && sh >= 2 && sw <= kMost && sh <= kMost && pitch >= 0 && pitch < (1LL << 32) ? fmt : 0;
}

template <int kFmt, bool kMaps>
static cudaError_t launchRemapAs(const Segment* segs, int nsegs, int total, int perSm, int* counter, int probePolls,
                                 cudaStream_t st)
{
    return launchPdl(k_remap<kFmt, kMaps>, gridFor(total, residentPerSm<k_remap<kFmt, kMaps>>(kRemapThreads), perSm),
                     kRemapThreads, st, segs, nsegs, total, counter, probePolls);
}

cudaError_t launchRemap(const Segment* segs, int nsegs, int total, int perSm, int* counter, int probePolls, int srcFmt,
                        bool maps, cudaStream_t st)
{
    if (total <= 0) return cudaSuccess;
    if (!maps) return launchRemapAs<0, false>(segs, nsegs, total, perSm, counter, probePolls, st);
    switch (srcFmt) {
    case PS_FMT_BGR32: return launchRemapAs<PS_FMT_BGR32, true>(segs, nsegs, total, perSm, counter, probePolls, st);
    case PS_FMT_BGR24: return launchRemapAs<PS_FMT_BGR24, true>(segs, nsegs, total, perSm, counter, probePolls, st);
    default: return launchRemapAs<0, true>(segs, nsegs, total, perSm, counter, probePolls, st);
    }
}

cudaError_t launchPyrDown(const Segment* segs, int nsegs, int total, int perSm, cudaStream_t st)
{
    if (total <= 0) return cudaSuccess;
    return launchPdl(k_pyrdown, gridFor(total, residentPerSm<k_pyrdown>(kDownThreads), perSm), kDownThreads, st, segs, nsegs,
                     total);
}

cudaError_t launchPyrDownPair(const Segment* segs, int nsegs, int total, cudaStream_t st)
{
    if (total <= 0) return cudaSuccess;
    return launchPdl(k_pyrdown_pair, gridFor(total, residentPerSm<k_pyrdown_pair>(kPairThreads)), kPairThreads, st, segs,
                     nsegs, total);
}

template <int kFmt>
static cudaError_t launchLinearAs(const Segment* segs, int nsegs, int total, int maxCams, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gridFor(total, residentPerSm<k_linear<kFmt>>(kLinearThreads, (size_t)PS_MAX_CAMS * 768)));
    cfg.blockDim = dim3(kLinearThreads);
    cfg.dynamicSmemBytes = (size_t)maxCams * 768;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_linear<kFmt>, segs, nsegs, total);
}

cudaError_t launchLinear(const Segment* segs, int nsegs, int total, int maxCams, int srcFmt, cudaStream_t st)
{
    if (total <= 0) return cudaSuccess;
    switch (srcFmt) {
    case PS_FMT_BGR32: return launchLinearAs<PS_FMT_BGR32>(segs, nsegs, total, maxCams, st);
    case PS_FMT_BGR24: return launchLinearAs<PS_FMT_BGR24>(segs, nsegs, total, maxCams, st);
    default: return launchLinearAs<0>(segs, nsegs, total, maxCams, st);
    }
}

cudaError_t launchBlend(const Segment* segs, int nsegs, int total, int work, int perSm, int* counter, int probePolls,
                        int early, cudaStream_t st)
{
    if (total <= 0) return cudaSuccess;
    if (work <= kRowsWork) {
        // a row pair a warp, two where the warps would take more than one
        const bool two = total * (kBlendTH / 4) >= smCount() * kRowsCtas * (kThreads / 32);
        const int ctas = (total * (kBlendTH / (two ? 4 : 2)) + kThreads / 32 - 1) / (kThreads / 32);
        auto* kernel = two ? k_blend_rows<2> : k_blend_rows<1>;
        return launchPdl(kernel, gridFor(ctas, kRowsCtas, perSm), kThreads, st, segs, nsegs, total, probePolls);
    }
    return launchPdl(k_blend, gridFor(total, residentPerSm<k_blend>(kBlendThreads), perSm), kBlendThreads, st, segs,
                     nsegs, total, counter, probePolls, (int)((early & kEarlyUp) != 0));
}

cudaError_t launchBlendSmall(const Segment* segs, int nsegs, int total, int early, cudaStream_t st)
{
    if (total <= 0) return cudaSuccess;
    return launchPdl(k_blend_small, gridFor(total, residentPerSm<k_blend_small>(kThreads)), kThreads, st, segs, nsegs,
                     total, early);
}

int tailClusterMax()
{
    static const int widest = [] {  // the attributes are set before any launch can see the width
        int size = kTailCluster;
        const int smem = (int)tailSmemBytes(kTailCams);
        cudaFuncSetAttribute(k_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (cudaFuncSetAttribute(k_tail, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(kTailClusterWide);
            cfg.blockDim = dim3(kTailThreads);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = kTailClusterWide;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, k_tail, &cfg) == cudaSuccess && clusters >= 1)
                size = kTailClusterWide;
        }
        cudaGetLastError();
        return size;
    }();
    return widest;
}

cudaError_t launchTail(const Segment* segs, int nsegs, int cluster, int cams, cudaStream_t st)
{
    if (nsegs <= 0) return cudaSuccess;
    cluster = tailClusterWidth(cluster, cams, tailClusterMax());
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nsegs * cluster);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = tailSmemBytes(cams);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, k_tail, segs, cluster, cams);
}

// A plane whose rows all start on a multiple of `to` bytes.
static bool aligned(const void* p, long long pitch, int to)
{
    return reinterpret_cast<uintptr_t>(p) % to == 0 && pitch % to == 0;
}

cudaError_t launchCvtYuv(const uint8_t* src, long long srcPitch, int w, int h, int fmt, uint8_t* y, long long yPitch,
                         uint8_t* u, long long uPitch, uint8_t* v, long long vPitch, cudaStream_t st)
{
    const long long blocks = (long long)(w / 2) * (h / 2);
    if (blocks <= 0) return cudaSuccess;
    const bool nv12 = fmt == PS_FMT_NV12;
    if (w % 8 == 0 && aligned(src, srcPitch, 16) && aligned(y, yPitch, 8) && aligned(u, uPitch, nv12 ? 8 : 4) &&
        (nv12 || aligned(v, vPitch, 4))) {
        const dim3 grid8((w / 8 + kYuvThreads - 1) / kYuvThreads, std::min(h / 2, 65535));
        k_cvt_yuv8<<<grid8, kYuvThreads, 0, st>>>(src, srcPitch, w, h, fmt, y, yPitch, u, uPitch, v, vPitch);
        return cudaGetLastError();
    }
    const int grid = (int)std::min<long long>((blocks + kThreads - 1) / kThreads, (long long)smCount() * 8);
    k_cvt_yuv<<<grid, kThreads, 0, st>>>(src, srcPitch, w, h, fmt, y, yPitch, u, uPitch, v, vPitch);
    return cudaGetLastError();
}

// Frames whose width and planes allow the 8-pixel path.
static bool yuvVector(const YuvFrame& F, int w)
{
    if (w % 8 || !aligned(F.y, F.yPitch, 8) || !aligned(F.dst, F.dstPitch, 16)) return false;
    if (F.fmt == PS_FMT_NV12) return aligned(F.u, F.uPitch, 8);
    return aligned(F.u, F.uPitch, 4) && aligned(F.v, F.vPitch, 4);
}

cudaError_t launchYuvToBgr32(const YuvFrames& frames, cudaStream_t st)
{
    const YuvFrames& f = frames;
    if (f.n <= 0 || f.w <= 0 || f.h <= 0) return cudaSuccess;
    if ((long long)f.w * f.h >= (1LL << 32)) return cudaErrorInvalidValue;
    // All frames one way: with one, three or six of six 1920x1080 NV12 frames
    // unaligned the per-block kernel takes 22.2, 21.9 and 21.8 us for all, a
    // launch for either kind of frame 24, 25.4 and 21.4 us.
    bool vec = true;
    for (int i = 0; i < f.n; i++) vec = vec && yuvVector(f.frame[i], f.w);
    if (vec) {
        const dim3 grid((f.w / 8 + kYuvThreads - 1) / kYuvThreads, std::min(f.h / 2, 65535), f.n);
        k_yuv_to_bgr32_8<<<grid, kYuvThreads, 0, st>>>(f);
        return cudaGetLastError();
    }
    // one wave of 8 CTAs per SM across all frames, or fewer CTAs if the work is smaller
    const long long items = (long long)(f.w / 2) * (f.h / 2);
    const long long want = std::max<long long>(1, (long long)smCount() * 8 / f.n);
    const int gx = (int)std::min<long long>((items + kThreads - 1) / kThreads, want);
    k_yuv_to_bgr32<<<dim3(gx, f.n), kThreads, 0, st>>>(f);
    return cudaGetLastError();
}

cudaError_t launchReprojectTo16S(const uint8_t* src, long long srcPitch, int srcW, int srcH, int srcFmt,
                                 const float* xmap, const float* ymap, long long mapPitch, int dstW, int dstH,
                                 const uint8_t* lut, int16_t* dst, long long dstPitch, cudaStream_t st)
{
    dim3 grid((dstW + 16 * kReprojectBlocks - 1) / (16 * kReprojectBlocks), (dstH + 15) / 16);
    const RemapSrc S{src, srcPitch, srcFmt, srcW, srcH};
    short4* const d = reinterpret_cast<short4*>(dst);
    auto go = [&](auto* few, auto* many) {
        // kReprojectMany CTAs and more: five a SM, at 48 registers and a few
        // spills, where the others hide each other's trips to memory
        auto* kernel = grid.x * grid.y >= kReprojectMany ? many : few;
        kernel<<<grid, kThreads, 0, st>>>(S, xmap, ymap, mapPitch, dstW, dstH, lut, d, dstPitch);
    };
    switch (remapSourceFormat(srcFmt, srcW, srcH, srcPitch)) {
    case PS_FMT_BGR32: go(k_reproject16s<PS_FMT_BGR32, 1>, k_reproject16s<PS_FMT_BGR32, 5>); break;
    case PS_FMT_BGR24: go(k_reproject16s<PS_FMT_BGR24, 1>, k_reproject16s<PS_FMT_BGR24, 5>); break;
    default: go(k_reproject16s<0, 1>, k_reproject16s<0, 5>);
    }
    return cudaGetLastError();
}

}  // namespace ps

// ---- the checked build's counter ------------------------------------------------
namespace ps {
long long boundsViolations(bool reset)
{
#ifdef PS_CHECK_BOUNDS
    unsigned long long v = 0;
    if (cudaDeviceSynchronize() != cudaSuccess) return -2;  // the renders run on their own streams
    if (cudaMemcpyFromSymbol(&v, g_boundsViolations, sizeof v) != cudaSuccess) return -2;
    if (reset) {
        const unsigned long long z = 0;
        if (cudaMemcpyToSymbol(g_boundsViolations, &z, sizeof z) != cudaSuccess) return -2;
    }
    return (long long)v;
#else
    (void)reset;
    return -1;
#endif
}
}  // namespace ps
