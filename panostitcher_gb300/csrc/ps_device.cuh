// ps_device.cuh -- device-side data layout shared by the stitch kernels.
//
// HBM layout of one rig (all cameras share the level geometry):
//   G[j]   uchar4 Gaussian pyramid of every camera, level j, camera-major,
//          row pitch lv[j].pitch pixels.  The reference keeps it as int16x4
//          (CV_16SC4); every value is provably in 0..255 (the level-0 remap
//          is a convex combination of bytes and each masked pyrDown is a
//          weighted average of the level below), so one byte per channel is
//          exact and halves the traffic.
//   Wt[j]  uint16 seam-weight pyramid (weightPyrs, 0..256), same pitch as G.
//   Am[j]  uint16 alpha divisor m = alphaPyr / 256 (alphaPyrs is always a
//          multiple of 256 because its level source is 0/256), level >= 1.
//   C[j]   collapsed result of level j >= 1 (resultPyr after normalise +
//          collapse), four int16 a pixel: B, R, G, each + kCBias, and 0;
//          |value| < 8700, so int16 is exact.
//   maps   float2 dst->src map, stored tile-compact for the level-0 tiles
//          that a camera covers (512 pixels per 32x16 tile, in 16x2 blocks).
// Work is described by item lists built at prepare time from the pyramids'
// supports, so no kernel touches canvas area a camera cannot influence.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/panostitch.h"

namespace ps {

// ---- tiles ------------------------------------------------------------------
constexpr int kRemapTW = 32, kRemapTH = 16;    // level-0 remap tile (16x2 blocks, a pixel a lane)
constexpr int kDownTW = 32, kDownTH = 16;      // pyrDown output tile (four pixels per thread)
constexpr int kBlendTW = 64, kBlendTH = 16;    // blend tile (a 2x2 pixel block per thread)
constexpr int kThreads = 256;
// k_pyrdown_pair takes two levels whose lower one has this many tiles at most
// (a CTA an SM): 40% of a tile's work is done twice, which levels of 380 tiles
// do not hide (a launch of 5.7 - 6.3 us, as long as two of k_pyrdown; eight
// frames in flight 918 us instead of 872).
constexpr int kPairTiles = 152;
constexpr int kTailW = 32, kTailH = 16, kTailCams = 16;  // largest level and most cameras of k_tail
constexpr int kCBias = 256;  // of the collapsed levels' values

// Pixel i of a remap tile (its map, its linear weight): the tile is 16 blocks
// of 16x2 pixels, two across and eight down, a warp's 32 pixels each.  The
// frame's texels under a 16x2 block lie on fewer lines than under a 32x1 row,
// whose image in the frame is tilted.
__host__ __device__ constexpr int mapTileX(int i) { return (i >> 5 & 1) * 16 + (i & 15); }
__host__ __device__ constexpr int mapTileY(int i) { return (i >> 6) * 2 + (i >> 4 & 1); }

struct LevelDev {
    int w, h;            // level size
    int pitch;           // row pitch in pixels of G / Wt / Am / C (multiple of 64)
    long long camStride; // pixels between cameras in G / Wt / Am
    uchar4* G;
    uint16_t* Wt;
    uint16_t* Am;
    short4* C;
};

// Work items (one per tile), resident per rig and built at prepare time.
struct RemapItem { uint16_t cam, pad; uint16_t tx, ty; uint32_t mapTile; };

// level: the output's; whole: every alpha of the tile is 256 (m == 256)
struct DownItem { uint8_t cam, level; uint16_t tx, ty; uint16_t whole; };
// A blend tile lists the cameras whose weight touches it: up to 8 inline,
// more through RigDev::camLists (cams[0..3] then hold the uint32 offset).
struct alignas(16) BlendItem { uint8_t level, cls, camCnt, flags; uint16_t tx, ty; uint8_t cams[8]; };
constexpr int kInlineCams = 8;
// flags bit 0: one camera, weight 256 on every pixel of the tile, so the
// normalised value is the Laplacian itself (R = 256 L, W = 256); at level 0 the
// tile is fully covered too (cls 1).
constexpr int kTileUniform = 1;
// cls of a level-0 blend tile: 0 uncovered (write zeros), 1 fully covered,
// 2 partially covered (read the union mask).  Unused above level 0.
// Linear-blend mode: one item per 32x16 canvas tile, naming the run
// [first, first + count) of remap items (cameras in index order) covering it.
struct LinearItem { uint16_t tx, ty; uint32_t first, count; };

// Remap::remapImage's parameters in fp32, for the map-free remap (the
// reference's dstToSrc, source/CudaAccel/CudaReproject.cu:81-264, keeps them
// in double).
struct RemapParamF {
    int type;  // 0 rectilinear, else fisheye
    float srcTX, srcTY, destTX, destTY;
    float scale0, scale1, shear0, shear1, rot0, rot1;
    float rad[6];
    float mt[9];
    float distance, horizontal, vertical;
};

// The tensor maps of one level for k_blend's producer (boxes of the bulk
// tensor copies): the level's G tile (64 x 16 x 1 of uint32 over pitch x h x
// cameras), its G footprint as the level above a blend (40 x 10 x 1), its
// collapsed C footprint (36 x 10 of 8-byte pixels over pitch x h) and its
// weight tile (64 x 16 x 1 of uint16).
constexpr int kTmG = 0, kTmGfp = 1, kTmC = 2, kTmW = 3, kTmapsPerLevel = 4;

// Bits of a frame's error word: a bounded wait of a blend kernel, of the remap
// ran out.
constexpr int kStatusBlend = 4, kStatusRemap = 8;

struct RigDev {
    int n, L, W, H;
    int full;                 // union of coverages == whole canvas
    int srcW, srcH;
    const float2* maps;       // tile-compact maps of all cameras (NULL when map-free)
    int numRemapItems;        // tiles of the maps (and of the map-free coverage words)
    // map-free remap: per camera its parameters, per remap tile (in map-tile
    // order) its coverage as 16 words of 32 bits, one word per tile row
    const RemapParamF* camsF;
    const uint32_t* covTiles;
    const uint8_t* unionMask; // level-0 union coverage (0/255), pitch = lv[0].pitch
    const uint8_t* camLists;  // camera indices of blend tiles with more than 8 cameras
    // TMA tensor maps of this state slot (CUtensorMap, 128 bytes each, 64-byte
    // aligned in device memory), kTmapsPerLevel per level: see kTmG ... kTmW;
    // NULL when they could not be encoded (k_blend's consumers then stage the
    // units themselves)
    const void* tmaps;
    LevelDev lv[PS_MAX_LEVELS + 1];
    // the top of the pyramid in one launch (k_tail): pyrDown and blend levels
    // tailStart..L (L + 1 = none), and of each the cameras with a pyrDown tile
    int tailStart;
    uint32_t tailCams[PS_MAX_LEVELS + 1];
    // linear-blend mode: the remap items (tile-major) and their weights,
    // 512 floats per item in the layout of the maps
    const RemapItem* remapItems;
    const float* linWeights;
};

// Per-frame arguments of one rig in a launch (device resident, rewritten
// before every launch sequence).
struct FrameDev {
    const uint8_t* src[PS_MAX_CAMS];
    long long srcPitch[PS_MAX_CAMS];
    int srcFmt;               // PS_FMT_BGR24 / PS_FMT_BGR32
    int outFmt;               // PS_FMT_BGR24 / BGR32 / YUV420P / NV12
    uint8_t* out;             // BGR canvas, or the Y plane
    long long outPitch;
    uint8_t* outU;            // YUV420P: U plane; NV12: interleaved UV plane
    uint8_t* outV;            // YUV420P: V plane
    long long outCPitch;      // pitch of the U (or UV) plane
    long long outVPitch;      // pitch of the V plane
    const uint8_t* luts;      // n * 768 device bytes (B, G, R tables)
    int* status;              // device error word (0 = ok; kStatusBlend ...)
};

// Decoder frames to convert to BGR32 (k_yuv_to_bgr32): YUV420P (u, v
// planes) or NV12 (u = the interleaved UV plane), all w x h (even).
struct YuvFrame {
    const uint8_t *y, *u, *v;
    long long yPitch, uPitch, vPitch;
    uint8_t* dst;
    long long dstPitch;
    int fmt;
};
struct YuvFrames {
    YuvFrame frame[PS_MAX_CAMS];
    int n, w, h;
};

// A launch runs the concatenation of segments: `count` items of one rig,
// numbered from `prefix` in the launch.  Several rigs (a batch, or the
// frames of a serving tick) share one launch this way.
struct Segment {
    const void* items;
    const RigDev* rig;
    const FrameDev* frame;
    int count, prefix;
};

#ifdef __CUDACC__
// Item `it` of a launch -> its segment, scanning forward from a hint (each
// CTA visits its items in increasing order).
__device__ __forceinline__ int findSegment(const Segment* segs, int nsegs, int it, int hint)
{
    int s = hint;
    while (s + 1 < nsegs && segs[s + 1].prefix <= it) s++;
    return s;
}

// Contiguous chunk of items for this CTA (k_pyrdown): neighbouring tiles of
// one camera stay on one SM, and no item is handed out through an atomic.  The
// CTAs' shares differ by one item at most: equal shares rounded up left the
// last CTAs, and with them some SMs, idle (a frame of 8 x 3840x2160 to 7680x3840
// 419.5 us, 417.3 us so; of 2048x1024 74.0 and 72.7).
__device__ __forceinline__ void itemRange(int total, int& begin, int& end)
{
    begin = (int)((long long)total * blockIdx.x / gridDim.x);
    end = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
}

// ---- borders: source/CudaAccel/CudaUtil.cuh:6-98 ------------------------------
// Vertical reflect-101 (BrdColReflect101) and horizontal wrap (BrdRowWrap),
// restated with the reference's exact index formulas.
// The divisions are for levels smaller than a filter's reach; they are a
// hundred cycles each, and the few-tile levels map every row and column.
__device__ __forceinline__ int rowLow(int y, int H) { return abs(y) % H; }
__device__ __forceinline__ int rowHigh(int y, int H) { int last = H - 1; return abs(last - abs(last - y)) % H; }
__device__ __forceinline__ int colLow(int x, int W) { return x >= 0 ? x : x - ((x - W + 1) / W) * W; }
__device__ __forceinline__ int colHigh(int x, int W) { return x < W ? x : x % W; }
// any row index of a pyramid tile -> the row the reference reads
__device__ __forceinline__ int rowMap(int y, int H)
{
    const int r = y < 0 ? -y : (y >= H ? 2 * (H - 1) - y : y);  // one reflection
    if ((unsigned)r < (unsigned)H) return r;
    return y < 0 ? rowLow(y, H) : rowHigh(y, H);
}
__device__ __forceinline__ int colMap(int x, int W)
{
    const int c = x < 0 ? x + W : (x >= W ? x - W : x);  // one turn
    if ((unsigned)c < (unsigned)W) return c;
    return x < 0 ? colLow(x, W) : colHigh(x, W);
}

// C truncating division a / d given rcp = __frcp_rn(d), exact for |a| < 2^24
// (exact in fp32), 1 <= d < 2^16 and |a| / d < 2^21: the fp32 quotient then
// has a relative error below 2^-22, so it is within 1 of the true one, and one
// remainder check fixes it.  The normalisation divides weighted sums of
// Laplacians by their weight sums: |a| <= 255 d < 2^23, quotients <= 255.
__device__ __forceinline__ int divTrunc(int a, int d, float rcp)
{
    const int m = abs(a);
    int q = (int)__fmul_rz((float)m, rcp);
    const int r = m - q * d;
    q += (r >= d) - (r < 0);
    return a < 0 ? -q : q;
}

// Programmatic dependent launch: wait until the previous kernel in the
// stream has completed and its writes are visible (everything before this
// call may only touch data that kernel does not write).
__device__ __forceinline__ void waitPrevGrid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Let the next kernel in the stream start launching (its CTAs block in
// waitPrevGrid until this grid completes).
__device__ __forceinline__ void allowNextGrid() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// ---- packed channel arithmetic -----------------------------------------------
// A BGRX byte quad splits into two words holding 16-bit lanes:
//   lo = B | R << 16,  hi = G | X << 16.
// Sums of up to 256 weighted bytes stay below 65536, so the 5x5 pyramid
// filters run two channels per 32-bit add with no carry between lanes.
__device__ __forceinline__ uint2 unpackBytes(uint32_t v)
{
    return make_uint2(v & 0x00FF00FFu, (v >> 8) & 0x00FF00FFu);
}
#endif  // __CUDACC__

}  // namespace ps
