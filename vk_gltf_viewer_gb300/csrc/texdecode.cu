// Block-compressed texture decode on the device: BC1-BC5 (the DXT1-5 /
// RGTC formats a DDS base-colour texture holds, MSFT_texture_dds) and BC7 into RGBA8
// for the textured resolve, and BC6H into float32 RGB.  The reference loads no images
// (src/vk_gltf_viewer/assets.cpp:467-471); the formats are the published
// ones, with the interpolation rounding, which they leave to the
// implementation, pinned here and in the oracle:
//   RGB565 -> 8 bits: (r5 << 3 | r5 >> 2), (g6 << 2 | g6 >> 4)
//   BC1 (c0 > c1) and BC2/BC3 colours: c2 = (2 c0 + c1 + 1) / 3,
//                                      c3 = (c0 + 2 c1 + 1) / 3
//   BC1 (c0 <= c1): c2 = (c0 + c1 + 1) / 2, c3 = transparent black (opaque
//     black for VKGV_BC1_OPAQUE, Vulkan's BC1_RGB formats)
//   BC2 alpha: a4 * 17
//   BC3 alpha / BC4 / BC5 channels (a0 > a1): a_i = ((7 - i) a0 + i a1 + 3) / 7
//     for the interpolated codes i = 1..6 (indices 2..7);
//     (a0 <= a1): a_i = ((5 - i) a0 + i a1 + 2) / 5 for i = 1..4 (indices 2..5),
//     index 6 = 0, index 7 = 255
//   BC4 -> (r, 0, 0, 255), BC5 -> (r, g, 0, 255)
// One thread per block: the palette is built once for its 16 texels.
#include <cuda_fp16.h>

#include <type_traits>

#include "kernels.cuh"

namespace vkgv {

namespace {

constexpr uint32_t kDecodeRows = 8;  // block rows per CTA of 32 x 8 threads (one warp per block row)

__device__ __forceinline__ uint32_t rgb565(uint32_t c) {
    const uint32_t r = (c >> 11) & 31u, g = (c >> 5) & 63u, b = c & 31u;
    return ((r << 3) | (r >> 2)) | (((g << 2) | (g >> 4)) << 8) | (((b << 3) | (b >> 2)) << 16);
}

__device__ __forceinline__ uint32_t ch(uint32_t c, int k) { return (c >> (8 * k)) & 255u; }

// The palette of a BC1-layout colour block (words lo = c0 | c1 << 16) by
// channel: byte j of plane[k] is entry j's channel k.
__device__ __forceinline__ void colour_palette(uint32_t lo, bool allow_three, bool opaque, uint32_t plane[4]) {
    const uint32_t c0 = lo & 0xFFFFu, c1 = lo >> 16;
    const uint32_t a = rgb565(c0), b = rgb565(c1);
    const bool four = !allow_three || c0 > c1;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t x = ch(a, k), y = ch(b, k);
        const uint32_t p2 = four ? (2 * x + y + 1) / 3 : (x + y + 1) / 2;
        const uint32_t p3 = four ? (x + 2 * y + 1) / 3 : 0u;
        plane[k] = x | (y << 8) | (p2 << 16) | (p3 << 24);
    }
    plane[3] = four || opaque ? 0xFFFFFFFFu : 0x00FFFFFFu;
}

// The 8-entry palette of an interpolated channel block, one byte an entry.
__device__ __forceinline__ void channel_palette(uint32_t lo, uint32_t& p0, uint32_t& p1) {
    const uint32_t a0 = lo & 255u, a1 = (lo >> 8) & 255u;
    uint32_t v[8];
    v[0] = a0;
    v[1] = a1;
    if (a0 > a1) {
#pragma unroll
        for (uint32_t j = 1; j <= 6; ++j) v[j + 1] = ((7 - j) * a0 + j * a1 + 3) / 7;
    } else {
#pragma unroll
        for (uint32_t j = 1; j <= 4; ++j) v[j + 1] = ((5 - j) * a0 + j * a1 + 2) / 5;
        v[6] = 0;
        v[7] = 255;
    }
    p0 = v[0] | (v[1] << 8) | (v[2] << 16) | (v[3] << 24);
    p1 = v[4] | (v[5] << 8) | (v[6] << 16) | (v[7] << 24);
}

// Four 2-bit (3-bit) codes, lowest first, as the four low nibbles of a byte
// selector: __byte_perm then looks four texels up at once.
__device__ __forceinline__ uint32_t nibbles2(uint32_t x) {
    return (x & 3u) | ((x & 0xCu) << 2) | ((x & 0x30u) << 4) | ((x & 0xC0u) << 6);
}

__device__ __forceinline__ uint32_t nibbles3(uint32_t x) {
    return (x & 7u) | ((x & 0x38u) << 1) | ((x & 0x1C0u) << 2) | ((x & 0xE00u) << 3);
}

// Row r (12 bits) of the 48 bits of 3-bit codes behind an interpolated
// channel block's two end points.
__device__ __forceinline__ uint32_t code_row(uint32_t lo, uint32_t hi, int r) {
    if (r == 0) return (lo >> 16) & 0xFFFu;
    if (r == 1) return __funnelshift_r(lo, hi, 28) & 0xFFFu;
    return (hi >> (r == 2 ? 8 : 20)) & 0xFFFu;
}

// Four texels from four channel planes (byte x of a plane is texel x's).
__device__ __forceinline__ uint4 interleave(uint32_t r, uint32_t g, uint32_t b, uint32_t a) {
    const uint32_t rg0 = __byte_perm(r, g, 0x5140), rg1 = __byte_perm(r, g, 0x7362);
    const uint32_t ba0 = __byte_perm(b, a, 0x5140), ba1 = __byte_perm(b, a, 0x7362);
    return make_uint4(__byte_perm(rg0, ba0, 0x5410), __byte_perm(rg0, ba0, 0x7632), __byte_perm(rg1, ba1, 0x5410),
                      __byte_perm(rg1, ba1, 0x7632));
}

// A warp's 32 consecutive rows of kWords words (lane l holds words
// [l * kWords, +kWords) of `words` contiguous words at dst) written with
// full-width stores: straight from the lanes when those are the contiguous
// 16 bytes, otherwise through the warp's shared-memory buffer in the widest
// word that dst's alignment allows (a lane's own stores would leave gaps of
// a block's row between lanes, and odd image widths misalign the rows).
template <int kWords>
__device__ __forceinline__ void store_rows(const uint32_t* v, uint32_t* buf, uint32_t lane, uint32_t* dst,
                                           uint32_t words) {
    const uint32_t align = (uint32_t)reinterpret_cast<uintptr_t>(dst) & 15u;
    if (kWords == 4 && align == 0 && words == 32 * kWords) {
        __stcs(reinterpret_cast<uint4*>(dst) + lane, make_uint4(v[0], v[1], v[2], v[3]));
        return;
    }
    __syncwarp();  // the buffer's previous row has been read
#pragma unroll
    for (int k = 0; k < kWords / 4; ++k)
        reinterpret_cast<uint4*>(buf)[lane * (kWords / 4) + k] =
            make_uint4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    __syncwarp();
    if (align == 0) {
        for (uint32_t i = lane; i < words / 4; i += 32)
            __stcs(reinterpret_cast<uint4*>(dst) + i, reinterpret_cast<const uint4*>(buf)[i]);
        const uint32_t i = (words & ~3u) + lane;
        if (i < words) __stcs(dst + i, buf[i]);
    } else if ((align & 7u) == 0) {
        for (uint32_t i = lane; i < words / 2; i += 32)
            __stcs(reinterpret_cast<uint2*>(dst) + i, reinterpret_cast<const uint2*>(buf)[i]);
        if ((words & 1u) && lane == 0) __stcs(dst + words - 1, buf[words - 1]);
    } else {
        for (uint32_t i = lane; i < words; i += 32) __stcs(dst + i, buf[i]);
    }
}

// BC1-BC5: one thread per block, a warp per 32 blocks of a block row, so that
// each of its four texel rows is one contiguous 512-byte store.  The codes of
// four texels pass through the palette's channel planes as byte selectors.
// Bound by its writes at 0.83-0.97 of the measured copy bandwidth (8192^2:
// BC1 94.9 -> 46.0 us, BC3 152 -> 59.4; with four lanes per block, one row each,
// the palette was built four times and looked up per texel).
// Where the image's rows are 16-byte words, each lane stores its own: through
// the warp's buffer whenever a row held fewer than 32 blocks, narrow images were
// slower than with four lanes per block (BC1 4x16384 3.0 -> 3.5 us, now 2.7; 4x4
// 1.1 -> 1.5, now 1.25; and 4096^2 12.1, now 9.9).
template <uint32_t FORMAT>
__global__ void __launch_bounds__(32 * kDecodeRows) k_decode_bc(const uint8_t* __restrict__ blocks, uint32_t w,
                                                                uint32_t h, uint32_t* __restrict__ rgba) {
    pdl_begin();
    __shared__ __align__(16) uint32_t s_row[kDecodeRows][128];
    constexpr bool kBc1 = FORMAT == VKGV_BC1 || FORMAT == VKGV_BC1_OPAQUE;
    constexpr bool kWide = !kBc1 && FORMAT != VKGV_BC4;
    constexpr bool kColour = FORMAT != VKGV_BC4 && FORMAT != VKGV_BC5;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t bx0 = blockIdx.x * 32, bx = bx0 + lane, by = blockIdx.y * kDecodeRows + warp;
    const uint32_t bw = (w + 3) / 4, bh = (h + 3) / 4;
    if (by >= bh) return;  // whole warps
    uint4 q = make_uint4(0u, 0u, 0u, 0u);
    if (bx < bw) {
        const size_t at = (size_t)by * bw + bx;
        if (kWide) {
            q = __ldg(reinterpret_cast<const uint4*>(blocks) + at);
        } else {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(blocks) + at);
            q.x = v.x, q.y = v.y;
        }
    }
    uint32_t plane[4] = {0u, 0u, 0u, 0u}, p0 = 0u, p1 = 0u, g0 = 0u, g1 = 0u;
    // the colour block: words 0-1 (BC1) or 2-3 (BC2 / BC3, always four colours)
    const uint32_t cidx = kBc1 ? q.y : q.w;
    if (kColour) colour_palette(kBc1 ? q.x : q.z, kBc1, FORMAT == VKGV_BC1_OPAQUE, plane);
    if (FORMAT == VKGV_BC3 || FORMAT == VKGV_BC4 || FORMAT == VKGV_BC5) channel_palette(q.x, p0, p1);
    if (FORMAT == VKGV_BC5) channel_palette(q.z, g0, g1);
    const auto texels = [&](int r) {  // row r's four
        if (kColour) {
            const uint32_t sel = nibbles2((cidx >> (8 * r)) & 255u);
            uint32_t a = __byte_perm(plane[3], 0u, sel);
            if (FORMAT == VKGV_BC2) {
                const uint32_t n = ((r < 2 ? q.x : q.y) >> (16 * (r & 1))) & 0xFFFFu;
                a = ((n & 15u) | ((n & 0xF0u) << 4) | ((n & 0xF00u) << 8) | ((n & 0xF000u) << 12)) * 17u;
            }
            if (FORMAT == VKGV_BC3) a = __byte_perm(p0, p1, nibbles3(code_row(q.x, q.y, r)));
            return interleave(__byte_perm(plane[0], 0u, sel), __byte_perm(plane[1], 0u, sel),
                              __byte_perm(plane[2], 0u, sel), a);
        }
        const uint32_t red = __byte_perm(p0, p1, nibbles3(code_row(q.x, q.y, r)));
        const uint32_t green = FORMAT == VKGV_BC5 ? __byte_perm(g0, g1, nibbles3(code_row(q.z, q.w, r))) : 0u;
        return interleave(red, green, 0u, 0xFFFFFFFFu);
    };
    if (((w & 3u) | ((uint32_t)reinterpret_cast<uintptr_t>(rgba) & 15u)) == 0) {
        // every row of a block is a 16-byte word of the image
        if (bx >= bw) return;
        uint4* at = reinterpret_cast<uint4*>(rgba) + (size_t)by * w + bx;
#pragma unroll
        for (int r = 0; r < 4; ++r, at += bw)
            if (by * 4 + r < h) __stcs(at, texels(r));
        return;
    }
    const uint32_t words = min(128u, w - 4 * bx0);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint32_t y = by * 4 + r;
        if (y >= h) break;
        const uint4 t = texels(r);
        const uint32_t v[4] = {t.x, t.y, t.z, t.w};
        store_rows<4>(v, s_row[warp], lane, rgba + (size_t)y * w + (size_t)bx0 * 4, words);
    }
}

// BC7 (BPTC UNORM), decoded as the published format defines it: the mode from the
// lowest set bit of the first byte; per mode the subset count, partition
// bits, rotation and index-selection bits, colour / alpha endpoint bits,
// p-bits (per endpoint or shared per subset) and one or two index sets;
// endpoints expanded to 8 bits by replicating their top bits; texels
// interpolated as ((64 - w) e0 + w e1 + 32) >> 6 with the 2-, 3- and 4-bit
// weight tables; the anchor texel of each subset stores one index bit less.
// A reserved mode (first byte 0) decodes to transparent black.  The
// partition and anchor tables below are the format's own.  They lie in global
// memory: a CTA copies them in a few coalesced loads.
__device__ const uint16_t g_bc7_p2[64] = {
    0xCCCC, 0x8888, 0xEEEE, 0xECC8, 0xC880, 0xFEEC, 0xFEC8, 0xEC80, 0xC800, 0xFFEC, 0xFE80, 0xE800,
    0xFFE8, 0xFF00, 0xFFF0, 0xF000, 0xF710, 0x008E, 0x7100, 0x08CE, 0x008C, 0x7310, 0x3100, 0x8CCE,
    0x088C, 0x3110, 0x6666, 0x366C, 0x17E8, 0x0FF0, 0x718E, 0x399C, 0xAAAA, 0xF0F0, 0x5A5A, 0x33CC,
    0x3C3C, 0x55AA, 0x9696, 0xA55A, 0x73CE, 0x13C8, 0x324C, 0x3BDC, 0x6996, 0xC33C, 0x9966, 0x0660,
    0x0272, 0x04E4, 0x4E40, 0x2720, 0xC936, 0x936C, 0x39C6, 0x639C, 0x9336, 0x9CC6, 0x817E, 0xE718,
    0xCCF0, 0x0FCC, 0x7744, 0xEE22};
// 3-subset partitions: two bits per texel, texel 0 in the lowest bits
__device__ const uint32_t g_bc7_p3[64] = {
    0xAA685050, 0x6A5A5040, 0x5A5A4200, 0x5450A0A8, 0xA5A50000, 0xA0A05050, 0x5555A0A0, 0x5A5A5050,
    0xAA550000, 0xAA555500, 0xAAAA5500, 0x90909090, 0x94949494, 0xA4A4A4A4, 0xA9A59450, 0x2A0A4250,
    0xA5945040, 0x0A425054, 0xA5A5A500, 0x55A0A0A0, 0xA8A85454, 0x6A6A4040, 0xA4A45000, 0x1A1A0500,
    0x0050A4A4, 0xAAA59090, 0x14696914, 0x69691400, 0xA08585A0, 0xAA821414, 0x50A4A450, 0x6A5A0200,
    0xA9A58000, 0x5090A0A8, 0xA8A09050, 0x24242424, 0x00AA5500, 0x24924924, 0x24499224, 0x50A50A50,
    0x500AA550, 0xAAAA4444, 0x66660000, 0xA5A0A5A0, 0x50A050A0, 0x69286928, 0x44AAAA44, 0x66666600,
    0xAA444444, 0x54A854A8, 0x95809580, 0x96969600, 0xA85454A8, 0x80959580, 0xAA141414, 0x96960000,
    0xAAAA1414, 0xA05050A0, 0xA0A5A5A0, 0x96000000, 0x40804080, 0xA9A8A9A8, 0xAAAAAA44, 0x2A4A5254};
__device__ const uint8_t g_bc7_a2[64] = {
    15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 2, 8, 2, 2, 8, 8, 15, 2, 8,
    2, 2, 8, 8, 2, 2, 15, 15, 6, 8, 2, 8, 15, 15, 2, 8, 2, 2, 2, 15, 15, 6, 6, 2, 6, 8, 15, 15, 2,
    2, 15, 15, 15, 15, 15, 2, 2, 15};
__device__ const uint8_t g_bc7_a3a[64] = {
    3, 3, 15, 15, 8, 3, 15, 15, 8, 8, 6, 6, 6, 5, 3, 3, 3, 3, 8, 15, 3, 3, 6, 10, 5, 8, 8, 6, 8, 5,
    15, 15, 8, 15, 3, 5, 6, 10, 8, 15, 15, 3, 15, 5, 15, 15, 15, 15, 3, 15, 5, 5, 5, 8, 5, 10, 5,
    10, 8, 13, 15, 12, 3, 3};
__device__ const uint8_t g_bc7_a3b[64] = {
    15, 8, 8, 3, 15, 15, 3, 8, 15, 15, 15, 15, 15, 15, 15, 8, 15, 8, 15, 3, 15, 8, 15, 8, 3, 15, 6,
    10, 15, 15, 10, 8, 15, 3, 15, 10, 10, 8, 9, 10, 6, 15, 8, 15, 3, 6, 6, 8, 15, 3, 15, 15, 15, 15,
    15, 15, 15, 15, 15, 15, 3, 15, 15, 8};

// The interpolation weights of 2-, 3- and 4-bit indices ({0, 21, 43, 64},
// {0, 9, 18, 27, 37, 46, 55, 64}, {0, 4, 9, 13, 17, 21, 26, 30, 34, 38, 43,
// 47, 51, 55, 60, 64}) by their arithmetic: of one index (3 or 4 bits), and four
// at a time below.
template <int BITS>
__device__ __forceinline__ uint32_t index_weight(uint32_t i) {
    if (BITS == 3) return i * 9u + (i >> 2);
    return (i * 17u + 2u) >> 2;
}

// The four BITS-bit indices in the low bits of `v` as the bytes of a word, and
// the weights of such a word, four at a time.
template <int BITS>
__device__ __forceinline__ uint32_t spread_indices(uint32_t v) {
    constexpr uint32_t one = (1u << BITS) - 1u, two = (1u << (2 * BITS)) - 1u;
    v = (v | (v << (16 - 2 * BITS))) & (two * 0x00010001u);
    return (v | (v << (8 - BITS))) & (one * 0x01010101u);
}

template <int BITS>
__device__ __forceinline__ uint32_t index_weights(uint32_t i) {
    if (BITS == 2) return i * 21u + ((i >> 1) & 0x01010101u);
    if (BITS == 3) return i * 9u + ((i >> 2) & 0x01010101u);
    return i * 4u + (((i + 0x02020202u) >> 2) & 0x07070707u);
}

// N bits of the 128-bit block at bit POS, least significant first.
template <int POS, int N>
__device__ __forceinline__ uint32_t block_bits(const uint4& q) {
    if constexpr (N == 0) {
        return 0u;
    } else {
        constexpr int k = POS / 32, s = POS % 32;
        const uint32_t lo = k == 0 ? q.x : (k == 1 ? q.y : (k == 2 ? q.z : q.w));
        const uint32_t hi = k == 0 ? q.y : (k == 1 ? q.z : (k == 2 ? q.w : 0u));
        const uint32_t v = s + N <= 32 ? lo >> s : __funnelshift_r(lo, hi, s);
        return N == 32 ? v : v & ((1u << (N & 31)) - 1u);
    }
}

// The block's bits from POS to its end (at most 64).
template <int POS>
__device__ __forceinline__ uint64_t block_tail(const uint4& q) {
    const uint64_t hi = (uint64_t)q.z | ((uint64_t)q.w << 32);
    if constexpr (POS >= 64) {
        return hi >> (POS - 64);
    } else {
        const uint64_t lo = (uint64_t)q.x | ((uint64_t)q.y << 32);
        return (lo >> POS) | (hi << (64 - POS));
    }
}

// Gives an anchor texel the index bit that the format leaves out: a zero bit
// at position p, the bits from p on moving up by one.
template <class T>
__device__ __forceinline__ T insert_zero(T v, uint32_t p) {
    return v + (v & ((T)~T(0) << p));
}

// One BC7 mode.  Stored fields in order: mode (unary), partition, rotation,
// index selection, R of every end point (subset-major), then G, B and alpha,
// the p-bits, then one or two index sets that end with the block.
template <int MODE>
struct Bc7Mode {
    static constexpr int kSubsets = MODE == 0 || MODE == 2 ? 3 : (MODE == 1 || MODE == 3 || MODE == 7 ? 2 : 1);
    static constexpr int kPartBits = MODE == 0 ? 4 : (kSubsets > 1 ? 6 : 0);
    static constexpr int kRotBits = MODE == 4 || MODE == 5 ? 2 : 0;
    static constexpr int kSelBits = MODE == 4 ? 1 : 0;
    static constexpr int kColour = MODE == 0 ? 4 : (MODE == 1 ? 6 : (MODE == 3 || MODE == 5 || MODE == 6 ? 7 : 5));
    static constexpr int kAlpha = MODE == 4 ? 6 : (MODE == 5 ? 8 : (MODE == 6 ? 7 : (MODE == 7 ? 5 : 0)));
    static constexpr bool kEndP = MODE == 0 || MODE == 3 || MODE == 6 || MODE == 7;  // a p-bit per end point
    static constexpr bool kSubP = MODE == 1;                                        // a p-bit per subset
    static constexpr int kIndex = MODE == 0 || MODE == 1 ? 3 : (MODE == 6 ? 4 : 2);
    static constexpr int kIndex2 = MODE == 4 ? 3 : (MODE == 5 ? 2 : 0);
    static constexpr int kEnds = 2 * kSubsets;
    static constexpr int kPartAt = MODE + 1;
    static constexpr int kRotAt = kPartAt + kPartBits;
    static constexpr int kSelAt = kRotAt + kRotBits;
    static constexpr int kColourAt = kSelAt + kSelBits;
    static constexpr int kAlphaAt = kColourAt + 3 * kEnds * kColour;
    static constexpr int kPAt = kAlphaAt + kEnds * kAlpha;
    static constexpr int kIndexAt = kPAt + (kEndP ? kEnds : (kSubP ? kSubsets : 0));
    static constexpr int kIndex2At = kIndexAt + 16 * kIndex - kSubsets;
    static_assert((kIndex2 ? kIndex2At + 16 * kIndex2 - 1 : kIndex2At) == 128, "a BC7 block is 128 bits");
};

// A stored end point value (with its p-bit) expanded to 8 bits.
template <int BITS>
__device__ __forceinline__ uint32_t bc7_expand(uint32_t v) {
    v <<= 8 - BITS;
    return v | (v >> BITS);
}

// End point K of a block: red and blue, green and alpha, in the two halves
// of a word each, so that one multiplication interpolates two channels.
template <int MODE, int K>
__device__ __forceinline__ void bc7_end(const uint4& q, uint32_t& rb, uint32_t& ga) {
    using M = Bc7Mode<MODE>;
    constexpr int cb = M::kColour, ab = M::kAlpha, n = M::kEnds;
    uint32_t r = block_bits<M::kColourAt + K * cb, cb>(q), g = block_bits<M::kColourAt + (n + K) * cb, cb>(q);
    uint32_t b = block_bits<M::kColourAt + (2 * n + K) * cb, cb>(q);
    uint32_t a = ab ? block_bits<M::kAlphaAt + K * ab, ab>(q) : 255u;
    constexpr int p = M::kEndP || M::kSubP ? 1 : 0;
    if constexpr (p) {
        const uint32_t bit = block_bits<M::kPAt + (M::kEndP ? K : K / 2), 1>(q);
        r = (r << 1) | bit, g = (g << 1) | bit, b = (b << 1) | bit;
        if constexpr (ab && M::kEndP) a = (a << 1) | bit;
    }
    if constexpr (ab != 0) a = bc7_expand<ab + (M::kEndP ? 1 : 0)>(a);
    rb = bc7_expand<cb + p>(r) | (bc7_expand<cb + p>(b) << 16);
    ga = bc7_expand<cb + p>(g) | (a << 16);
}

// The partition and anchor tables in shared memory, by partition: the lanes
// of a warp look up different ones.
struct Bc7Tables {
    uint32_t two[64];    // 2 subsets: the partition, the anchor in bits 16-19
    uint32_t three[64];  // 3 subsets: the partition
    uint16_t after[64];  // and its anchors in ascending order, 8 bits each
};

__device__ __forceinline__ void bc7_load_tables(Bc7Tables& t) {
    const uint32_t i = threadIdx.x;
    if (i < 64) {
        t.two[i] = g_bc7_p2[i] | ((uint32_t)g_bc7_a2[i] << 16);
        t.three[i] = g_bc7_p3[i];
        const uint32_t a = g_bc7_a3a[i], b = g_bc7_a3b[i];
        t.after[i] = (uint16_t)(min(a, b) | (max(a, b) << 8));
    }
}

// Decodes one block of MODE; row r goes to out[r * pitch].  Every field is at
// a position known at compile time, and the index stream is brought to a
// fixed width a texel by inserting the anchors' zero bits.
// A texel's ((64 - w) e0 + w e1 + 32) >> 6 is the high byte of
// 4 (64 e0 + 32) + w 4 (e1 - e0), at most 65,408: a word holds two channels,
// whose sums are exact modulo 2^32, so a texel is two multiply-adds and one
// byte permutation.
template <int MODE>
__device__ __forceinline__ void bc7_block(const Bc7Tables& T, const uint4& q, uint4* out, uint32_t pitch) {
    using M = Bc7Mode<MODE>;
    constexpr int ib = M::kIndex, ib2 = M::kIndex2;
    uint32_t base[2 * M::kSubsets], step[2 * M::kSubsets];  // red and blue, green and alpha of each subset
    uint32_t e0, e1, f0, f1;
    const auto line = [&](int k) {
        base[2 * k] = 256u * e0 + 0x00800080u, step[2 * k] = 4u * (e1 - e0);
        base[2 * k + 1] = 256u * f0 + 0x00800080u, step[2 * k + 1] = 4u * (f1 - f0);
    };
    bc7_end<MODE, 0>(q, e0, f0);
    bc7_end<MODE, 1>(q, e1, f1);
    uint32_t base_a = 0, step_a = 0;
    if constexpr (ib2 != 0) {  // alpha has weights of its own
        base_a = 256u * (f0 >> 16) + 0x80u, step_a = 4u * ((f1 >> 16) - (f0 >> 16));
        f0 &= 255u, f1 &= 255u;
    }
    line(0);
    if constexpr (M::kSubsets > 1) {
        bc7_end<MODE, 2>(q, e0, f0);
        bc7_end<MODE, 3>(q, e1, f1);
        line(1);
    }
    if constexpr (M::kSubsets > 2) {
        bc7_end<MODE, 4>(q, e0, f0);
        bc7_end<MODE, 5>(q, e1, f1);
        line(2);
    }
    const uint32_t part = block_bits<M::kPartAt, M::kPartBits>(q);
    using Stream = std::conditional_t<ib == 2, uint32_t, uint64_t>;
    using Stream2 = std::conditional_t<ib2 == 2, uint32_t, uint64_t>;
    Stream ix = (Stream)block_tail<M::kIndexAt>(q);
    Stream2 ix2 = 0;
    if constexpr (ib2 != 0) {
        ix &= (Stream)((1ull << (16 * ib - 1)) - 1ull);
        ix2 = insert_zero((Stream2)block_tail<M::kIndex2At>(q), ib2 - 1);
    }
    ix = insert_zero(ix, ib - 1);
    uint32_t pmask = 0u;
    if constexpr (M::kSubsets == 2) {
        pmask = T.two[part];
        ix = insert_zero(ix, (pmask >> 16) * ib + ib - 1);
    } else if constexpr (M::kSubsets == 3) {
        pmask = T.three[part];
        const uint32_t after = T.after[part];
        ix = insert_zero(ix, (after & 255u) * ib + ib - 1);
        ix = insert_zero(ix, (after >> 8) * ib + ib - 1);
    }
    // alpha (byte 5 of the last permutation) swaps with R (1), G (2) or B (3)
    uint32_t order = 0x5210u;
    bool second = false;  // mode 4: the colours take the second index set
    if constexpr (M::kRotBits != 0) {
        const uint32_t rot = block_bits<M::kRotAt, 2>(q);
        order = rot == 0 ? 0x5210u : (rot == 1 ? 0x0215u : (rot == 2 ? 0x1250u : 0x2510u));
        second = block_bits<M::kSelAt, M::kSelBits>(q) != 0;
    }
#pragma unroll 1
    for (int r = 0; r < 4; ++r) {
        uint32_t t[4];
        uint32_t wc = index_weights<ib>(spread_indices<ib>((uint32_t)(ix >> (4 * ib * r)) & ((1u << (4 * ib)) - 1u)));
        uint32_t wa = 0;
        if constexpr (ib2 != 0) {
            wa = index_weights<ib2>(spread_indices<ib2>((uint32_t)(ix2 >> (4 * ib2 * r)) & ((1u << (4 * ib2)) - 1u)));
            const uint32_t w = wc;
            wc = second ? wa : w, wa = second ? w : wa;
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = 4 * r + x;
            uint32_t b0 = base[0], d0 = step[0], b1 = base[1], d1 = step[1];
            if constexpr (M::kSubsets == 2) {
                const bool s = (pmask >> i) & 1u;
                b0 = s ? base[2] : b0, d0 = s ? step[2] : d0, b1 = s ? base[3] : b1, d1 = s ? step[3] : d1;
            } else if constexpr (M::kSubsets == 3) {
                const bool s = (pmask >> (2 * i)) & 1u, s2 = (pmask >> (2 * i)) & 2u;
                b0 = s ? base[2] : (s2 ? base[4] : b0), d0 = s ? step[2] : (s2 ? step[4] : d0);
                b1 = s ? base[3] : (s2 ? base[5] : b1), d1 = s ? step[3] : (s2 ? step[5] : d1);
            }
            const uint32_t w = (wc >> (8 * x)) & 255u, v = b0 + w * d0, u = b1 + w * d1;
            t[x] = __byte_perm(v, u, 0x7351u);
            if constexpr (ib2 != 0) t[x] = __byte_perm(t[x], base_a + ((wa >> (8 * x)) & 255u) * step_a, order);
        }
        out[r * pitch] = make_uint4(t[0], t[1], t[2], t[3]);
    }
}

// BC7: a CTA decodes a tile of 512 blocks (tw wide, a power of two) sorted by
// mode, so that each warp runs one mode's code, whose fields are at constant
// positions; a thread decodes a whole block, and the rows leave through
// shared memory, each as one bulk copy where the image's rows are 16-byte
// aligned.  The lists of the modes are padded to whole warps (some 20 warp
// jobs a tile instead of 16).  Bound by instruction issue (ALU pipe 65% of its
// cycles).  8192^2, modes as encoders choose them: 551 us with four lanes per
// block in image order, every field at a position looked up at run time;
// 191 sorted; 84 with packed weights, a multiply-add for two channels, jobs
// found by a ballot, the row loop rolled (the eight modes unrolled overran the
// instruction cache: 112) and the bulk copies (97 without).  Stores straight
// to the image saved the last barrier (4096^2: 1,024-block tiles 23.6 us, this
// 25.0), but their half sectors went to memory and back once the image was
// past L2 (8192^2: 148 us).
constexpr uint32_t kBc7Blocks = 512, kBc7Threads = 256, kBc7Each = kBc7Blocks / kBc7Threads;

__global__ void __launch_bounds__(kBc7Threads, 6)
    k_decode_bc7(const uint8_t* __restrict__ blocks, uint32_t w, uint32_t h, uint32_t tw_log2,
                 uint32_t* __restrict__ rgba) {
    __shared__ Bc7Tables T;
    __shared__ uint32_t s_count[9];                     // blocks of each mode (8: reserved)
    __shared__ uint16_t s_list[kBc7Blocks + 9 * 32];    // tile positions by mode, each mode's padded to a warp
    __shared__ __align__(16) uint4 s_out[4 * kBc7Blocks];
    bc7_load_tables(T);
    if (threadIdx.x < 9) s_count[threadIdx.x] = 0;
    pdl_begin();
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t tw = 1u << tw_log2, th = kBc7Blocks >> tw_log2;
    const uint32_t bw = (w + 3) / 4, bh = (h + 3) / 4;
    const uint32_t bx0 = blockIdx.x * tw, by0 = blockIdx.y * th;
    const uint4* src = reinterpret_cast<const uint4*>(blocks) + ((size_t)by0 * bw + bx0);
    uint32_t mode[kBc7Each], rank[kBc7Each];
#pragma unroll
    for (uint32_t k = 0; k < kBc7Each; ++k) {
        const uint32_t i = threadIdx.x + k * kBc7Threads, x = i & (tw - 1), y = i >> tw_log2;
        // the mode is the lowest set bit of the first byte; none: reserved
        mode[k] = 9u;
        if (bx0 + x < bw && by0 + y < bh) {
            const uint32_t q = __ldg(&src[(size_t)y * bw + x].x) & 0xFFu;
            mode[k] = q ? (uint32_t)__ffs((int)q) - 1u : 8u;
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < kBc7Each; ++k) {
        const unsigned same = __match_any_sync(0xffffffffu, mode[k]);
        const int leader = __ffs((int)same) - 1;
        uint32_t base = 0;
        if ((int)lane == leader && mode[k] < 9) base = atomicAdd(&s_count[mode[k]], (uint32_t)__popc(same));
        rank[k] = __shfl_sync(0xffffffffu, base, leader) + (uint32_t)__popc(same & ((1u << lane) - 1u));
    }
    __syncthreads();
    // warp jobs: mode m owns jobs [first_m, first_m + ceil(count_m / 32)),
    // lane m of every warp holds its count and first
    const uint32_t count = lane < 9 ? s_count[lane] : 0u;
    uint32_t jobs = (count + 31) / 32;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const uint32_t below = __shfl_up_sync(0xffffffffu, jobs, d);
        if ((int)lane >= d) jobs += below;
    }
    const uint32_t first = jobs - (count + 31) / 32;
    jobs = __shfl_sync(0xffffffffu, jobs, 9);
#pragma unroll
    for (uint32_t k = 0; k < kBc7Each; ++k) {
        const uint32_t base = __shfl_sync(0xffffffffu, first, (int)mode[k]);
        if (mode[k] < 9) s_list[32 * base + rank[k]] = (uint16_t)(threadIdx.x + k * kBc7Threads);
    }
    __syncthreads();
    for (uint32_t j = warp; j < jobs; j += kBc7Threads / 32) {
        const uint32_t m = 31u - (uint32_t)__clz((int)__ballot_sync(0xffffffffu, count != 0 && first <= j));
        const uint32_t at = 32 * (j - __shfl_sync(0xffffffffu, first, (int)m));
        if (at + lane < __shfl_sync(0xffffffffu, count, (int)m)) {
            const uint32_t i = s_list[32 * j + lane], x = i & (tw - 1), y = i >> tw_log2;
            const uint4 q = __ldg(src + (size_t)y * bw + x);
            uint4* out = s_out + ((y << (tw_log2 + 2)) + x);
            switch (m) {  // the same for the whole warp
                case 0: bc7_block<0>(T, q, out, tw); break;
                case 1: bc7_block<1>(T, q, out, tw); break;
                case 2: bc7_block<2>(T, q, out, tw); break;
                case 3: bc7_block<3>(T, q, out, tw); break;
                case 4: bc7_block<4>(T, q, out, tw); break;
                case 5: bc7_block<5>(T, q, out, tw); break;
                case 6: bc7_block<6>(T, q, out, tw); break;
                case 7: bc7_block<7>(T, q, out, tw); break;
                default:  // a reserved mode decodes to transparent black
                    for (uint32_t r = 0; r < 4; ++r) out[r * tw] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    }
    // the tile's texel rows, each 4 tw texels, contiguous in the image
    const uint32_t px = min(4 * tw, w - 4 * bx0), rows = min(4 * th, h - 4 * by0);
    uint32_t* dst = rgba + (size_t)by0 * 4 * w + (size_t)bx0 * 4;
    if ((w & 3u) == 0 && ((uint32_t)reinterpret_cast<uintptr_t>(rgba) & 15u) == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x < rows) {  // a bulk copy a row
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst + (size_t)threadIdx.x * w),
                         "r"((uint32_t)__cvta_generic_to_shared(s_out + (threadIdx.x << tw_log2))), "r"(4 * px)
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else {
        __syncthreads();
        const uint32_t* texels = reinterpret_cast<const uint32_t*>(s_out);
        for (uint32_t i = threadIdx.x; i < 16 * kBc7Blocks; i += kBc7Threads) {
            const uint32_t x = i & (4 * tw - 1), y = i >> (tw_log2 + 2);
            if (x < px && y < rows) __stcs(dst + (size_t)y * w + x, texels[i]);
        }
    }
}

// ------------------------------------------------------------------- BC6H
// BC6H (BPTC float; UF16 unsigned, SF16 signed) into float32 RGB (a linear
// VKGV_TEXTURE_RGB32F texture): the published format and the steps the
// oracle restates (oracle/texture.c), with the same partition, anchor and
// weight tables.  A 2-bit mode (values 0, 1) or a 5-bit one selects one of
// fourteen header layouts (the oracle's stream-order tokens regrouped by
// field, so that each field is assembled in its own register), transformed
// modes add signed
// deltas to the base endpoint, endpoints are unquantised to 16 bits, texels
// interpolated with the 3- or 4-bit BC7 weights and scaled to binary16
// (unsigned v * 31 >> 6; signed magnitude * 31 >> 5, sign only on a
// non-zero result).  Reserved modes decode to 0.
// Header tokens grouped by field (endpoint w, x, y, z x channel R, G, B;
// 12 = partition), per mode: the bit position in the block (bits 0-6), the
// lowest field bit (7-10), bit count - 1 (11-14) and reversed (15: the first
// block bit is the highest field bit); the counts follow.  Compile-time
// tables: each mode's parse is code of its own.
constexpr uint16_t kBc6Tok[14][13][6] = {
    {{0x4805, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x480F, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4819, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2023, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x202D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2037, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2041, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0202, 0x1829, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0203, 0x183D, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2047, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0228, 0x1833, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0204, 0x0032, 0x00BC, 0x0146, 0x01CC, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x00
    {{0x3005, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x300F, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x3019, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2823, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x282D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2837, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2841, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0282, 0x0218, 0x1829, 0x0000, 0x0000, 0x0000}, {0x020E, 0x0296, 0x183D, 0x0000, 0x0000, 0x0000}, {0x2847, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0A03, 0x1833, 0x0000, 0x0000, 0x0000, 0x0000}, {0x080C, 0x0117, 0x01A0, 0x02A1, 0x0222, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x01
    {{0x4805, 0x0528, 0x0000, 0x0000, 0x0000, 0x0000}, {0x480F, 0x0531, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4819, 0x053B, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2023, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x182D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1837, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2041, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1829, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x183D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2047, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1833, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0032, 0x00BC, 0x0146, 0x01CC, 0x0000, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x02
    {{0x4805, 0x0527, 0x0000, 0x0000, 0x0000, 0x0000}, {0x480F, 0x0532, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4819, 0x053B, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1823, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x202D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1837, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1841, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1829, 0x024B, 0x0000, 0x0000, 0x0000, 0x0000}, {0x183D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1847, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0228, 0x1833, 0x0000, 0x0000, 0x0000, 0x0000}, {0x00BC, 0x0045, 0x0146, 0x01CC, 0x0000, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x06
    {{0x4805, 0x0527, 0x0000, 0x0000, 0x0000, 0x0000}, {0x480F, 0x0531, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4819, 0x053C, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1823, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x182D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2037, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1841, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1829, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0228, 0x183D, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1847, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1833, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0032, 0x08C5, 0x024B, 0x01CC, 0x0000, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x0A
    {{0x4005, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x400F, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4019, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2023, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x202D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2037, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2041, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0218, 0x1829, 0x0000, 0x0000, 0x0000, 0x0000}, {0x020E, 0x183D, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2047, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0228, 0x1833, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0222, 0x0032, 0x00BC, 0x0146, 0x01CC, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x0E
    {{0x3805, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x380F, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x3819, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2823, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x202D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2037, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2841, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0218, 0x1829, 0x0000, 0x0000, 0x0000, 0x0000}, {0x020E, 0x183D, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2847, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x020D, 0x1833, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0117, 0x09A1, 0x0032, 0x00BC, 0x0000, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x12
    {{0x3805, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x380F, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x3819, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2023, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x282D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2037, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2041, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0297, 0x0218, 0x1829, 0x0000, 0x0000, 0x0000}, {0x020E, 0x183D, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2047, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x02A1, 0x0228, 0x1833, 0x0000, 0x0000, 0x0000}, {0x000D, 0x0222, 0x00BC, 0x0146, 0x01CC, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x16
    {{0x3805, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x380F, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x3819, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2023, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x202D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2837, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2041, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0218, 0x1829, 0x0000, 0x0000, 0x0000, 0x0000}, {0x020E, 0x0297, 0x183D, 0x0000, 0x0000, 0x0000}, {0x2047, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0228, 0x1833, 0x0000, 0x0000, 0x0000, 0x0000}, {0x008D, 0x02A1, 0x0222, 0x0032, 0x0146, 0x01CC}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x1A
    {{0x2805, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x280F, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2819, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2823, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x282D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2837, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x2841, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0295, 0x0218, 0x1829, 0x0000, 0x0000, 0x0000}, {0x020E, 0x0296, 0x183D, 0x0000, 0x0000, 0x0000}, {0x2847, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x020B, 0x029F, 0x1833, 0x0000, 0x0000, 0x0000}, {0x080C, 0x0117, 0x01A0, 0x02A1, 0x0222, 0x0000}, {0x204D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x1E
    {{0x4805, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x480F, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4819, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4823, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x482D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4837, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x03
    {{0x4805, 0x052C, 0x0000, 0x0000, 0x0000, 0x0000}, {0x480F, 0x0536, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4819, 0x0540, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4023, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x402D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4037, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x07
    {{0x4805, 0x8D2B, 0x0000, 0x0000, 0x0000, 0x0000}, {0x480F, 0x8D35, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4819, 0x8D3F, 0x0000, 0x0000, 0x0000, 0x0000}, {0x3823, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x382D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x3837, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x0B
    {{0x4805, 0xAD27, 0x0000, 0x0000, 0x0000, 0x0000}, {0x480F, 0xAD31, 0x0000, 0x0000, 0x0000, 0x0000}, {0x4819, 0xAD3B, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1823, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x182D, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x1837, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}, {0x0000, 0x0000, 0x0000, 0x0000, 0x0000, 0x0000}},  // mode 0x0F
};
constexpr uint8_t kBc6Count[14][13] = {
    {1, 1, 1, 1, 1, 1, 1, 2, 2, 1, 2, 5, 1},  // mode 0x00
    {1, 1, 1, 1, 1, 1, 1, 3, 3, 1, 2, 5, 1},  // mode 0x01
    {2, 2, 2, 1, 1, 1, 1, 1, 1, 1, 1, 4, 1},  // mode 0x02
    {2, 2, 2, 1, 1, 1, 1, 2, 1, 1, 2, 4, 1},  // mode 0x06
    {2, 2, 2, 1, 1, 1, 1, 1, 2, 1, 1, 4, 1},  // mode 0x0A
    {1, 1, 1, 1, 1, 1, 1, 2, 2, 1, 2, 5, 1},  // mode 0x0E
    {1, 1, 1, 1, 1, 1, 1, 2, 2, 1, 2, 4, 1},  // mode 0x12
    {1, 1, 1, 1, 1, 1, 1, 3, 2, 1, 3, 5, 1},  // mode 0x16
    {1, 1, 1, 1, 1, 1, 1, 2, 3, 1, 2, 6, 1},  // mode 0x1A
    {1, 1, 1, 1, 1, 1, 1, 3, 3, 1, 3, 5, 1},  // mode 0x1E
    {1, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0},  // mode 0x03
    {2, 2, 2, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0},  // mode 0x07
    {2, 2, 2, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0},  // mode 0x0B
    {2, 2, 2, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0},  // mode 0x0F
};
// Per mode (fields 0x00, 0x01, 0x02, 0x06, .. 0x1E, 0x03, 0x07, 0x0B, 0x0F):
// transformed, endpoint bits, delta bits R, G, B, regions
constexpr uint8_t kBc6Mode[14][6] = {
    {1, 10, 5, 5, 5, 2}, {1, 7, 6, 6, 6, 2}, {1, 11, 5, 4, 4, 2}, {1, 11, 4, 5, 4, 2}, {1, 11, 4, 4, 5, 2},
    {1, 9, 5, 5, 5, 2}, {1, 8, 6, 5, 5, 2}, {1, 8, 5, 6, 5, 2}, {1, 8, 5, 5, 6, 2}, {0, 6, 6, 6, 6, 2},
    {0, 10, 10, 10, 10, 1}, {1, 11, 9, 9, 9, 1}, {1, 12, 8, 8, 8, 1}, {1, 16, 4, 4, 4, 1}};

__device__ __forceinline__ int32_t bc6_sext(uint32_t v, uint32_t n) {
    const uint32_t s = 32u - n;
    return (int32_t)(v << s) >> s;
}

__device__ __forceinline__ int32_t bc6_unquantize(int32_t c, uint32_t bits, bool sgn) {
    if (!sgn) {
        if (bits >= 15u) return c;
        if (c == 0) return 0;
        if (c == (int32_t)((1u << bits) - 1u)) return 0xFFFF;
        return (int32_t)((((uint32_t)c << 16) + 0x8000u) >> bits);
    }
    if (bits >= 16u) return c;
    const bool neg = c < 0;
    const int32_t m = neg ? -c : c;
    int32_t u;
    if (m == 0) u = 0;
    else if (m >= (int32_t)((1u << (bits - 1u)) - 1u)) u = 0x7FFF;
    else u = (int32_t)((((uint32_t)m << 15) + 0x4000u) >> (bits - 1u));
    return neg ? -u : u;
}

__device__ __forceinline__ uint16_t bc6_finish(int32_t v, bool sgn) {
    if (!sgn) return (uint16_t)((v * 31) >> 6);
    if (v < 0) {
        const int32_t m = ((-v) * 31) >> 5;
        return (uint16_t)(m ? (m | 0x8000) : 0);
    }
    return (uint16_t)((v * 31) >> 5);
}

// Field F of a mode's header, from its tokens (all at known positions).
template <int MI, int F, int T = 0>
__device__ __forceinline__ uint32_t bc6_field(const uint4& q) {
    if constexpr (T >= kBc6Count[MI][F]) {
        return 0u;
    } else {
        constexpr uint32_t tok = kBc6Tok[MI][F][T];
        constexpr int n = (int)((tok >> 11) & 15u) + 1;
        uint32_t v = block_bits<(int)(tok & 127u), n>(q);
        if constexpr ((tok >> 15) != 0) v = __brev(v) >> (32 - n);
        return (v << ((tok >> 7) & 15u)) | bc6_field<MI, F, T + 1>(q);
    }
}

// Channel C of end point E, unquantised to 16 bits.
template <int MI, int E, int C>
__device__ __forceinline__ uint32_t bc6_end(const uint4& q, uint32_t base, bool sgn) {
    constexpr uint32_t bits = kBc6Mode[MI][1], delta = kBc6Mode[MI][2 + C];
    uint32_t v = E == 0 ? base : bc6_field<MI, E * 3 + C>(q);
    if constexpr (E > 0 && kBc6Mode[MI][0] != 0)  // a signed delta to the base end point
        v = (base + (uint32_t)bc6_sext(v, delta)) & ((1u << bits) - 1u);
    return (uint32_t)bc6_unquantize(sgn ? bc6_sext(v, bits) : (int32_t)v, bits, sgn) & 0xFFFFu;
}

// The end points of one block of mode row MI: word 3 k + c holds region k's
// pair of channel c, six words in all.
template <int MI>
__device__ __forceinline__ void bc6_header(const uint4& q, bool sgn, uint32_t* out, uint32_t pitch) {
    const uint32_t b0 = bc6_field<MI, 0>(q), b1 = bc6_field<MI, 1>(q), b2 = bc6_field<MI, 2>(q);
    out[0 * pitch] = bc6_end<MI, 0, 0>(q, b0, sgn) | (bc6_end<MI, 1, 0>(q, b0, sgn) << 16);
    out[1 * pitch] = bc6_end<MI, 0, 1>(q, b1, sgn) | (bc6_end<MI, 1, 1>(q, b1, sgn) << 16);
    out[2 * pitch] = bc6_end<MI, 0, 2>(q, b2, sgn) | (bc6_end<MI, 1, 2>(q, b2, sgn) << 16);
    if constexpr (kBc6Mode[MI][5] == 2) {
        out[3 * pitch] = bc6_end<MI, 2, 0>(q, b0, sgn) | (bc6_end<MI, 3, 0>(q, b0, sgn) << 16);
        out[4 * pitch] = bc6_end<MI, 2, 1>(q, b1, sgn) | (bc6_end<MI, 3, 1>(q, b1, sgn) << 16);
        out[5 * pitch] = bc6_end<MI, 2, 2>(q, b2, sgn) | (bc6_end<MI, 3, 2>(q, b2, sgn) << 16);
    }
}

// The mode row of a 5-bit mode field (one whose two low bits are 0 or 1 is a
// 2-bit mode), 14 for a reserved mode: rows in kBc6Mode's order.
__device__ __forceinline__ uint32_t bc6_mode_row(uint32_t f) {
    const uint32_t two = f & 3u, k = f >> 2;
    if (two < 2u) return two;
    if (two == 2u) return 2u + k;        // 0x02, 0x06, .. 0x1E
    return k < 4u ? 10u + k : 14u;       // 0x03, 0x07, 0x0B, 0x0F; then reserved
}

// One texel channel from its weight, 64 e0 + 32 and e1 - e0.
template <bool SGN>
__device__ __forceinline__ float bc6_channel(int32_t w, int32_t base, int32_t diff) {
    // ((64 - w) e0 + w e1 + 32) >> 6, arithmetic: floor division
    return __half2float(__ushort_as_half(bc6_finish((base + w * diff) >> 6, SGN)));
}

// BC6H: a CTA decodes 32 x 8 blocks, one thread each.  The headers, fourteen
// layouts, are parsed in an order sorted by mode (a warp then runs two or
// three parses instead of up to fourteen) and handed to the blocks' own
// threads through shared memory as unquantised end points; the texels are
// decoded in image order, so that a warp's row of 128 texels leaves as one
// contiguous 1,536-byte store.  8192^2: 1,060 -> 232 us (UF16) and 1,158 -> 304
// us (SF16); 2050 x 1023, whose rows are 8-byte aligned: 67.7 -> 13.3 us (four
// lanes per block each parsed the header from a token table and stored their
// 48 bytes of a row themselves).
template <bool SGN>
__global__ void __launch_bounds__(32 * kDecodeRows) k_decode_bc6h(const uint8_t* __restrict__ blocks, uint32_t w,
                                                                  uint32_t h, float* __restrict__ rgb) {
    constexpr uint32_t kBlocks = 32 * kDecodeRows;
    __shared__ uint32_t s_count[15];
    __shared__ uint16_t s_list[kBlocks];
    __shared__ __align__(16) uint4 s_block[kBlocks];
    __shared__ uint32_t s_end[6][kBlocks];
    __shared__ __align__(16) uint32_t s_row[kDecodeRows][384];
    __shared__ uint16_t s_p2[32];
    __shared__ uint8_t s_a2[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid < 15) s_count[tid] = 0;
    if (tid < 32) {
        s_p2[tid] = g_bc7_p2[tid];
        s_a2[tid] = g_bc7_a2[tid];
    }
    pdl_begin();
    __syncthreads();
    const uint32_t bw = (w + 3) / 4, bh = (h + 3) / 4;
    const uint32_t bx0 = blockIdx.x * 32, bx = bx0 + lane, by = blockIdx.y * kDecodeRows + warp;
    const bool live = bx < bw && by < bh;
    uint4 q = make_uint4(0x13u, 0u, 0u, 0u);  // past the image: a reserved mode
    if (live) q = __ldg(reinterpret_cast<const uint4*>(blocks) + ((size_t)by * bw + bx));
    s_block[tid] = q;
    const uint32_t row = bc6_mode_row(q.x & 31u);
    const unsigned same = __match_any_sync(0xffffffffu, row);
    const int leader = __ffs((int)same) - 1;
    uint32_t rank = 0;
    if ((int)lane == leader) rank = atomicAdd(&s_count[row], (uint32_t)__popc(same));
    rank = __shfl_sync(0xffffffffu, rank, leader) + (uint32_t)__popc(same & ((1u << lane) - 1u));
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (uint32_t m = 0; m < 14; ++m) before += m < row ? s_count[m] : 0u;
    s_list[before + rank] = (uint16_t)tid;
    __syncthreads();
    {
        const uint32_t i = s_list[tid];
        const uint4 p = s_block[i];
        uint32_t* e = &s_end[0][i];
        switch (bc6_mode_row(p.x & 31u)) {
            case 0: bc6_header<0>(p, SGN, e, kBlocks); break;
            case 1: bc6_header<1>(p, SGN, e, kBlocks); break;
            case 2: bc6_header<2>(p, SGN, e, kBlocks); break;
            case 3: bc6_header<3>(p, SGN, e, kBlocks); break;
            case 4: bc6_header<4>(p, SGN, e, kBlocks); break;
            case 5: bc6_header<5>(p, SGN, e, kBlocks); break;
            case 6: bc6_header<6>(p, SGN, e, kBlocks); break;
            case 7: bc6_header<7>(p, SGN, e, kBlocks); break;
            case 8: bc6_header<8>(p, SGN, e, kBlocks); break;
            case 9: bc6_header<9>(p, SGN, e, kBlocks); break;
            case 10: bc6_header<10>(p, SGN, e, kBlocks); break;
            case 11: bc6_header<11>(p, SGN, e, kBlocks); break;
            case 12: bc6_header<12>(p, SGN, e, kBlocks); break;
            case 13: bc6_header<13>(p, SGN, e, kBlocks); break;
            default:
                for (int k = 0; k < 6; ++k) e[k * kBlocks] = 0u;
        }
    }
    __syncthreads();
    if (by >= bh) return;  // whole warps
    // two regions, but for the modes whose two low bits are set
    const bool two = (q.x & 3u) != 3u;
    int32_t base[2][3], diff[2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const uint32_t e = k == 0 || two ? s_end[3 * k + c][tid] : 0u;
            const int32_t e0 = SGN ? (int32_t)(int16_t)(e & 0xFFFFu) : (int32_t)(e & 0xFFFFu);
            const int32_t e1 = SGN ? (int32_t)(int16_t)(e >> 16) : (int32_t)(e >> 16);
            base[k][c] = 64 * e0 + 32;
            diff[k][c] = e1 - e0;
        }
    // the index stream at a fixed width a texel: the anchors' missing bits
    // inserted (two regions: 3 bits a texel from bit 82; one: 4 from bit 65)
    const uint32_t part = block_bits<77, 5>(q);
    const uint32_t pmask = two ? s_p2[part] : 0u;
    const uint32_t ib = two ? 3u : 4u;
    uint64_t ix = insert_zero(two ? block_tail<82>(q) : block_tail<65>(q), ib - 1u);
    if (two) ix = insert_zero(ix, s_a2[part] * 3u + 2u);
    const uint32_t words = 3u * min(128u, w - 4 * bx0);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint32_t y = by * 4 + r;
        if (y >= h) break;
        uint32_t v[12];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = 4 * r + x;
            const uint32_t idx = (uint32_t)ix & (two ? 7u : 15u);
            ix >>= ib;
            const int32_t wt = (int32_t)(two ? index_weight<3>(idx) : index_weight<4>(idx));
            const bool s = (pmask >> i) & 1u;
#pragma unroll
            for (int c = 0; c < 3; ++c)
                v[3 * x + c] = __float_as_uint(
                    bc6_channel<SGN>(wt, s ? base[1][c] : base[0][c], s ? diff[1][c] : diff[0][c]));
        }
        store_rows<12>(v, s_row[warp], lane,
                       reinterpret_cast<uint32_t*>(rgb) + ((size_t)y * w + (size_t)bx0 * 4) * 3, words);
    }
}

// ------------------------------------------------------------------- JPEG
// The device half of a JPEG decode (the host half, jpeg.cpp, writes the
// dequantized coefficient planes).  Pinned fixed-point arithmetic, shared
// with the oracle:
//   IDCT: K[x][u] = round(8192 * c(u) / 2 * cos((2x + 1) u pi / 16)),
//     c(0) = 1 / sqrt(2), c(u > 0) = 1; rows t[v][x] = (sum_u K[x][u] F[v][u]
//     + 512) >> 10 (int32, 3 fractional bits kept), then columns
//     s[y][x] = (sum_v K[y][v] t[v][x] + 2^15) >> 16 (int64), + 128, clamped
//     to 0..255; right shifts are arithmetic.
//   upsampling: component c at pixel (x, y) is its sample
//     (x / (hmax / h_c), y / (vmax / v_c)) (replication).
//   YCbCr -> RGB (JFIF): with cb = Cb - 128, cr = Cr - 128,
//     R = Y + ((91881 cr + 32768) >> 16),
//     G = Y + ((-22554 cb - 46802 cr + 32768) >> 16),
//     B = Y + ((116130 cb + 32768) >> 16), each clamped to 0..255.

__constant__ int32_t c_idct[8][8] = {
    {2896, 4017, 3784, 3406, 2896, 2276, 1567, 799},     {2896, 3406, 1567, -799, -2896, -4017, -3784, -2276},
    {2896, 2276, -1567, -4017, -2896, 799, 3784, 3406},  {2896, 799, -3784, -2276, 2896, 3406, -1567, -4017},
    {2896, -799, -3784, 2276, 2896, -3406, -1567, 4017}, {2896, -2276, -1567, 4017, -2896, -799, 3784, -3406},
    {2896, -3406, 1567, 799, -2896, 4017, -3784, 2276},  {2896, -4017, 3784, -3406, 2896, -2276, 1567, -799},
};

constexpr int kIdctBlocks = 32;  // 8x8 blocks per CTA, one thread per block row

// Coefficient blocks (raster order over a blocks_w-wide grid) -> 8-bit
// samples of a (blocks_w * 8)-wide plane.
__global__ void __launch_bounds__(kIdctBlocks * 8) k_jpeg_idct(const int16_t* __restrict__ coef, uint32_t blocks,
                                                               uint32_t blocks_w, uint8_t* __restrict__ plane) {
    pdl_begin();
    __shared__ int32_t t[kIdctBlocks][8][9];
    const uint32_t local = threadIdx.x >> 3, r = threadIdx.x & 7u;
    const uint32_t b = blockIdx.x * kIdctBlocks + local;
    const bool live = b < blocks;
    if (live) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(coef + (size_t)b * 64 + r * 8));
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        int32_t f[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = int32_t(int16_t(w[i] & 0xFFFFu));
            f[2 * i + 1] = int32_t(int16_t(w[i] >> 16));
        }
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            int32_t acc = 0;
#pragma unroll
            for (int u = 0; u < 8; ++u) acc += c_idct[x][u] * f[u];
            t[local][r][x] = (acc + 512) >> 10;
        }
    }
    __syncthreads();
    if (!live) return;
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        int64_t acc = 0;
#pragma unroll
        for (int v = 0; v < 8; ++v) acc += int64_t(c_idct[r][v]) * t[local][v][x];
        const int32_t s = min(255, max(0, int32_t((acc + 32768) >> 16) + 128));
        if (x < 4) lo |= uint32_t(s) << (8 * x);
        else hi |= uint32_t(s) << (8 * (x - 4));
    }
    const uint32_t bx = b % blocks_w, by = b / blocks_w;
    *reinterpret_cast<uint2*>(plane + ((size_t)by * 8 + r) * ((size_t)blocks_w * 8) + (size_t)bx * 8) = make_uint2(lo, hi);
}

__global__ void __launch_bounds__(256) k_jpeg_color(JpegPlanes P, uint32_t* __restrict__ rgba) {
    pdl_begin();
    const uint32_t x = blockIdx.x * 32 + (threadIdx.x & 31u), y = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (x >= P.width || y >= P.height) return;
    int32_t c[3] = {0, 0, 0};
#pragma unroll
    for (uint32_t k = 0; k < 3; ++k)  // constant indices keep the parameters out of local memory
        if (k < P.components) c[k] = P.plane[k][(size_t)(y / P.ry[k]) * P.pitch[k] + x / P.rx[k]];
    uint32_t r, g, b;
    if (P.components == 1) {
        r = g = b = uint32_t(c[0]);
    } else if (P.rgb) {
        r = uint32_t(c[0]);
        g = uint32_t(c[1]);
        b = uint32_t(c[2]);
    } else {
        const int32_t cb = c[1] - 128, cr = c[2] - 128;
        r = uint32_t(min(255, max(0, c[0] + ((91881 * cr + 32768) >> 16))));
        g = uint32_t(min(255, max(0, c[0] + ((-22554 * cb - 46802 * cr + 32768) >> 16))));
        b = uint32_t(min(255, max(0, c[0] + ((116130 * cb + 32768) >> 16))));
    }
    rgba[(size_t)y * P.width + x] = r | (g << 8) | (b << 16) | 0xFF000000u;
}

}  // namespace

void launch_jpeg_idct(const int16_t* coef, uint32_t blocks_w, uint32_t blocks_h, uint8_t* plane, cudaStream_t stream) {
    const uint32_t blocks = blocks_w * blocks_h;
    launch_pdl(k_jpeg_idct, dim3((blocks + kIdctBlocks - 1) / kIdctBlocks), dim3(kIdctBlocks * 8), 0, stream, coef,
               blocks, blocks_w, plane);
}

void launch_jpeg_color(const JpegPlanes& P, uint32_t* rgba, cudaStream_t stream) {
    launch_pdl(k_jpeg_color, dim3((P.width + 31) / 32, (P.height + 7) / 8), dim3(256), 0, stream, P, rgba);
}

void launch_decode_bc6h(const uint8_t* blocks, bool is_signed, uint32_t w, uint32_t h, float* rgb,
                        cudaStream_t stream) {
    const uint32_t bw = (w + 3) / 4, bh = (h + 3) / 4;
    const dim3 grid((bw + 31) / 32, (bh + kDecodeRows - 1) / kDecodeRows), block(32 * kDecodeRows);
    if (is_signed)
        launch_pdl(k_decode_bc6h<true>, grid, block, 0, stream, blocks, w, h, rgb);
    else
        launch_pdl(k_decode_bc6h<false>, grid, block, 0, stream, blocks, w, h, rgb);
}

void launch_decode_bc(const uint8_t* blocks, uint32_t format, uint32_t w, uint32_t h, uint32_t* rgba,
                      cudaStream_t stream) {
    const uint32_t bw = (w + 3) / 4, bh = (h + 3) / 4;
    if (format == VKGV_BC7) {
        // tiles 128 blocks wide, narrower ones for narrower images
        const uint32_t tw_log2 = bw <= 32 ? 5u : (bw <= 64 ? 6u : 7u);
        const uint32_t th = kBc7Blocks >> tw_log2;
        const dim3 grid((bw + (1u << tw_log2) - 1) >> tw_log2, (bh + th - 1) / th);
        launch_pdl(k_decode_bc7, grid, dim3(kBc7Threads), 0, stream, blocks, w, h, tw_log2, rgba);
        return;
    }
    const dim3 grid((bw + 31) / 32, (bh + kDecodeRows - 1) / kDecodeRows), block(32 * kDecodeRows);
    switch (format) {
        case VKGV_BC1: launch_pdl(k_decode_bc<VKGV_BC1>, grid, block, 0, stream, blocks, w, h, rgba); break;
        case VKGV_BC2: launch_pdl(k_decode_bc<VKGV_BC2>, grid, block, 0, stream, blocks, w, h, rgba); break;
        case VKGV_BC3: launch_pdl(k_decode_bc<VKGV_BC3>, grid, block, 0, stream, blocks, w, h, rgba); break;
        case VKGV_BC4: launch_pdl(k_decode_bc<VKGV_BC4>, grid, block, 0, stream, blocks, w, h, rgba); break;
        case VKGV_BC5: launch_pdl(k_decode_bc<VKGV_BC5>, grid, block, 0, stream, blocks, w, h, rgba); break;
        default: launch_pdl(k_decode_bc<VKGV_BC1_OPAQUE>, grid, block, 0, stream, blocks, w, h, rgba); break;
    }
}

}  // namespace vkgv
