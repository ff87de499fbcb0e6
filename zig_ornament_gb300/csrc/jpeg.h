// jpeg.h — sequential (baseline / extended Huffman) JPEG parsing and entropy
// decoding on the host (jpeg.cpp); the GPU stage (jpeg.cu) dequantises,
// inverse-transforms, upsamples and colour-converts the coefficients.
//
// This is the texture path of the reference's example app: textures are
// loaded with zstbi (stb_image) as 4-component images, flipped vertically
// (glfw_example/examples.zig:492-503 loadTexture; app_no_interop.zig:17
// setFlipVerticallyOnLoad(true)) and handed to Scene.createTexture
// (src/scene.zig:339-351).
#pragma once

#include <stdint.h>

#include <memory>
#include <string>
#include <vector>

namespace orn {
namespace jpeg {

constexpr int kMaxComponents = 3;

struct Component {
    uint32_t id = 0;
    uint32_t h = 1, v = 1;       // sampling factors
    uint32_t tq = 0;             // quantisation table
    uint32_t bw = 0, bh = 0;     // coefficient plane in 8x8 blocks (MCU-padded)
    bool decoded = false;
    size_t first_block = 0;      // of the plane in Image::blocks, [bh][bw]
};

// A block's nonzero coefficients: entries [start, start + count) of
// Image::entries (a photograph has some six in 64: the planes written out
// would be ten times the size, on the host, on the way and on the GPU).
struct Block {
    uint32_t start;
    uint32_t count;
};
// natural (row-major) index << 16 | value as 16 bits, not dequantised
inline uint32_t entry_of(int index, int value) { return ((uint32_t)index << 16) | (uint16_t)(int16_t)value; }

struct Image {
    uint32_t width = 0, height = 0, ncomp = 0;
    uint32_t hmax = 1, vmax = 1;
    uint32_t mcux = 0, mcuy = 0;
    bool ycbcr = true;           // false: the three components are R, G, B
    Component comp[kMaxComponents];
    uint16_t quant[4][64] = {};  // natural order
    bool quant_present[4] = {};
    std::vector<Block> blocks;   // all components' planes, one after another
    std::unique_ptr<uint32_t[]> entries;
    size_t entry_count = 0, entry_room = 0;
};

// Status codes are the library's ORN_* values.  With header_only the scan
// data is not decoded (width, height and components only).
int parse(const uint8_t* data, size_t len, bool header_only, Image* out, std::string* err);

// The calling thread's last error message of the orn_jpeg_* entry points.
std::string& last_error();

}  // namespace jpeg
}  // namespace orn
