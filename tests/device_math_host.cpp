// Host build of shading helpers for tests/test_device_math.py.
#include "host_shims.h"

#include "wf_traverse.cuh"

using namespace wf;

// sincos() against sin() and cos(): the number of arguments whose bits differ.
extern "C" uint64_t sincos_differences(const double* x, uint64_t count) {
    uint64_t differ = 0;
    for (uint64_t i = 0; i < count; ++i) {
        double s, c, s0 = wfm::sin(x[i]), c0 = wfm::cos(x[i]);
        wfm::sincos(x[i], s, c);
        bool nan = s0 != s0;
        differ += nan ? (s == s || c == c) : (std::memcmp(&s, &s0, 8) != 0 || std::memcmp(&c, &c0, 8) != 0);
    }
    return differ;
}

// texture_fetch of a w x h texture whose texel values are given, at count
// (u, v) points.
extern "C" void fetch_texture(const unsigned char* rgba, uint32_t w, uint32_t h, const float* uv, uint64_t count,
                              float* out) {
    DeviceScene s{};
    uint4 info = make_uint4(w, h, 0, 0);
    s.textures = &info;
    s.texels = reinterpret_cast<const uchar4*>(rgba);
    s.texture_count = 1;
    for (uint64_t i = 0; i < count; ++i) {
        float4 r = texture_fetch(s, 0, uv[2 * i], uv[2 * i + 1]);
        std::memcpy(out + 4 * i, &r, 16);
    }
}

// tile_pixel of every k of a w x h tile.
extern "C" void tile_pixels(uint32_t w, uint32_t h, uint32_t* xy) {
    for (uint32_t k = 0; k < w * h; ++k) {
        uint2 at = tile_pixel(k, w, h);
        xy[2 * k] = at.x;
        xy[2 * k + 1] = at.y;
    }
}
