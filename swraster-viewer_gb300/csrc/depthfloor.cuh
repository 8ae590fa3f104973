// Depth floor of a triangle, for the raster's occlusion culling: a lower bound
// of every depth the raster's own arithmetic can produce for a covered lane.
// The same source compiles for the device and for the host, so the bound can
// be checked on a CPU against an exhaustive walk of the triangle's packets.
//
// The raster's depth is z = zi * (1 / oi) with zi, oi the interpolants of
// z/w and 1/w at computed barycentrics b1, b2. With u = 2^-24:
//  - edge values: the origin evaluation (a x + b y) + c errs by at most
//    u (3 |a| X + 3 |b| Y + 2 |c|), X and Y the largest sample or vertex
//    coordinates and |c| <= |a| X + |b| Y + 1; the at most 16 additions after
//    it pass through values of the edge function at samples within 64
//    subpixels of the bounding box (extents ex, ey), at most
//    |a| (ex + 64) + |b| (ey + 64) plus the errors so far. Over the three
//    edges the |a| sum to 2 ey and the |b| to 2 ex: together at most
//    u (10 m + 6 + 64 ex ey + 2048 (ex + ey)), m = ey X + ex Y. A covered lane
//    has all three computed edge values >= 0 and the exact values sum to the
//    doubled area A plus top-left biases (<= 0), so b1, b2 >= 0 and
//    b1 + b2 <= B = (1 + (sum of the three errors) / A)(1 + u)^3;
//  - zi and oi are three-term sums, within 5u (|Z0| + B |D1| + B |D2|) (with
//    1/w's O0, P1, P2 likewise) of the exact affine values;
//  - those are a convex combination of the corners (rounded differences
//    from vertex 0, so up to 4u relative the vertices' values), plus at most
//    (B - 1) (|D1| + |D2|) beyond the far edge.
// So EZ = (B - 1) (|D1| + |D2|) + 16u (|Z0| + |D1| + |D2|) and EO likewise
// bound what numerator and denominator are off from a point of the triangle,
// and (Z - EZ) / (O +- EO), a ratio of affine functions with a positive
// denominator, is smallest at a corner. At the corner of depth z and w
//    (Z - EZ) / (O +- EO) >= z - (EZ + |z| EO) w / (1 - EO w) - 16u |z|.
// All error terms are positive sums and products; a factor 1 + 2^-8 covers
// their own rounding. The bound takes at most one division (with directed
// rounding at the corners of the widened triangle it took six, 20 us of a 4K
// frame).
// No floor is taken (false) when the int32 setup arithmetic could have wrapped
// or a coordinate is beyond f32's integers, when EO is over 0.9 of a corner's
// 1/w, for non-finite inputs, or when B would exceed 1.25.
#pragma once

#include <cfloat>
#include <cmath>
#include <cstdint>

namespace swr {

constexpr float kUlp24 = 5.9604645e-8f;  // 2^-24

// Triangle of subpixel vertices p (x0, y0, x1, y1, x2, y2) with doubled area
// `area` (int32, wrapped; front faces are negative), depth and 1/w
// interpolants zow and oow (value at vertex 0, then differences to vertices
// 1 and 2), vertex depths z and w (within 4 ulp), and sample coordinates below xe + 32 and ye + 32 (subpixels).
__host__ __device__ inline bool depth_floor(const int32_t p[6], int32_t area, const float zow[3], const float oow[3],
                                            const float z[3], const float w[3], int32_t xe, int32_t ye, float& zlo) {
    const float x0 = (float)p[0], y0 = (float)p[1], x1 = (float)p[2], y1 = (float)p[3], x2 = (float)p[4], y2 = (float)p[5];
    const float lx = fminf(fminf(x0, x1), x2), hx = fmaxf(fmaxf(x0, x1), x2);
    const float ly = fminf(fminf(y0, y1), y2), hy = fmaxf(fmaxf(y0, y1), y2);
    const float X = fmaxf(fmaxf(fabsf(lx), fabsf(hx)), (float)(xe + 32));
    const float Y = fmaxf(fmaxf(fabsf(ly), fabsf(hy)), (float)(ye + 32));
    const float ex = hx - lx, ey = hy - ly;
    // Coordinates exact in f32; a X + b Y <= m and |c| <= m + 1 within int32,
    // the doubled area (at most ex ey) too.
    const float m = ey * X + ex * Y;
    if (!(X < 1.6e7f && Y < 1.6e7f && ex < 1.6e7f && ey < 1.6e7f && m < 2.0e9f && ex * ey < 1.0e9f) || area >= 0)
        return false;
    // Where no term of an edge reaches 2^24, its values are exact integers.
    const bool exact = (2.0f * m + 2.0f) + 256.0f * (ex + ey) < 1.6e7f;
    const float rel =
        exact ? 0.0f : kUlp24 * ((12.0f * m + 12.0f) + (72.0f * ex * ey + 2400.0f * (ex + ey))) / -(float)area;
    if (!(rel < 0.24f)) return false;
    const float dz = fabsf(zow[1]) + fabsf(zow[2]), dw = fabsf(oow[1]) + fabsf(oow[2]);
    constexpr float kU = 20.0f * kUlp24, kSlack = 1.00390625f;
    const float EZ = ((rel + kU) * dz + kU * fabsf(zow[0])) * kSlack + 1e-30f;
    const float EO = ((rel + kU) * dw + kU * fabsf(oow[0])) * kSlack + 1e-30f;
    zlo = INFINITY;
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        const float r = EO * w[v];
        if (!(r < 0.9f) || !(w[v] > 0.0f)) return false;  // false for NaN too
        const float f = r < 0.01f ? 1.02f : (r < 0.5f ? 2.02f : 10.1f);  // above 1 / (1 - r)
        const float az = fabsf(z[v]);
        const float err = (EZ + az * EO) * (w[v] * f) + (16.0f * kUlp24) * az;
        const float lo = z[v] - (err * kSlack + 1e-30f);
        if (!(lo - lo == 0.0f)) return false;  // not finite
        zlo = fminf(zlo, lo);
    }
    return true;
}

}  // namespace swr
