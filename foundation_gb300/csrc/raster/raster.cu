// raster.cu — the reference renderer's raster pass as CUDA kernels (see
// raster.hpp for the rules).
//
//  setup_kernel   per triangle: its vertices' clip = proj (view (model
//                 (x, y, 0, 1))), the matrix products in FP32 with sums taken
//                 left to right (Triangle.slang:23-31 computes mul(proj,
//                 mul(view, model))), perspective divide, viewport transform
//                 (Vulkan: y grows downwards), vertex snap to 1/256 pixel,
//                 signed area (front face counter-clockwise: Vulkan's
//                 a = -1/2 sum(x_i y_{i+1} - x_{i+1} y_i) > 0), culling,
//                 edge orientation and top-left flags, pixel bounding box
//  pixel_kernel   per pixel: coverage of every triangle (no depth test: the
//                 last covering triangle in index order wins), perspective-
//                 correct barycentrics, bilinear texel fetch with repeat
//                 addressing, colour = texel * (vertex colour, 1), UNORM
//                 encoding round(clamp(c, 0, 1) * 255)
// Triangles with a vertex at w <= 0 (behind the eye) or outside a +-2^20
// pixel guard band are skipped rather than clipped.
//
// A byte is defined by FP64 arithmetic (shade_exact), about 400 operations and
// 27 divisions a pixel at a rate of two a clock and SM: 177 us for the
// reference quad at 1920x1080. But the byte is floor(v + 1/2) of a continuous
// function, so a pixel first takes v to about 2e-4 (texture coordinates in
// FP64, the rest in FP32: 23 FP64 operations) and is done unless a channel
// lies within the error bound of a rounding boundary; then it takes v in FP64
// (to 1e-7, or what the coordinates allow), and only if that too cannot tell it
// evaluates the definition.
// The same frame then takes 26 us, and the whole draw (1 MB texture copied in)
// 47 us instead of 169.
#include "raster.hpp"

#include <cstdint>

namespace Foundation {
namespace Raster {
namespace {

constexpr int kSub = 256;  // sub-pixel steps per pixel
constexpr double kUvOne = 1099511627776.0;  // 2^40: fixed-point texture coordinates
// Error bounds (see shade): of a code per unit of colour, without the texture
// coordinates' errors, and of a coordinate relative to the triangle's largest.
constexpr double kEps1 = 2.5e-4, kEps2 = 1e-7, kEpsUv = 2.5e-14;

struct alignas(16) Tri {
    int x0, y0, x1, y1;    // inclusive pixel bounds; x0 > x1 when the triangle is skipped
    long long e0[3];       // edge functions at the centre of pixel (0, 0), inside >= 0,
    long long sx[3], sy[3];  // and their steps per pixel
    uint32_t topleft;      // bit i: edge opposite vertex i is a top or left edge
    float eps1, eps2;      // error bounds of the two quick evaluations, in codes (see shade)
    // per vertex, over its w: texture coordinates times 2^40, 1, colours
    double cu[3], cv[3], iw[3], cd[3][3];
    float cf[3][3];
    // the definition's inputs
    long long A;           // twice the area (> 0)
    double w[3];           // clip w per vertex (after orientation)
    uint32_t vid[3];       // vertex ids (after orientation)
};

__device__ __forceinline__ float madd4(const float* a, const float* b, int r, int c) {
    // (A B)[r][c] with column-major storage m[col * 4 + row]
    float s = __fmul_rn(a[0 * 4 + r], b[c * 4 + 0]);
    s = __fadd_rn(s, __fmul_rn(a[1 * 4 + r], b[c * 4 + 1]));
    s = __fadd_rn(s, __fmul_rn(a[2 * 4 + r], b[c * 4 + 2]));
    return __fadd_rn(s, __fmul_rn(a[3 * 4 + r], b[c * 4 + 3]));
}

__device__ __forceinline__ long long edge(long long ax, long long ay, long long bx, long long by, long long px,
                                          long long py) {
    return (bx - ax) * (py - ay) - (by - ay) * (px - ax);
}

__device__ __forceinline__ void setup(const DrawArgs& A, const Vertex* verts, const uint16_t* idx, Tri* tris) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= A.ntri) return;
    float vm[16], pvm[16];
    for (int c = 0; c < 4; ++c)
        for (int r = 0; r < 4; ++r) vm[c * 4 + r] = madd4(A.u.view, A.u.model, r, c);
    for (int c = 0; c < 4; ++c)
        for (int r = 0; r < 4; ++r) pvm[c * 4 + r] = madd4(A.u.proj, vm, r, c);
    Tri T;
    T.x0 = 1;
    T.x1 = 0;
    T.y0 = T.y1 = 0;
    bool ok = true;
    long long X[3], Y[3];
    double w[3];
    uint32_t vid[3];
    for (int k = 0; k < 3; ++k) {
        vid[k] = idx[3 * (size_t)t + k];
        if (vid[k] >= A.nv) {  // (checked on the host)
            ok = false;
            break;
        }
        const float p[4] = {verts[vid[k]].pos[0], verts[vid[k]].pos[1], 0.0f, 1.0f};
        double c[4];
        for (int r = 0; r < 4; ++r) {
            float s = __fmul_rn(pvm[0 * 4 + r], p[0]);
            s = __fadd_rn(s, __fmul_rn(pvm[1 * 4 + r], p[1]));
            s = __fadd_rn(s, __fmul_rn(pvm[2 * 4 + r], p[2]));
            c[r] = __fadd_rn(s, __fmul_rn(pvm[3 * 4 + r], p[3]));
        }
        w[k] = c[3];
        if (!(c[3] > 0.0)) {
            ok = false;
            break;
        }
        const double xd = __ddiv_rn(c[0], c[3]), yd = __ddiv_rn(c[1], c[3]);
        const double xf = __dadd_rn(__dmul_rn(0.5 * (double)A.width, xd), 0.5 * (double)A.width);
        const double yf = __dadd_rn(__dmul_rn(0.5 * (double)A.height, yd), 0.5 * (double)A.height);
        if (!(fabs(xf) < 1048576.0 && fabs(yf) < 1048576.0)) {
            ok = false;
            break;
        }
        X[k] = __double2ll_rn(__dmul_rn(xf, (double)kSub));
        Y[k] = __double2ll_rn(__dmul_rn(yf, (double)kSub));
    }
    if (ok) {
        // 2x the shoelace area; Vulkan's a = -area, front-facing when a > 0
        const long long s2 = edge(X[0], Y[0], X[1], Y[1], X[2], Y[2]);
        const bool front = s2 < 0;
        if (s2 == 0 || (A.cull_back && !front)) ok = false;
        if (ok) {
            if (s2 < 0) {  // orient so the inside has positive edge functions
                long long tx = X[1], ty = Y[1];
                X[1] = X[2];
                Y[1] = Y[2];
                X[2] = tx;
                Y[2] = ty;
                const double tw = w[1];
                w[1] = w[2];
                w[2] = tw;
                const uint32_t tv = vid[1];
                vid[1] = vid[2];
                vid[2] = tv;
            }
            T.A = s2 < 0 ? -s2 : s2;
            T.topleft = 0;
            for (int k = 0; k < 3; ++k) {
                // edge opposite vertex k runs from vertex k+1 to vertex k+2
                const int a = (k + 1) % 3, b = (k + 2) % 3;
                const long long dx = X[b] - X[a], dy = Y[b] - Y[a];
                if ((dy == 0 && dx > 0) || dy < 0) T.topleft |= 1u << k;
            }
            long long mnx = X[0], mxx = X[0], mny = Y[0], mxy = Y[0];
            for (int k = 1; k < 3; ++k) {
                mnx = X[k] < mnx ? X[k] : mnx;
                mxx = X[k] > mxx ? X[k] : mxx;
                mny = Y[k] < mny ? Y[k] : mny;
                mxy = Y[k] > mxy ? Y[k] : mxy;
            }
            // pixel p is tested at p * 256 + 128
            long long px0 = (mnx - kSub / 2 + kSub - 1) / kSub, py0 = (mny - kSub / 2 + kSub - 1) / kSub;
            long long px1 = (mxx - kSub / 2) / kSub, py1 = (mxy - kSub / 2) / kSub;
            if (mnx - kSub / 2 < 0) px0 = 0;
            if (mny - kSub / 2 < 0) py0 = 0;
            if (mxx - kSub / 2 < 0) px1 = -1;
            if (mxy - kSub / 2 < 0) py1 = -1;
            px1 = px1 < (long long)A.width - 1 ? px1 : (long long)A.width - 1;
            py1 = py1 < (long long)A.height - 1 ? py1 : (long long)A.height - 1;
            T.x0 = (int)px0;
            T.y0 = (int)py0;
            T.x1 = (int)px1;
            T.y1 = (int)py1;
            float cm = 1.0f;
            for (int k = 0; k < 3; ++k) {
                T.w[k] = w[k];
                T.vid[k] = vid[k];
                const int a = (k + 1) % 3, b = (k + 2) % 3;
                T.e0[k] = edge(X[a], Y[a], X[b], Y[b], kSub / 2, kSub / 2);
                T.sx[k] = -(Y[b] - Y[a]) * kSub;
                T.sy[k] = (X[b] - X[a]) * kSub;
                const Vertex& V = verts[vid[k]];
                const double iw = 1.0 / w[k];
                T.iw[k] = iw;
                T.cu[k] = (double)V.uv[0] * iw * kUvOne;
                T.cv[k] = (double)V.uv[1] * iw * kUvOne;
                for (int c = 0; c < 3; ++c) {
                    T.cd[k][c] = (double)V.color[c] * iw;
                    T.cf[k][c] = (float)T.cd[k][c];
                    // an infinite or NaN colour makes the bound infinite: always the definition
                    cm = V.color[c] == V.color[c] ? fmaxf(cm, fabsf(V.color[c])) : __int_as_float(0x7F800000);
                }
            }
            // texture coordinates are floored to 2^-40 of a repeat and rounded in
            // proportion to the vertices' (kEpsUv), and a repeat of n texels
            // takes a channel through n slopes of at most 255 codes
            double coords = 0.0;
            for (int c = 0; c < 2; ++c) {
                const float *a = verts[vid[0]].uv, *b = verts[vid[1]].uv, *d = verts[vid[2]].uv;
                const double m = fmaxf(fabsf(a[c]), fmaxf(fabsf(b[c]), fabsf(d[c])));  // (a NaN's pixels fail anyway)
                coords += 255.0 * (double)(c ? A.tex_h : A.tex_w) * (1.0 / kUvOne + kEpsUv * m);
            }
            T.eps1 = __double2float_ru((double)cm * (kEps1 + coords));
            T.eps2 = __double2float_ru((double)cm * (kEps2 + coords));
        }
    }
    tris[t] = T;
}

__global__ void setup_kernel(const DrawArgs A, Tri* tris) { setup(A, A.verts, A.idx, tris); }
// The mesh as a kernel argument; pixel_kernel reads the vertices from memory.
__global__ void setup_small_kernel(const DrawArgs A, const __grid_constant__ SmallMesh mesh, Tri* tris) {
    if (blockIdx.x == 0)
        for (uint32_t i = threadIdx.x; i < A.nv; i += blockDim.x) A.verts[i] = mesh.verts[i];
    setup(A, mesh.verts, mesh.idx, tris);
}

__device__ __forceinline__ double unit_frac(double u) {
    if (!(u == u) || fabs(u) > 4.0e15) return 0.0;  // NaN / beyond exact fractions
    return __dsub_rn(u, floor(u));
}

__device__ __forceinline__ double texel(const DrawArgs& A, long long i, long long j, int ch) {
    const uint32_t v = A.texture[(size_t)j * A.tex_w + (size_t)i];
    return (double)((v >> (8 * ch)) & 0xFFu) / 255.0;
}

__device__ __forceinline__ uint32_t unorm8(double c) {
    c = c < 0.0 ? 0.0 : (c > 1.0 ? 1.0 : c);
    return (uint32_t)floor(__dadd_rn(__dmul_rn(c, 255.0), 0.5));
}

// The definition of a covered pixel's colour.
__device__ __noinline__ uint32_t shade_exact(const DrawArgs& A, const Tri& T, long long E0, long long E1, long long E2) {
    const long long E[3] = {E0, E1, E2};
    const double area = (double)T.A;
    double b[3];
    for (int k = 0; k < 3; ++k) b[k] = __ddiv_rn(__ddiv_rn((double)E[k], area), T.w[k]);
    const double s = __dadd_rn(__dadd_rn(b[0], b[1]), b[2]);
    double attr[5];  // u, v, r, g, b
    for (int q = 0; q < 5; ++q) {
        double acc = 0.0;
        for (int k = 0; k < 3; ++k) {
            const Vertex& V = A.verts[T.vid[k]];
            const double a = q < 2 ? (double)V.uv[q] : (double)V.color[q - 2];
            acc = k == 0 ? __dmul_rn(b[0], a) : __dadd_rn(acc, __dmul_rn(b[k], a));
        }
        attr[q] = __ddiv_rn(acc, s);
    }
    const double ut = __dsub_rn(__dmul_rn(unit_frac(attr[0]), (double)A.tex_w), 0.5);
    const double vt = __dsub_rn(__dmul_rn(unit_frac(attr[1]), (double)A.tex_h), 0.5);
    const double fu = floor(ut), fv = floor(vt);
    const double au = __dsub_rn(ut, fu), av = __dsub_rn(vt, fv);
    const long long W = A.tex_w, H = A.tex_h;
    const long long i0 = (((long long)fu % W) + W) % W, i1 = (i0 + 1) % W;
    const long long j0 = (((long long)fv % H) + H) % H, j1 = (j0 + 1) % H;
    const double w00 = __dmul_rn(__dsub_rn(1.0, au), __dsub_rn(1.0, av)), w10 = __dmul_rn(au, __dsub_rn(1.0, av));
    const double w01 = __dmul_rn(__dsub_rn(1.0, au), av), w11 = __dmul_rn(au, av);
    uint32_t out = 0;
    for (int ch = 0; ch < 4; ++ch) {
        double c = __dmul_rn(w00, texel(A, i0, j0, ch));
        c = __dadd_rn(c, __dmul_rn(w10, texel(A, i1, j0, ch)));
        c = __dadd_rn(c, __dmul_rn(w01, texel(A, i0, j1, ch)));
        c = __dadd_rn(c, __dmul_rn(w11, texel(A, i1, j1, ch)));
        out |= unorm8(ch < 3 ? __dmul_rn(c, attr[2 + ch]) : c) << (8 * ch);
    }
    return out;
}

// One channel's byte from v = 255 c with |error| <= eps; false when a rounding
// boundary lies that near. (Not finite, or eps not: false.)
template <typename T>
__device__ __forceinline__ bool settle(T v, T eps, uint32_t& byte) {
    const T x = (v < (T)0 ? (T)0 : v > (T)255 ? (T)255 : v) + (T)0.5;
    const T f = floor(x);
    byte = (uint32_t)f;
    return x - f > eps && x - f < (T)1 - eps;
}

// Fixed-point texture coordinate (2^40 per repeat) on n texels: the two texel
// indices and the weight of the second (2^40 per texel).
__device__ __forceinline__ void wrap(long long c, uint32_t n, uint32_t& i0, uint32_t& i1, unsigned long long& frac) {
    const unsigned long long one = 1ull << 40;
    const long long t = (long long)(((unsigned long long)c & (one - 1)) * n) - (long long)(one >> 1);
    const int i = (int)(t >> 40);  // -1 .. n - 1
    i0 = i < 0 ? n - 1u : (uint32_t)i;
    i1 = i0 + 1u == n ? 0u : i0 + 1u;
    frac = (unsigned long long)t & (one - 1);
}

// Colour of a covered pixel. Errors of the first try, relative to the largest
// colour x 255: colours 4.2e-7 (float edge functions, products, sums and
// reciprocal), two lerps of texels 1.6e-7, their product 1.2e-7: 1.8e-4 of a
// code, kEps1 2.5e-4. Second try, in FP64: colours and lerps below 1e-11, kEps2
// 1e-7. To both comes what the error of the texture coordinates can do (setup):
// 255 (w + h) 2^-40 of a code, 2.4e-7 for 512 texels a side, 7.6e-6 for 16,384,
// and their rounding, which scales with the vertices' coordinates where these
// cancel: 1 / D 128 units of 2^-53 (the square of the float reciprocal's 2^-23),
// the quick sums and quotients 12, the definition's 12: 1.7e-14, kEpsUv 2.5e-14.
__device__ __forceinline__ uint32_t shade(const DrawArgs& A, const Tri& T, const long long E[3]) {
    const double e[3] = {(double)E[0], (double)E[1], (double)E[2]};
    const double D = fma(e[2], T.iw[2], fma(e[1], T.iw[1], e[0] * T.iw[0]));
    const float Df = (float)D;
    if (Df > 1e-30f && Df < 1e30f && A.tex_w <= 16384u && A.tex_h <= 16384u) {
        // 1 / D by one Newton step from the float reciprocal: 1.4e-14
        const double r0 = (double)(1.0f / Df);
        const double r = fma(r0, fma(-D, r0, 1.0), r0);
        const double U = fma(e[2], T.cu[2], fma(e[1], T.cu[1], e[0] * T.cu[0])) * r;
        const double V = fma(e[2], T.cv[2], fma(e[1], T.cv[1], e[0] * T.cv[0])) * r;
        if (fabs(U) <= 1024.0 * kUvOne && fabs(V) <= 1024.0 * kUvOne) {
            uint32_t i0, i1, j0, j1;
            unsigned long long fu, fv;
            wrap(__double2ll_rd(U), A.tex_w, i0, i1, fu);
            wrap(__double2ll_rd(V), A.tex_h, j0, j1, fv);
            const uint32_t t00 = __ldg(A.texture + (size_t)j0 * A.tex_w + i0), t10 = __ldg(A.texture + (size_t)j0 * A.tex_w + i1);
            const uint32_t t01 = __ldg(A.texture + (size_t)j1 * A.tex_w + i0), t11 = __ldg(A.texture + (size_t)j1 * A.tex_w + i1);
            {
                const float au = (float)(uint32_t)(fu >> 8) * 2.3283064365386963e-10f;  // 2^-32
                const float av = (float)(uint32_t)(fv >> 8) * 2.3283064365386963e-10f;
                const float ef[3] = {(float)e[0], (float)e[1], (float)e[2]};
                const float rf = (float)r, eps = T.eps1;
                uint32_t out = 0;
                bool ok = true;
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    const float a = (float)(t00 >> 8 * ch & 255u), b = (float)(t10 >> 8 * ch & 255u);
                    const float c = (float)(t01 >> 8 * ch & 255u), d = (float)(t11 >> 8 * ch & 255u);
                    const float lo = fmaf(au, b - a, a), hi = fmaf(au, d - c, c);
                    float v = fmaf(av, hi - lo, lo);
                    if (ch < 3)
                        v *= fmaf(ef[2], T.cf[2][ch], fmaf(ef[1], T.cf[1][ch], ef[0] * T.cf[0][ch])) * rf;
                    uint32_t byte;
                    ok = settle(v, eps, byte) && ok;
                    out |= byte << 8 * ch;
                }
                if (ok) return out;
            }
            const double au = (double)(long long)fu * (1.0 / kUvOne), av = (double)(long long)fv * (1.0 / kUvOne);
            uint32_t out = 0;
            bool ok = true;
            for (int ch = 0; ch < 4; ++ch) {
                const double a = (double)(t00 >> 8 * ch & 255u), b = (double)(t10 >> 8 * ch & 255u);
                const double c = (double)(t01 >> 8 * ch & 255u), d = (double)(t11 >> 8 * ch & 255u);
                const double lo = fma(au, b - a, a), hi = fma(au, d - c, c);
                double v = fma(av, hi - lo, lo);
                if (ch < 3) v *= fma(e[2], T.cd[2][ch], fma(e[1], T.cd[1][ch], e[0] * T.cd[0][ch])) * r;
                uint32_t byte;
                ok = settle(v, (double)T.eps2, byte) && ok;
                out |= byte << 8 * ch;
            }
            if (ok) return out;
        }
    }
    return shade_exact(A, T, E[0], E[1], E[2]);
}

// Four neighbouring pixels of a row per thread; the triangles from the last to
// the first, until all four are covered.
constexpr int kPixels = 4;

__global__ void __launch_bounds__(128) pixel_kernel(const DrawArgs A, const Tri* __restrict__ tris, bool wide) {
    const uint32_t x = (blockIdx.x * blockDim.x + threadIdx.x) * kPixels, y = blockIdx.y;
    if (x >= A.width) return;
    uint32_t open = (1u << min((uint32_t)kPixels, A.width - x)) - 1u;
    const uint32_t here = open;
    uint32_t out[kPixels] = {A.clear_rgba, A.clear_rgba, A.clear_rgba, A.clear_rgba};
    for (uint32_t t = A.ntri; t-- > 0u && open;) {
        const Tri& T = tris[t];
        const int4 box = *reinterpret_cast<const int4*>(&T);
        if ((int)y < box.y || (int)y > box.w || (int)x + kPixels - 1 < box.x || (int)x > box.z) continue;
        long long e[3], least[3];
        for (int k = 0; k < 3; ++k) {
            e[k] = T.e0[k] + T.sx[k] * (long long)x + T.sy[k] * (long long)y;
            least[k] = (T.topleft >> k & 1u) ? 0 : 1;
        }
#pragma unroll
        for (int q = 0; q < kPixels; ++q) {
            if ((open >> q & 1u) && (int)x + q >= box.x && (int)x + q <= box.z && e[0] >= least[0] &&
                e[1] >= least[1] && e[2] >= least[2]) {
                out[q] = shade(A, T, e);
                open &= ~(1u << q);
            }
            for (int k = 0; k < 3; ++k) e[k] += T.sx[k];
        }
    }
    uint32_t* to = A.target + (size_t)y * A.width + x;
    if (wide) {  // rows start on 16 bytes
        *reinterpret_cast<uint4*>(to) = make_uint4(out[0], out[1], out[2], out[3]);
    } else {
#pragma unroll
        for (int q = 0; q < kPixels; ++q)
            if (here >> q & 1u) to[q] = out[q];
    }
}

}  // namespace

size_t TriBytes(uint32_t ntri) { return sizeof(Tri) * (size_t)ntri; }

cudaError_t LaunchDraw(const DrawArgs& a, cudaStream_t s) {
    Tri* tris = static_cast<Tri*>(a.tris);
    const dim3 grid((a.ntri + 63) / 64);
    if (a.ntri && a.mesh)
        setup_small_kernel<<<grid, 64, 0, s>>>(a, *a.mesh, tris);
    else if (a.ntri)
        setup_kernel<<<grid, 64, 0, s>>>(a, tris);
    const bool wide = a.width % kPixels == 0 && ((uintptr_t)a.target & 15u) == 0;
    const uint32_t per_block = 128 * kPixels;
    pixel_kernel<<<dim3((a.width + per_block - 1) / per_block, a.height), 128, 0, s>>>(a, tris, wide);
    return cudaGetLastError();
}

}  // namespace Raster
}  // namespace Foundation
