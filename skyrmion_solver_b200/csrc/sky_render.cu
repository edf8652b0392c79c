// Headless volume path: the reference viewer's RGBA volume and its ray-marched
// image, computed on the device into plain buffers (no graphics API).
//
//  * Volume (build_rgba_volume_kernel, th/nuclear_skyrme/render_gl.py:157-222,
//    with the density extrema of its _reduce_density_extrema, :455-500):
//    channel 0 = (e - min e) / (max e - min e + 1e-30), channels 1..3 = the unit
//    pion vector ((0, 0, 1) where |pi|^2 <= 1e-20), FP64 arithmetic stored as
//    FP32, layout (z, y, x, channel).
//  * Image (the fragment shader of visualization/gl_backend.py:519-710):
//    per pixel a ray from the inverse view rows, clipped to the box, marched
//    front to back with early exit at alpha > 0.95; samples are trilinear with
//    clamp-to-edge (GL_LINEAR / GL_CLAMP_TO_EDGE of the volume texture), colour
//    from the 1-D transfer table (color_mode 0) or from the pion vector's HSL
//    colour (otherwise); pixels whose ray misses the box keep the white clear
//    colour.  Rows are stored top first.
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <type_traits>

#include "sky_host.h"

namespace sky {

// ---------------------------------------------------------------------------
// volume
// ---------------------------------------------------------------------------
constexpr int kMMBlocks = 592;  // partial extrema per launch (4 x 148 SMs)

__global__ void k_minmax_partial(const double* __restrict__ d, int64_t n, double* __restrict__ part) {
    __shared__ double smin[256], smax[256];
    double lo = 1.0e300, hi = -1.0e300;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double v = d[i];
        lo = fmin(lo, v);
        hi = fmax(hi, v);
    }
    smin[threadIdx.x] = lo;
    smax[threadIdx.x] = hi;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            smin[threadIdx.x] = fmin(smin[threadIdx.x], smin[threadIdx.x + s]);
            smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + s]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = smin[0];
        part[2 * blockIdx.x + 1] = smax[0];
    }
}

// One block: the global extrema of nb partials into out[0], out[1].
__global__ void k_minmax_final(const double* __restrict__ part, int nb, double* __restrict__ out) {
    __shared__ double smin[256], smax[256];
    double lo = 1.0e300, hi = -1.0e300;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        lo = fmin(lo, part[2 * b]);
        hi = fmax(hi, part[2 * b + 1]);
    }
    smin[threadIdx.x] = lo;
    smax[threadIdx.x] = hi;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            smin[threadIdx.x] = fmin(smin[threadIdx.x], smin[threadIdx.x + s]);
            smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + s]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = smin[0];
        out[1] = smax[0];
    }
}

// One block per (32 x) x (32 z) tile of one y plane.  The field and density are
// read along z, their fastest axis, and the volume is written along x, its
// fastest axis; the tile is transposed through shared memory so both sides
// stay coalesced.
__global__ void __launch_bounds__(256) k_build_volume(int X, int Y, int Z, const double* __restrict__ dens,
                                                      const double* __restrict__ field,
                                                      const double* __restrict__ mm, float4* __restrict__ vol) {
    __shared__ float4 tile[32][33];
    const int64_t N = (int64_t)X * Y * Z;
    const int z0 = blockIdx.x * 32, y = blockIdx.y, x0 = blockIdx.z * 32;
    const double vmin = mm[0], vmax = mm[1];
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int x = x0 + i, z = z0 + threadIdx.x;
        if (x < X && z < Z) {
            const int64_t s = ((int64_t)x * Y + y) * Z + z;
            const double dn = (dens[s] - vmin) / (vmax - vmin + 1.0e-30);
            const double p1 = field[N + s], p2 = field[2 * N + s], p3 = field[3 * N + s];
            const double n2 = p1 * p1 + p2 * p2 + p3 * p3;
            double nx = 0.0, ny = 0.0, nz = 1.0;
            if (!(n2 <= 1.0e-20)) {
                const double inv = 1.0 / sqrt(n2);
                nx = p1 * inv;
                ny = p2 * inv;
                nz = p3 * inv;
            }
            tile[i][threadIdx.x] = make_float4((float)dn, (float)nx, (float)ny, (float)nz);
        }
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int z = z0 + j, x = x0 + threadIdx.x;
        if (z < Z && x < X) vol[((int64_t)z * Y + y) * X + x] = tile[threadIdx.x][j];
    }
}

// ---------------------------------------------------------------------------
// ray march
// ---------------------------------------------------------------------------
struct RenderParams {
    float inv0[4], inv1[4], inv2[4];
    float box[3];
    float zoom, brightness, levelset, dmin, dmax, tscale, oscale, tstep;
    int max_steps, color_mode, width, height;
};

// The viewer's 1-D transfer texture (gl_backend.py:839), nine RGBA entries.
__constant__ float c_transfer[9][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {1.0f, 0.0f, 0.0f, 1.0f}, {1.0f, 0.5f, 0.0f, 1.0f},
                                       {1.0f, 1.0f, 0.0f, 1.0f}, {0.0f, 1.0f, 0.0f, 1.0f}, {0.0f, 1.0f, 1.0f, 1.0f},
                                       {0.0f, 0.0f, 1.0f, 1.0f}, {1.0f, 0.0f, 1.0f, 1.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};

// Linear filtering with clamp-to-edge along one axis: texel indices and weight.
__device__ __forceinline__ void lin_axis(float s, int n, int& i0, int& i1, float& w) {
    const float u = s * (float)n - 0.5f;
    const float f = floorf(u);
    w = u - f;
    const int i = (int)f;
    i0 = min(max(i, 0), n - 1);
    i1 = min(max(i + 1, 0), n - 1);
}

// What a trilinear cell's corners hold: the density alone (transfer table), or density and pion
// vector.
__device__ __forceinline__ float texel(const float4* v, float) { return __ldg(&v->x); }
__device__ __forceinline__ float4 texel(const float4* v, float4) { return __ldg(v); }
__device__ __forceinline__ float density(float v) { return v; }
__device__ __forceinline__ float density(const float4& v) { return v.x; }
// What makes a vector's colour a number (pion_rgb: its third component gives the lightness; a
// direction in the other two that is none gives black).
__device__ __forceinline__ float lightness(float) { return 0.0f; }
__device__ __forceinline__ float lightness(const float4& v) { return fabsf(v.w); }
__device__ __forceinline__ float mix1(float a, float b, float t) { return a + (b - a) * t; }
template <class F, class C>
__device__ __forceinline__ float trilinear(const C (&c)[8], F get, float wx, float wy, float wz) {
    return mix1(mix1(mix1(get(c[0]), get(c[1]), wx), mix1(get(c[2]), get(c[3]), wx), wy),
                mix1(mix1(get(c[4]), get(c[5]), wx), mix1(get(c[6]), get(c[7]), wx), wy), wz);
}

// The transfer table is read from a shared-memory copy: lanes index different entries,
// which the constant cache would serialise.
__device__ __forceinline__ float4 transfer(const float4* tf, float s) {
    int i0, i1;
    float w;
    lin_axis(s, 9, i0, i1, w);
    const float4 a = tf[i0], b = tf[i1];
    return make_float4(a.x + (b.x - a.x) * w, a.y + (b.y - a.y) * w, a.z + (b.z - a.z) * w, a.w + (b.w - a.w) * w);
}

// pionVectorToRGB (gl_backend.py:573-592): HSL with saturation 1, lightness from n_z
// and hue from the azimuth of (n_x, n_y).
__device__ __forceinline__ float3 pion_rgb(float nx, float ny, float nz) {
    const float PI = 3.14159265359f;
    const float l = 0.5f * (nz + 1.0f);
    const float c = 1.0f - fabsf(2.0f * l - 1.0f);
    float h = atan2f(ny, nx);
    if (h < 0.0f) h += 2.0f * PI;
    const float q = 3.0f * h / PI;
    const float md = q - 2.0f * floorf(q / 2.0f);  // GLSL mod(q, 2)
    const float x = c * (1.0f - fabsf(md - 1.0f));
    const float m = l - 0.5f * c;
    if (q >= 0.0f && q < 1.0f) return make_float3(c + m, x + m, m);
    if (q >= 1.0f && q < 2.0f) return make_float3(x + m, c + m, m);
    if (q >= 2.0f && q < 3.0f) return make_float3(m, c + m, x + m);
    if (q >= 3.0f && q < 4.0f) return make_float3(m, x + m, c + m);
    if (q >= 4.0f && q < 5.0f) return make_float3(x + m, m, c + m);
    if (q >= 5.0f && q < 6.0f) return make_float3(c + m, m, x + m);
    return make_float3(0.0f, 0.0f, 0.0f);
}

// The march is bound by instruction issue: about a thousand samples a ray, eight or so of which
// fall into one cell of eight texels.  So the eight corners stay in registers while the ray is
// in their cell, and a cell whose corners all lie below what the colouring shows -- by a margin
// far above the interpolation's rounding, so that every sample in it adds exactly nothing -- is
// crossed without sampling: the position is advanced by the same additions, up to the last step
// that is sure to stay in the cell.  Cells within reach of two box faces, whose edges are drawn
// black, are always sampled.  1200 x 900 pixels of a 128^3 volume with pion colours: 10.9 ms when
// every sample fetched its corners, 2.1 ms now.
// With pion colours a sample interpolates the density first, and the vector and its colour only above
// the level set: in a noisy volume few cells are empty, and there holding corners alone was slower
// than fetching them (density noise of 30 %, 128^3, 400 x 300 pixels: 1.76 ms fetched, 2.21 held, 1.70
// with the density first; 1200 x 900 11.0, 12.9, 9.8).
//
// The march's roundings are written out -- the position's step fused, the texel coordinate not,
// the pion colouring's excess over the level set fused -- so that a position and a colour do not
// depend on which expressions the two instances and the skip let the compiler contract.
template <bool PION>
__global__ void __launch_bounds__(256) k_render(const float4* __restrict__ vol, int X, int Y, int Z, RenderParams rp,
                                                float4* __restrict__ img) {
    using Tex = typename std::conditional<PION, float4, float>::type;
    __shared__ float4 tf[9];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    if (tid < 9) tf[tid] = make_float4(c_transfer[tid][0], c_transfer[tid][1], c_transfer[tid][2], c_transfer[tid][3]);
    __syncthreads();
    // a warp is 8 x 4 pixels: its rays cross the same cells for longer than those of 16 x 2
    const int px = blockIdx.x * 16 + ((tid >> 5) & 1) * 8 + (tid & 7);
    const int row = blockIdx.y * 16 + (tid >> 6) * 4 + ((tid >> 3) & 3);
    if (px >= rp.width || row >= rp.height) return;
    float4* out = img + (int64_t)row * rp.width + px;
    const float u = ((px + 0.5f) / (float)rp.width) * 2.0f - 1.0f;
    const float v = (1.0f - (row + 0.5f) / (float)rp.height) * 2.0f - 1.0f;
    // eye ray: origin = translation column of the inverse view, direction = R^-1 (u, v, -zoom)
    const float ox = rp.inv0[3], oy = rp.inv1[3], oz = rp.inv2[3];
    float dx = rp.inv0[0] * u + rp.inv0[1] * v + rp.inv0[2] * -rp.zoom;
    float dy = rp.inv1[0] * u + rp.inv1[1] * v + rp.inv1[2] * -rp.zoom;
    float dz = rp.inv2[0] * u + rp.inv2[1] * v + rp.inv2[2] * -rp.zoom;
    const float dl = sqrtf(dx * dx + dy * dy + dz * dz);
    dx /= dl;
    dy /= dl;
    dz /= dl;
    // box intersection (slab test)
    const float bx = rp.box[0], by = rp.box[1], bz = rp.box[2];
    const float ix = 1.0f / dx, iy = 1.0f / dy, iz = 1.0f / dz;
    const float tbx = ix * (-bx - ox), tby = iy * (-by - oy), tbz = iz * (-bz - oz);
    const float ttx = ix * (bx - ox), tty = iy * (by - oy), ttz = iz * (bz - oz);
    const float tnear0 = fmaxf(fmaxf(fminf(ttx, tbx), fminf(tty, tby)), fminf(ttz, tbz));
    const float tfar = fminf(fminf(fmaxf(ttx, tbx), fmaxf(tty, tby)), fmaxf(ttz, tbz));
    if (!(tfar > tnear0)) {
        *out = make_float4(1.0f, 1.0f, 1.0f, 1.0f);  // discarded: the clear colour
        return;
    }
    const float tnear = tnear0 < 0.0f ? 0.0f : tnear0;
    float sr = 0.0f, sg = 0.0f, sb = 0.0f, sa = 0.0f;
    float t = tnear;
    float p0 = ox + dx * tnear, p1 = oy + dy * tnear, p2 = oz + dz * tnear;
    const float st0 = dx * rp.tstep, st1 = dy * rp.tstep, st2 = dz * rp.tstep;
    const float inv_denom = 1.0f / fmaxf(rp.dmax - rp.dmin, 1.0e-30f);
    // texel-space coordinate per axis: ((p / b) / 2 + 1/2) n - 1/2 = p (n / 2b) + (n - 1) / 2
    const float kx = 0.5f * (float)X / bx, ky = 0.5f * (float)Y / by, kz = 0.5f * (float)Z / bz;
    const float cx = 0.5f * (float)(X - 1), cy = 0.5f * (float)(Y - 1), cz = 0.5f * (float)(Z - 1);
    // cells that a sample within 0.005 of a face may lie in (with room for rounding)
    const float nf = 0.0052f;
    const float nlx = (nf - bx) * kx + cx, nhx = (bx - nf) * kx + cx - 1.0f;
    const float nly = (nf - by) * ky + cy, nhy = (by - nf) * ky + cy - 1.0f;
    const float nlz = (nf - bz) * kz + cz, nhz = (bz - nf) * kz + cz - 1.0f;
    // steps per cell of each axis
    const float qx = 1.0f / (st0 * kx), qy = 1.0f / (st1 * ky), qz = 1.0f / (st2 * kz);
    // density below which a sample adds nothing: the transfer table is transparent below its
    // second entry, the pion colouring below the level set
    const bool finite_scale = isfinite(rp.oscale);
    const bool may_skip = !PION || (rp.tscale >= 0.0f && isfinite(rp.tscale));
    const float floor_norm = PION ? rp.levelset - 2.0e-6f * (1.0f + fabsf(rp.levelset)) : 0.5f / 9.0f - 2.0e-6f;
    float gx = INFINITY, gy = 0.0f, gz = 0.0f;  // the cell whose corners are held
    Tex c[8];
    bool empty = false;  // every sample of the cell adds nothing
    bool black = false;  // a sample of the cell that does not exceed the level set adds nothing
    for (int i = 0; i < rp.max_steps;) {
        const float ux = __fadd_rn(__fmul_rn(p0, kx), cx), uy = __fadd_rn(__fmul_rn(p1, ky), cy), uz = __fadd_rn(__fmul_rn(p2, kz), cz);
        const float fx = floorf(ux), fy = floorf(uy), fz = floorf(uz);
        if (fx != gx || fy != gy || fz != gz) {
            gx = fx, gy = fy, gz = fz;
            // clamp to edge
            const int jx = (int)fx, jy = (int)fy, jz = (int)fz;
            const int x0 = min(max(jx, 0), X - 1), x1 = min(max(jx + 1, 0), X - 1);
            const int y0 = min(max(jy, 0), Y - 1), y1 = min(max(jy + 1, 0), Y - 1);
            const int z0 = min(max(jz, 0), Z - 1), z1 = min(max(jz + 1, 0), Z - 1);
            const float4* r00 = vol + ((int64_t)z0 * Y + y0) * X;
            const float4* r10 = vol + ((int64_t)z0 * Y + y1) * X;
            const float4* r01 = vol + ((int64_t)z1 * Y + y0) * X;
            const float4* r11 = vol + ((int64_t)z1 * Y + y1) * X;
            c[0] = texel(r00 + x0, Tex{}), c[1] = texel(r00 + x1, Tex{});
            c[2] = texel(r10 + x0, Tex{}), c[3] = texel(r10 + x1, Tex{});
            c[4] = texel(r01 + x0, Tex{}), c[5] = texel(r01 + x1, Tex{});
            c[6] = texel(r11 + x0, Tex{}), c[7] = texel(r11 + x1, Tex{});
            float hi = density(c[0]), ab = fabsf(hi), light = lightness(c[0]);
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                const float d = density(c[k]);
                hi = fmaxf(hi, d);
                ab += fabsf(d);
                light += lightness(c[k]);
            }
            // (a sum that a NaN or an infinity enters is not below the bound)
            black = finite_scale && light < 1.0e30f;
            const bool number = ab < 1.0e30f;
            const float top = (hi + 4.0e-6f * ab - rp.dmin) * inv_denom;
            const int faces = (fx <= nlx || fx >= nhx) + (fy <= nly || fy >= nhy) + (fz <= nlz || fz >= nhz);
            empty = may_skip && black && number && faces < 2 && top + 2.0e-6f * fabsf(top) < floor_norm;
        }
        if (empty) {
            // the samples up to the last one sure to be in this cell, and the step out of it
            const float rx = (qx > 0.0f ? fx + 1.0f - ux : fx - ux) * qx;
            const float ry = (qy > 0.0f ? fy + 1.0f - uy : fy - uy) * qy;
            const float rz = (qz > 0.0f ? fz + 1.0f - uz : fz - uz) * qz;
            const float r = fminf(fminf(rx, ry), rz) * 0.999f - 0.05f;
            const int n = 1 + (r > 0.0f ? (int)fminf(r, 64.0f) : 0);
            for (int m = 0; m < n; ++m) {
                t += rp.tstep;
                p0 = __fmaf_rn(dx, rp.tstep, p0);
                p1 = __fmaf_rn(dy, rp.tstep, p1);
                p2 = __fmaf_rn(dz, rp.tstep, p2);
            }
            i += n;
            if (t > tfar) break;
            continue;
        }
        // box edges are drawn black
        const float e0 = fminf(fabsf(p0 + bx), fabsf(p0 - bx));
        const float e1 = fminf(fabsf(p1 + by), fabsf(p1 - by));
        const float e2 = fminf(fabsf(p2 + bz), fabsf(p2 - bz));
        const int near_faces = (e0 < 0.005f) + (e1 < 0.005f) + (e2 < 0.005f);
        if (near_faces >= 2) {
            *out = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
            return;
        }
        const float wx = ux - fx, wy = uy - fy, wz = uz - fz;
        const float d = trilinear(c, [](const Tex& q) { return density(q); }, wx, wy, wz);
        float cr, cg, cb, ca;
        if constexpr (!PION) {
            const float4 e = transfer(tf, fminf(fmaxf(__fmul_rn(d - rp.dmin, inv_denom), 0.0f), 1.0f));
            cr = e.x, cg = e.y, cb = e.z, ca = e.w * rp.oscale;
        } else {
            float inp = __fmul_rn(__fmaf_rn(d - rp.dmin, inv_denom, -rp.levelset), rp.tscale);
            if (inp < 0.0f) inp = 0.0f;
            if (inp == 0.0f && black) {
                // below the level set: the colour would be multiplied by zero
                cr = cg = cb = ca = 0.0f;
            } else {
                const float3 rgb = pion_rgb(trilinear(c, [](const Tex& q) { return q.y; }, wx, wy, wz),
                                            trilinear(c, [](const Tex& q) { return q.z; }, wx, wy, wz),
                                            trilinear(c, [](const Tex& q) { return q.w; }, wx, wy, wz));
                cr = inp * rgb.x, cg = inp * rgb.y, cb = inp * rgb.z, ca = inp * rp.oscale;
            }
        }
        cr *= ca;
        cg *= ca;
        cb *= ca;
        const float k = 1.0f - sa;
        sr += cr * k;
        sg += cg * k;
        sb += cb * k;
        sa += ca * k;
        if (sa > 0.95f) break;
        t += rp.tstep;
        if (t > tfar) break;
        p0 = __fmaf_rn(dx, rp.tstep, p0);
        p1 = __fmaf_rn(dy, rp.tstep, p1);
        p2 = __fmaf_rn(dz, rp.tstep, p2);
        ++i;
    }
    auto cl = [](float a) { return fminf(fmaxf(a, 0.0f), 1.0f); };
    *out = make_float4(cl(sr * rp.brightness), cl(sg * rp.brightness), cl(sb * rp.brightness),
                       cl(sa * rp.brightness));
}

}  // namespace sky

using namespace sky;

extern "C" {

int64_t sky_volume_scratch_size(void) { return 2 * kMMBlocks + 2; }

int sky_build_rgba_volume(const int32_t* p_i, int32_t n_pi, const double* density, const double* field,
                          double* scratch, int64_t n_scratch, float* volume, double* minmax_host, void* stream) {
    Params p;
    int rc = pack_core(p_i, n_pi, nullptr, 0, &p, false);
    if (rc) return rc;
    if (p.C < 4) return invalid("the volume needs the four pion components");
    if (!density || !field || !volume) return invalid("null buffer");
    if (reinterpret_cast<uintptr_t>(volume) % 16) return invalid("the volume must be 16-byte aligned");
    if (p.Y > 65535 || (p.X + 31) / 32 > 65535) return invalid("lattice too large for the volume builder");
    if (!scratch || n_scratch < 2 * kMMBlocks + 2) return SKY_ERR_NOMEM;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int64_t N = n_sites(p);
    int nb = ew_blocks(N);
    if (nb > kMMBlocks) nb = kMMBlocks;
    // partial extrema at scratch[2 ..], the global pair at scratch[0], scratch[1]
    k_minmax_partial<<<nb, 256, 0, st>>>(density, N, scratch + 2);
    k_minmax_final<<<1, 256, 0, st>>>(scratch + 2, nb, scratch);
    const dim3 vgrid((p.Z + 31) / 32, p.Y, (p.X + 31) / 32);
    k_build_volume<<<vgrid, dim3(32, 8), 0, st>>>(p.X, p.Y, p.Z, density, field, scratch,
                                                  reinterpret_cast<float4*>(volume));
    rc = check_cuda(cudaGetLastError(), "launch volume", __LINE__);
    if (rc || !minmax_host) return rc;
    rc = check_cuda(cudaMemcpyAsync(minmax_host, scratch, 2 * sizeof(double), cudaMemcpyDeviceToHost, st),
                    "read extrema", __LINE__);
    if (rc) return rc;
    return check_cuda(cudaStreamSynchronize(st), "sync", __LINE__);
}

int sky_render_volume(const float* volume, int32_t xlen, int32_t ylen, int32_t zlen, const float* params,
                      int32_t n_params, int32_t max_steps, int32_t color_mode, int32_t width, int32_t height,
                      float* image, void* stream) {
    if (!volume || !params || !image) return invalid("null buffer");
    if (n_params < 23) return invalid("the shader parameters are 23 floats");
    if (reinterpret_cast<uintptr_t>(volume) % 16 || reinterpret_cast<uintptr_t>(image) % 16)
        return invalid("the volume and the image must be 16-byte aligned");
    if (xlen < 1 || ylen < 1 || zlen < 1 || width < 1 || height < 1) return invalid("empty volume or image");
    if ((height + 15) / 16 > 65535) return invalid("image too tall");
    if (max_steps < 0) return invalid("max_steps must be >= 0");
    RenderParams rp;
    for (int k = 0; k < 4; ++k) rp.inv0[k] = params[k], rp.inv1[k] = params[4 + k], rp.inv2[k] = params[8 + k];
    for (int k = 0; k < 3; ++k) rp.box[k] = params[12 + k];
    rp.zoom = params[15];
    rp.brightness = params[16];
    rp.levelset = params[17];
    rp.dmin = params[18];
    rp.dmax = params[19];
    rp.tscale = params[20];
    rp.oscale = params[21];
    rp.tstep = params[22];
    rp.max_steps = max_steps;
    rp.color_mode = color_mode;
    rp.width = width;
    rp.height = height;
    if (!(rp.box[0] > 0.0f && rp.box[1] > 0.0f && rp.box[2] > 0.0f)) return invalid("box scale must be > 0");
    if (!(rp.tstep > 0.0f)) return invalid("tstep must be > 0");
    const dim3 block(16, 16);
    const dim3 grid((width + 15) / 16, (height + 15) / 16);
    auto kern = color_mode == 0 ? k_render<false> : k_render<true>;
    kern<<<grid, block, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const float4*>(volume), xlen, ylen, zlen, rp, reinterpret_cast<float4*>(image));
    return check_cuda(cudaGetLastError(), "launch render", __LINE__);
}

}  // extern "C"
