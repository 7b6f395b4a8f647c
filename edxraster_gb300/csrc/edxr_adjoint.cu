// Differentiable form: shading of the visible surface with visibility held
// fixed, and its hand-written adjoint.
//
// Forward (k_shade_visible), per pixel with a winning triangle t (the
// triangle-id buffer of the last pass):
//   clip_k = MVP (p_k, 1) for t's three input vertices (Shader.h:45)
//   (u, v) = NDC of the pixel centre; a_k = X_k - u W_k, c_k = Y_k - v W_k
//   b = (a x c) / sum(a x c)   perspective-correct barycentrics of the point
//                              of t's plane that projects to the pixel centre
//                              (the same weights Fragment::Interpolate forms,
//                              Shader.h:142-170, without the 1/16 snap, so they
//                              are smooth in the vertex positions; clipping
//                              does not change them)
//   P, N, A = sum b_k (p_k, n_k, albedo_k); colour = shading model (the same
//   one the raster kernel uses, edxr_device.cuh shade_model).
// Adjoint (k_backward): the same recomputation, then reverse-mode through
// the shading model, the interpolation, the barycentric solve and the MVP
// transform.  Per-vertex gradients are accumulated with float reductions (in
// packed scratch sums that k_finish adds to the caller's arrays, or straight
// there); the light, ks and shininess gradients in float pairs per lane and in
// double over the blocks.  Nothing per pixel is stored between the passes.
#include <cuda_runtime.h>

#include "edxr_device.cuh"

namespace edxr {

namespace {

// A warp takes kSpan or fewer consecutive pixels, lists the covered ones and
// shades those 32 at a time: with a thread per pixel, rows that the mesh covers
// in part left lanes and whole warps of a block idle (21 to 31 % of the warps
// active on 64 views of a torus, 30 % of the pixels covered).
constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr int kSpan = 256;

struct V3
{
    float x, y, z;
};
__device__ __forceinline__ V3 v3(float x, float y, float z) { return { x, y, z }; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return { a.x + b.x, a.y + b.y, a.z + b.z }; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return { a.x - b.x, a.y - b.y, a.z - b.z }; }
__device__ __forceinline__ V3 operator*(float s, V3 a) { return { s * a.x, s * a.y, s * a.z }; }
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float inv_len(V3 a) { return 1.0f / sqrtf(dot(a, a)); }
__device__ __forceinline__ V3 ld(const char* base, uint32_t stride, uint32_t i, float dflt)
{
    if (!base)
        return v3(dflt, dflt, dflt);
    const float* p = reinterpret_cast<const float*>(base + (size_t)i * stride);
    return v3(__ldg(p), __ldg(p + 1), __ldg(p + 2));
}
// gradient of y = normalize(x) applied to dy: (dy - y (y . dy)) / |x|
__device__ __forceinline__ V3 normalize_grad(V3 y, float invx, V3 dy) { return invx * (dy - dot(y, dy) * y); }

// Pairs of the barycentric solve, renormalised after every operation and with
// no product fused beyond the exact remainders: where a triangle is seen
// edge-on the solve cancels nearly all 48 bits, and the order of the roundings
// is then part of the result.
__device__ __forceinline__ FF pair_add(FF x, FF y) { return ff_norm(ff_sum(x, y)); }
__device__ __forceinline__ FF pair_sub(FF x, FF y) { return pair_add(x, ff_neg(y)); }
__device__ __forceinline__ FF pair_mul(FF x, FF y)
{
    const FF p = two_prod(x.hi, y.hi);
    return quick_two_sum(p.hi, p.lo + (x.hi * y.lo + x.lo * y.hi));
}
__device__ __forceinline__ FF pair_mul_f(FF x, float y)
{
    const FF p = two_prod(x.hi, y);
    return quick_two_sum(p.hi, p.lo + x.lo * y);
}
// m0 x + m1 y + m2 z + m3 as a pair.
__device__ __forceinline__ FF pair_dot4(float m0, float m1, float m2, float m3, float x, float y, float z)
{
    return pair_add(pair_add(two_prod(m0, x), two_prod(m1, y)), pair_add(two_prod(m2, z), { m3, 0.0f }));
}
// Everything the forward computes for one pixel, kept for the adjoint.
struct PixelState
{
    uint32_t vi[3];
    V3 p[3], n[3], a[3];
    float ac[3], cc[3];
    float bt[3], S, b[3];
    float u, v;
    V3 P, Nraw, A;
};

__device__ __forceinline__ bool pixel_forward(const FrameDesc& f, const DiffMesh& m, uint32_t tri, int px, int py,
                                              PixelState& s)
{
    if (tri >= m.nt)
        return false;
    for (int k = 0; k < 3; k++)
    {
        s.vi[k] = __ldg(m.indices + 3 * (size_t)tri + k);
        if (s.vi[k] >= m.nv)
            return false;
        s.p[k] = ld(m.positions, m.pos_stride, s.vi[k], 0.0f);
        s.n[k] = ld(m.normals, m.nrm_stride, s.vi[k], 0.0f);
        s.a[k] = ld(m.albedo, m.alb_stride, s.vi[k], 1.0f);
    }
    // The solve cancels heavily: a_k, c_k are the small projected distances of
    // the vertices from the pixel centre, each a difference of O(1) terms.
    // The clip coordinates and the pixel centre are therefore carried as
    // float pairs (hi + lo, about 48 bits; error-free products and sums,
    // Dekker 1971 / Knuth), and so are a_k, c_k, the cross products and their
    // sum, each rounded to float once: FP32 arithmetic throughout, accurate
    // to a few float ulps of the results, without the FP64 unit (slow on
    // this GPU).
    const float* M = f.mvp;
    FF X[3], Y[3], Wd[3];
    for (int k = 0; k < 3; k++)
    {
        const float x = s.p[k].x, y = s.p[k].y, z = s.p[k].z;
        X[k] = pair_dot4(M[0], M[1], M[2], M[3], x, y, z);
        Y[k] = pair_dot4(M[4], M[5], M[6], M[7], x, y, z);
        Wd[k] = pair_dot4(M[12], M[13], M[14], M[15], x, y, z);
    }
    const float rx = (float)px + 0.5f, ry = (float)py + 0.5f;  // exact
    const float* Rh = f.ndc_from_raster;
    const float* Rl = f.ndc_from_raster_lo;
    const FF u = pair_add(pair_add(pair_mul_f({ Rh[0], Rl[0] }, rx), pair_mul_f({ Rh[1], Rl[1] }, ry)), { Rh[2], Rl[2] });
    const FF v = pair_add(pair_add(pair_mul_f({ Rh[3], Rl[3] }, rx), pair_mul_f({ Rh[4], Rl[4] }, ry)), { Rh[5], Rl[5] });
    s.u = u.hi + u.lo;
    s.v = v.hi + v.lo;
    FF ac[3], cc[3];
    for (int k = 0; k < 3; k++)
    {
        ac[k] = pair_sub(X[k], pair_mul(u, Wd[k]));
        cc[k] = pair_sub(Y[k], pair_mul(v, Wd[k]));
        s.ac[k] = ac[k].hi + ac[k].lo;
        s.cc[k] = cc[k].hi + cc[k].lo;
    }
    // the cross products and their sum stay pairs too: near an edge, or on a
    // thin triangle, they cancel again
    FF bt[3];
    bt[0] = pair_sub(pair_mul(ac[1], cc[2]), pair_mul(ac[2], cc[1]));
    bt[1] = pair_sub(pair_mul(ac[2], cc[0]), pair_mul(ac[0], cc[2]));
    bt[2] = pair_sub(pair_mul(ac[0], cc[1]), pair_mul(ac[1], cc[0]));
    const FF Sf = pair_add(pair_add(bt[0], bt[1]), bt[2]);
    const float S = Sf.hi + Sf.lo;
    if (!(S != 0.0f) || !(fabsf(S) < 3.0e38f))
        return false;
    s.S = S;
    for (int k = 0; k < 3; k++)
    {
        s.bt[k] = bt[k].hi + bt[k].lo;
        s.b[k] = s.bt[k] / S;
    }
    s.P = s.b[0] * s.p[0] + s.b[1] * s.p[1] + s.b[2] * s.p[2];
    s.Nraw = s.b[0] * s.n[0] + s.b[1] * s.n[1] + s.b[2] * s.n[2];
    s.A = s.b[0] * s.a[0] + s.b[1] * s.a[1] + s.b[2] * s.a[2];
    return true;
}

// Shading model on (P, N, A); flags of the pixel shader kinds of edxr.h.
struct ShadeTerms
{
    V3 Nn, L, E, H;
    float ninv, einv, hinv;  // 1 / length before normalisation
    float nl, nh, nhc, powv, diffuse, spec;
    bool albedo, specular, clamp;
};

// Light (normalised, and 1 / its length), ks and shininess in effect for frame f.
struct Shading
{
    float light[3], light_inv, ks, shininess;
};
__device__ __forceinline__ Shading shading_of(const FrameDesc& f, const DiffMesh& m)
{
    if (m.override_shading)
        return { { m.light[0], m.light[1], m.light[2] }, m.light_inv, m.ks, m.shininess };
    return { { f.light_unit[0], f.light_unit[1], f.light_unit[2] }, f.light_inv, f.ks, f.shininess };
}

__device__ __forceinline__ V3 shade_forward(const FrameDesc& f, const Shading& sh, const PixelState& s,
                                            ShadeTerms& t)
{
    t.albedo = (f.ps_kind == 0 || f.ps_kind == 2);
    t.specular = (f.ps_kind <= 1);
    t.clamp = (f.ps_kind == 0);
    t.ninv = inv_len(s.Nraw);
    t.Nn = t.ninv * s.Nraw;
    t.L = v3(sh.light[0], sh.light[1], sh.light[2]);
    t.nl = dot(t.L, t.Nn);
    t.diffuse = (fmaxf(t.nl, 0.0f) + 0.2f) * 0.954929658551372f;
    t.spec = 0.0f;
    if (t.specular)
    {
        const V3 Er = v3(f.eye[0], f.eye[1], f.eye[2]) - s.P;
        t.einv = inv_len(Er);
        t.E = t.einv * Er;
        const V3 Hr = t.L + t.E;
        t.hinv = inv_len(Hr);
        t.H = t.hinv * Hr;
        t.nh = dot(t.Nn, t.H);
        t.nhc = t.clamp ? fmaxf(t.nh, 0.0f) : t.nh;
        t.powv = powf(t.nhc, sh.shininess);
        t.spec = sh.ks * t.powv;
    }
    if (t.albedo)
        return v3(s.A.x * t.diffuse + t.spec, s.A.y * t.diffuse + t.spec, s.A.z * t.diffuse + t.spec);
    return v3(t.diffuse + t.spec, t.diffuse + t.spec, t.diffuse + t.spec);
}

// Where a span's pixels lie: the frame of its first pixel and that pixel's
// place in it.  The frames of a pass have one size, so this is one 64-bit
// division per warp; a pixel's row is a 32-bit one.
struct Span
{
    uint32_t frame, offset;
};
__device__ __forceinline__ Span span_of(uint64_t base, uint32_t frame_pixels)
{
    const uint32_t frame = (uint32_t)(base / frame_pixels);
    return { frame, (uint32_t)(base - (uint64_t)frame * frame_pixels) };
}
__device__ __forceinline__ const FrameDesc& locate(const PassArgs& a, Span span, uint32_t at, uint32_t frame_pixels,
                                                   int& px, int& py)
{
    uint32_t offset = span.offset + at, frame = span.frame;
    while (offset >= frame_pixels)
    {
        offset -= frame_pixels;
        frame++;
    }
    const FrameDesc& f = a.frames[frame];
    const uint32_t row = offset / (uint32_t)f.width;
    py = (int)row;
    px = (int)(offset - row * (uint32_t)f.width);
    return f;
}

// The covered pixels of a warp's span, in order.
struct Covered
{
    uint32_t tri[kSpan];
    uint8_t at[kSpan];
};

// Lists the covered pixels among [base, base + 32 * rows) below `total`;
// `empty(pixel)` is called for the others.  Every lane of the warp calls it.
template <typename Empty>
__device__ __forceinline__ int list_covered(const PassArgs& a, uint64_t base, int rows, uint64_t total, uint32_t nt,
                                            Covered& list, Empty empty)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t tri[kSpan / 32];
#pragma unroll
    for (int k = 0; k < kSpan / 32; k++)
        tri[k] = k < rows && base + 32 * k + lane < total ? __ldg(a.tri_id + base + 32 * k + lane) : kNoTriangle;
    int n = 0;
#pragma unroll
    for (int k = 0; k < kSpan / 32; k++)
    {
        const bool covered = tri[k] < nt;
        const uint32_t lanes = __ballot_sync(0xffffffffu, covered);
        if (covered)
        {
            const int slot = n + __popc(lanes & ((1u << lane) - 1u));
            list.tri[slot] = tri[k];
            list.at[slot] = (uint8_t)(32 * k + lane);
        }
        else if (k < rows && base + 32 * k + lane < total)
            empty(base + 32 * k + lane);
        n += __popc(lanes);
    }
    __syncwarp();
    return n;
}

// Bound by the chain indices -> vertices -> solve and the solve's arithmetic:
// 6 blocks of 128 per SM (80 registers) 84.4 us on 50,000 triangles in 64 views
// of 256x256, 5 (91) 87, 8 (64, spilled) 90.
__global__ void __launch_bounds__(kThreads, 6) k_shade_visible(PassArgs a, uint64_t total, uint32_t frame_pixels,
                                                               int rows, DiffMesh m, float4* out)
{
    __shared__ Covered s_list[kWarps];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = ((uint64_t)blockIdx.x * kWarps + warp) * (32u * (uint32_t)rows);
    const int n = list_covered(a, base, rows, total, m.nt, s_list[warp],
                               [&](uint64_t i) { out[i] = make_float4(0.f, 0.f, 0.f, 0.f); });
    const Span span = span_of(base, frame_pixels);
    for (int b = (int)lane; b < n; b += 32)
    {
        const uint64_t i = base + s_list[warp].at[b];
        int px, py;
        const FrameDesc& f = locate(a, span, s_list[warp].at[b], frame_pixels, px, py);
        PixelState s;
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
        if (pixel_forward(f, m, s_list[warp].tri[b], px, py, s))
        {
            ShadeTerms t;
            const V3 x = shade_forward(f, shading_of(f, m), s, t);
            c = make_float4(x.x, x.y, x.z, 1.0f);
        }
        out[i] = c;
    }
}

__device__ __forceinline__ void add3(float* g, uint32_t v, V3 d)
{
    if (!g)
        return;
    atomicAdd(g + 3 * (size_t)v + 0, d.x);
    atomicAdd(g + 3 * (size_t)v + 1, d.y);
    atomicAdd(g + 3 * (size_t)v + 2, d.z);
}

// *p += v, four floats in one reduction (p 16-byte aligned).
__device__ __forceinline__ void add4(float4* p, float x, float y, float z, float w)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// A vertex's nine gradients in the packed sums (kPackedFloats floats a
// vertex): albedo, normal, position.
__device__ __forceinline__ void add_packed(float* sums, uint32_t v, V3 da, V3 dn, V3 dp)
{
    float* p = sums + kPackedFloats * (size_t)v;
    add4(reinterpret_cast<float4*>(p), da.x, da.y, da.z, dn.x);
    add4(reinterpret_cast<float4*>(p) + 1, dn.y, dn.z, dp.x, dp.y);
    atomicAdd(p + 8, dp.z);
}

// Per-vertex gradients: with few vertices to the pixels (Packed, see
// launch_backward) they are summed in a packed scratch array, three
// reductions a vertex (two of 16 bytes), and added to the caller's arrays by
// k_finish; otherwise straight into the caller's arrays, nine 4-byte
// reductions a vertex.  The reductions bounded the kernel: 50,000 triangles
// in 64 views of 256x256, 1.3 M covered pixels, 51 M reduction sectors in L2,
// 311 us; packed 236; with the covered pixels of a span listed first (and
// one double reduction of the global sums per block) and no 64-bit division
// per pixel 138, and k_shade_visible 118 -> 84.  What is left is the solve's
// arithmetic.  4 blocks of 128 per SM against 5 (some spilled) measured 151 and
// 148 us before the divisions went, 6 157.
template <bool Packed>
__global__ void __launch_bounds__(kThreads, 4) k_backward(PassArgs a, uint64_t total, uint32_t frame_pixels, int rows,
                                                          DiffMesh m, const float4* grad, DiffGrads g)
{
    __shared__ Covered s_list[kWarps];
    __shared__ double red[kWarps][5];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = ((uint64_t)blockIdx.x * kWarps + warp) * (32u * (uint32_t)rows);
    const int n = list_covered(a, base, rows, total, m.nt, s_list[warp], [](uint64_t) {});
    const Span span = span_of(base, frame_pixels);
    // The five global gradients are sums of large terms of both signs: each lane
    // keeps them as pairs, so that the order of the pixels leaves no trace.
    FF sums[5] = {};
    for (int b0 = 0; b0 < n; b0 += 32)
    {
        V3 dl = v3(0.f, 0.f, 0.f);
        float dks = 0.0f, dshin = 0.0f;
        if (b0 + (int)lane < n)
        {
            const uint64_t i = base + s_list[warp].at[b0 + lane];
            const uint32_t tri = s_list[warp].tri[b0 + lane];
            int px, py;
            const FrameDesc& f = locate(a, span, s_list[warp].at[b0 + lane], frame_pixels, px, py);
            PixelState s;
            if (pixel_forward(f, m, tri, px, py, s))
            {
                ShadeTerms t;
                const Shading sh = shading_of(f, m);
                shade_forward(f, sh, s, t);
                const float4 gc = grad[i];
                const V3 gcol = v3(gc.x, gc.y, gc.z);
                // colour = (albedo ? A * diffuse : diffuse) + spec
                const V3 dA = t.albedo ? t.diffuse * gcol : v3(0.f, 0.f, 0.f);
                const float ddiff = t.albedo ? dot(gcol, s.A) : (gcol.x + gcol.y + gcol.z);
                const float dspec = t.specular ? (gcol.x + gcol.y + gcol.z) : 0.0f;
                V3 dNn = v3(0.f, 0.f, 0.f), dL = v3(0.f, 0.f, 0.f), dP = v3(0.f, 0.f, 0.f);
                // diffuse = (max(nl, 0) + 0.2) * 3/pi
                const float dnl = (t.nl > 0.0f) ? ddiff * 0.954929658551372f : 0.0f;
                dL = dL + dnl * t.Nn;
                dNn = dNn + dnl * t.L;
                if (t.specular)
                {
                    // spec = ks * nhc^s
                    dks = dspec * t.powv;
                    if (t.nhc > 0.0f)
                        dshin = dspec * sh.ks * t.powv * logf(t.nhc);
                    float dnh = 0.0f;
                    if (!t.clamp || t.nh > 0.0f)
                        dnh = (sh.shininess == 0.0f)
                                  ? 0.0f
                                  : dspec * sh.ks * sh.shininess * powf(t.nhc, sh.shininess - 1.0f);
                    dNn = dNn + dnh * t.H;
                    const V3 dH = dnh * t.Nn;
                    const V3 dHr = normalize_grad(t.H, t.hinv, dH);  // H = normalize(L + E)
                    dL = dL + dHr;
                    const V3 dEr = normalize_grad(t.E, t.einv, dHr);  // E = normalize(eye - P)
                    dP = dP - dEr;
                }
                const V3 dNraw = normalize_grad(t.Nn, t.ninv, dNn);
                dl = normalize_grad(t.L, sh.light_inv, dL);
                // P, N, A = sum b_k (p_k, n_k, a_k)
                float db[3];
                for (int k = 0; k < 3; k++)
                    db[k] = dot(dP, s.p[k]) + dot(dNraw, s.n[k]) + dot(dA, s.a[k]);
                // b = bt / S
                const float bdb = s.b[0] * db[0] + s.b[1] * db[1] + s.b[2] * db[2];
                float dbt[3];
                for (int k = 0; k < 3; k++)
                    dbt[k] = (db[k] - bdb) / s.S;
                // bt = a x c
                float dac[3] = { 0.f, 0.f, 0.f }, dcc[3] = { 0.f, 0.f, 0.f };
                dac[1] += dbt[0] * s.cc[2]; dcc[2] += dbt[0] * s.ac[1]; dac[2] -= dbt[0] * s.cc[1]; dcc[1] -= dbt[0] * s.ac[2];
                dac[2] += dbt[1] * s.cc[0]; dcc[0] += dbt[1] * s.ac[2]; dac[0] -= dbt[1] * s.cc[2]; dcc[2] -= dbt[1] * s.ac[0];
                dac[0] += dbt[2] * s.cc[1]; dcc[1] += dbt[2] * s.ac[0]; dac[1] -= dbt[2] * s.cc[0]; dcc[0] -= dbt[2] * s.ac[1];
                // a_k = X_k - u W_k, c_k = Y_k - v W_k, (X, Y, W) = rows 0, 1, 3 of MVP (p, 1)
                for (int k = 0; k < 3; k++)
                {
                    V3 dp = v3(0.f, 0.f, 0.f);
                    if (g.positions)
                    {
                        const float dX = dac[k], dY = dcc[k], dW = -s.u * dac[k] - s.v * dcc[k];
                        const float* M = f.mvp;
                        dp = v3(M[0] * dX + M[4] * dY + M[12] * dW, M[1] * dX + M[5] * dY + M[13] * dW,
                                M[2] * dX + M[6] * dY + M[14] * dW);
                        dp = dp + s.b[k] * dP;
                    }
                    if (Packed)
                        add_packed(g.packed, s.vi[k], s.b[k] * dA, s.b[k] * dNraw, dp);
                    else
                    {
                        add3(g.albedo, s.vi[k], s.b[k] * dA);
                        add3(g.normals, s.vi[k], s.b[k] * dNraw);
                        add3(g.positions, s.vi[k], dp);
                    }
                }
            }
        }
        const float vals[5] = { dl.x, dl.y, dl.z, dks, dshin };
#pragma unroll
        for (int q = 0; q < 5; q++)
        {
            const FF t = two_sum(sums[q].hi, vals[q]);
            sums[q] = { t.hi, sums[q].lo + t.lo };
        }
    }
    if (n > 0)
#pragma unroll
        for (int q = 0; q < 5; q++)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                sums[q] = ff_sum(sums[q], { __shfl_down_sync(0xffffffffu, sums[q].hi, o),
                                            __shfl_down_sync(0xffffffffu, sums[q].lo, o) });
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 5; q++)
            red[warp][q] = fabsf(sums[q].hi) < INFINITY ? (double)sums[q].hi + (double)sums[q].lo : (double)sums[q].hi;
    __syncthreads();
    if (threadIdx.x < 5)
    {
        double r = 0.0;
        for (int w = 0; w < kWarps; w++)
            r += red[w][threadIdx.x];
        if (r != 0.0)
            atomicAdd(g.scratch + threadIdx.x, r);
    }
}

// Adds the packed sums to the caller's arrays, the light, ks and shininess
// sums to theirs, and leaves both zero for the next call.
__global__ void __launch_bounds__(kThreads) k_finish(DiffGrads g, uint32_t nv)
{
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (g.packed && v < nv)
    {
        float4* p = reinterpret_cast<float4*>(g.packed + kPackedFloats * (size_t)v);
        const float4 x = p[0], y = p[1], z = p[2];
        // (atomic: passes of other renderers may be adding to the same arrays;
        // a vertex that no pixel saw is left alone)
        auto add = [&](float* out, float a, float b, float c) {
            if (!out)
                return;
            out += 3 * (size_t)v;
            if (a != 0.0f) atomicAdd(out, a);
            if (b != 0.0f) atomicAdd(out + 1, b);
            if (c != 0.0f) atomicAdd(out + 2, c);
        };
        add(g.albedo, x.x, x.y, x.z);
        add(g.normals, x.w, y.x, y.y);
        add(g.positions, y.z, y.w, z.x);
        p[0] = p[1] = p[2] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (v == 0)
    {
        if (g.light)
            for (int q = 0; q < 3; q++)
                g.light[q] += (float)g.scratch[q];
        if (g.ks)
            g.ks[0] += (float)g.scratch[3];
        if (g.shininess)
            g.shininess[0] += (float)g.scratch[4];
        for (int q = 0; q < 5; q++)
            g.scratch[q] = 0.0;
    }
}

}  // namespace

// Rows of 32 pixels per warp: as many as leave each SM about 48 warps of
// work, so that small images still spread over the chip.
static int span_rows(const PassArgs& a, uint64_t total)
{
    const uint64_t sms = a.num_sms > 0 ? (uint64_t)a.num_sms : 148, rows = total / (32 * 48 * sms);
    return rows < 1 ? 1 : rows > kSpan / 32 ? kSpan / 32 : (int)rows;
}

cudaError_t launch_shade_visible(const PassArgs& a, uint64_t total, const DiffMesh& m, float4* out, cudaStream_t s)
{
    const int rows = span_rows(a, total);
    if (total)
        k_shade_visible<<<(unsigned)((total + kThreads * rows - 1) / (kThreads * rows)), kThreads, 0, s>>>(
            a, total, (uint32_t)(total / a.num_frames), rows, m, out);
    return cudaGetLastError();
}

cudaError_t launch_backward(const PassArgs& a, uint64_t total, const DiffMesh& m, const float4* grad,
                            const DiffGrads& g, cudaStream_t s)
{
    const int rows = span_rows(a, total);
    const unsigned blocks = (unsigned)((total + kThreads * rows - 1) / (kThreads * rows));
    const uint32_t frame_pixels = (uint32_t)(total / a.num_frames);
    if (total && g.packed)
        k_backward<true><<<blocks, kThreads, 0, s>>>(a, total, frame_pixels, rows, m, grad, g);
    else if (total)
        k_backward<false><<<blocks, kThreads, 0, s>>>(a, total, frame_pixels, rows, m, grad, g);
    k_finish<<<g.packed ? (m.nv + kThreads - 1) / kThreads : 1, kThreads, 0, s>>>(g, m.nv);
    return cudaGetLastError();
}

}  // namespace edxr
