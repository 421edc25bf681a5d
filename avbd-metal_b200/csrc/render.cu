// render.cu — headless render and observation compute: instance transforms
// of rigid colliders, smooth normals of the soft surface, skinned render
// meshes and Push-T pixel observations, written to plain device buffers.
//
// Follows Shaders/50_render.metal:7-212 and Shaders/60_robotics.metal:8-69.
// All of them are one pass over independent records; the Push-T kernel is
// the byte-heavy one (num_envs x res^2 x 3 bytes).
#include "dmath.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace avbd {

namespace {

__device__ __forceinline__ float fract_(float x) { return x - floorf(x); }

// Golden-ratio hue cycling lifted toward white (50_render.metal:25-32).
__device__ float3 palette(uint32_t i) {
    const float h = fract_((float)i * 0.61803398875f);
    const float3 off = mk3(5.0f / 6.0f, 3.0f / 6.0f, 1.0f / 6.0f);
    float3 p;
    p.x = fabsf(fract_(h + off.x) * 6.0f - 3.0f) - 1.0f;
    p.y = fabsf(fract_(h + off.y) * 6.0f - 3.0f) - 1.0f;
    p.z = fabsf(fract_(h + off.z) * 6.0f - 3.0f) - 1.0f;
    const float3 hue = clamp3(p, s3(0.0f), s3(1.0f));
    const float3 base = s3(0.92f);
    return (base + (hue - base) * 0.62f) * 0.98f;
}

__device__ __forceinline__ float3 safe_normalize(float3 v) {
    const float l = len3(v);
    return l > 1e-12f ? v / l : s3(0.0f);
}

__device__ __forceinline__ void store4(float* o, float a, float b, float c, float w) {
    *reinterpret_cast<float4*>(o) = make_float4(a, b, c, w);
}

}  // namespace

// One record per listed collider (50_render.metal:34-97).
__global__ void k_build_instances(const DevPtrs d, const uint32_t* ids, const float4* colors, uint32_t n,
                                  uint32_t colorMode, float* out) {
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n) return;
    const uint32_t col = ids[gid];
    const uint32_t body = d.colOwner[col];
    const float4 pl = d.posLin[body];
    const float4 qb = d.posAng[body];
    const float4 q = q_mul(qb, d.colLocalRot[col]);
    const float3 center = xyz(pl) + q_rotate(qb, xyz(d.colLocalPos[col]));
    const float x = q.x, y = q.y, z = q.z, w = q.w;
    const float xx = x * x, yy = y * y, zz = z * z;
    const float xy = x * y, xz = x * z, yz = y * z;
    const float wx = w * x, wy = w * y, wz = w * z;
    const float3 c0 = mk3(1.0f - 2.0f * (yy + zz), 2.0f * (xy + wz), 2.0f * (xz - wy));
    const float3 c1 = mk3(2.0f * (xy - wz), 1.0f - 2.0f * (xx + zz), 2.0f * (yz + wx));
    const float3 c2 = mk3(2.0f * (xz + wy), 2.0f * (yz - wx), 1.0f - 2.0f * (xx + yy));
    const uint32_t st = d.colShapeType[col] & SHAPE_KIND_MASK;
    const float4 sh = d.colShape[col];
    const float3 sz = st >= 2 ? s3(1.0f) : xyz(sh);
    float* o = out + 24 * (size_t)gid;
    // the static ground slab is not drawn (a floor replaces it)
    if (st == 0 && pl.w <= 0.0f && sh.x > 150.0f) {
        for (int k = 0; k < 24; k += 4) store4(o + k, 0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    store4(o + 0, c0.x * sz.x, c0.y * sz.x, c0.z * sz.x, 0.0f);
    store4(o + 4, c1.x * sz.y, c1.y * sz.y, c1.z * sz.y, 0.0f);
    store4(o + 8, c2.x * sz.z, c2.y * sz.z, c2.z * sz.z, 0.0f);
    store4(o + 12, center.x, center.y, center.z, 1.0f);
    float3 c = pl.w > 0.0f ? palette(colorMode == 1 ? d.colorsA[body] : body) : mk3(0.58f, 0.60f, 0.66f);
    if (colors) {
        const float4 rc = colors[gid];
        if (rc.w > 0.0f) c = xyz(rc);
    }
    store4(o + 16, c.x, c.y, c.z, (float)st);
    store4(o + 20, sh.x, sh.y, sh.w, pl.w > 0.0f ? 1.0f : 0.0f);
}

// Angle x area weighted vertex normals with the curvature-thinned render
// thickness (50_render.metal:104-180).  The raw face normals (twice the area
// along the normal, (b - a) x (c - a) in the triangle's own order) are formed
// here, from positions that the angles need anyway, instead of by a kernel and
// a buffer of their own: the call is bounded by its launches (24^3 soft cube,
// normals and skin, 11.6 us a pass with three launches, 9.5 with two).
__global__ void k_vertex_normals(const DevPtrs d, const uint32_t* surfVerts, const uint32_t* vtStart,
                                 const uint32_t* vtCount, const uint32_t* vtList, uint32_t numSurf,
                                 float clothScale, float4* out) {
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= numSurf) return;
    const uint32_t v = surfVerts[gid];
    const float3 p = xyz(d.posLin[v]);
    float3 acc = s3(0.0f), firstFace = s3(0.0f);
    float wsum = 0.0f;
    const uint32_t s = vtStart[gid], e = s + vtCount[gid];
    for (uint32_t k = s; k < e; k++) {
        const uint4 tr = d.tris[vtList[k]];
        const float3 a = xyz(d.posLin[tr.x]), b = xyz(d.posLin[tr.y]), c = xyz(d.posLin[tr.z]);
        const float3 fn = cross(b - a, c - a);
        if (k == s) firstFace = fn;
        const float area = 0.5f * len3(fn);
        const float3 ea = (tr.x == v ? b : a) - p, eb = (tr.x == v || tr.y == v ? c : b) - p;
        const float ang = acosf(clampf(dot(safe_normalize(ea), safe_normalize(eb)), -1.0f, 1.0f));
        const float w = area * ang;
        acc += safe_normalize(fn) * w;
        wsum += w;
    }
    // a fold-over can cancel the weighted sum: fall back to the first face
    const float coherence = wsum > 1e-9f ? len3(acc) / wsum : 0.0f;
    if (len3(acc) < 1e-6f && e > s) acc = firstFace;
    const float sc = d.clothVert[v] != 0u ? clothScale : 1.0f;
    const float c2 = clampf(coherence * coherence, 0.0f, 1.0f);
    const float thick = fabsf(d.shape[v].w) * sc * (0.25f + (1.0f - 0.25f) * c2);
    out[v] = mk4(safe_normalize(acc), thick);
}

// Skinned render vertices (50_render.metal:182-212).
__global__ void k_skin_deform(const float4* posLin, const SkinBinding* bind, uint32_t n, float4* out) {
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n) return;
    const SkinBinding b = bind[gid];
    const float3 q0 = xyz(posLin[b.ids.x]), q1 = xyz(posLin[b.ids.y]);
    const float3 q2 = xyz(posLin[b.ids.z]), q3 = xyz(posLin[b.ids.w]);
    const float3 p = q0 * b.weights.x + q1 * b.weights.y + q2 * b.weights.z + q3 * b.weights.w;
    // F = Ds Dm^-1 column by column; the normal maps by cof(F)
    const float3 e0 = q1 - q0, e1 = q2 - q0, e2 = q3 - q0;
    const float3 f0 = e0 * b.inv0.x + e1 * b.inv1.x + e2 * b.inv2.x;
    const float3 f1 = e0 * b.inv0.y + e1 * b.inv1.y + e2 * b.inv2.y;
    const float3 f2 = e0 * b.inv0.z + e1 * b.inv1.z + e2 * b.inv2.z;
    const float3 n0 = xyz(b.restNormal);
    float3 nn = cross(f1, f2) * n0.x + cross(f2, f0) * n0.y + cross(f0, f1) * n0.z;
    if (len3(nn) < 1e-10f) nn = n0;
    out[2 * gid] = mk4(p, 1.0f);
    out[2 * gid + 1] = mk4(safe_normalize(nn), 0.0f);
}

namespace {

__device__ __forceinline__ bool in_box(float px, float py, float cx, float cy, float cs, float sn, float hx,
                                       float hy) {
    const float dx = px - cx, dy = py - cy;
    const float lx = cs * dx + sn * dy;
    const float ly = -sn * dx + cs * dy;
    return fabsf(lx) <= hx && fabsf(ly) <= hy;
}

__device__ __forceinline__ uint32_t to_byte(float c) { return (uint32_t)(clampf(c, 0.0f, 1.0f) * 255.0f); }

// Heading of a body in the ground plane as (cos, sin) of atan2(fwd.y, fwd.x)
// for fwd = its rotated +x axis: the normalised (fwd.x, fwd.y), (1, 0) when
// the axis is vertical.
__device__ __forceinline__ void heading(float4 q, float& cs, float& sn) {
    const float3 f = q_rotate(q, mk3(1.0f, 0.0f, 0.0f));
    const float l = sqrtf(f.x * f.x + f.y * f.y);
    if (l > 0.0f) { cs = f.x / l; sn = f.y / l; }
    else { cs = 1.0f; sn = 0.0f; }
}

}  // namespace

// Push-T observations (60_robotics.metal:21-69) in two passes.
// k_pusht_shapes: one thread per environment places its shapes (goal T from
// the table, block T and pusher from the body poses) and bounds each of the
// five (two bars, two stems, the disc) by a range of pixel columns and rows.
// k_pusht_obs: a block takes tiles of whole pixel rows of one environment: it
// fills the tile in shared memory with the background (whose three bytes are
// equal), classifies the pixels of the five ranges only — each by all five
// tests, so ranges may overlap in any order — and writes the tile out as
// 16-byte stores.  The tile stands in shared memory at the destination's
// offset in a 16-byte word, so every resolution takes the same path; the
// bytes before and after the whole words go out singly.  The next tile's
// shapes are fetched while the current one is drawn.
//
// A range covers the shape's extent plus two pixels and a rounding allowance
// of the coordinates; a pixel outside it cannot pass the shape's test.  A
// bound that is not finite (an empty window, a lost pose) covers everything.
//
// What bounds it: issue slots (0.6 of them used) and the barriers between a
// tile's fill, its shapes and its copy; 4096 environments of 64 x 64 in 24.7 us a
// call (41.2 us when every quad of pixels ran five bounding-circle tests).
constexpr uint32_t kObsThreads = 256;
constexpr uint32_t kObsTile = 16384;             // bytes of whole rows a block draws at once
constexpr uint32_t kObsRecord = PUSHT_RECORD;    // float4 per environment: 24 floats, five ranges

// pixel range [lo, hi] of world coordinates [c - e, c + e] on an axis whose
// pixel j has coordinate origin + (j / denom - 0.5) * size; hi < lo if empty
__device__ __forceinline__ void pixel_range(float c, float e, float origin, float size, float denom, int& lo,
                                            int& hi) {
    const float m = e + 2.0f * fabsf(size) / denom + 1.0e-6f * (fabsf(origin) + fabsf(c));
    const float a = ((c - m - origin) / size + 0.5f) * denom, b = ((c + m - origin) / size + 0.5f) * denom;
    if (!(fabsf(a) <= 3.0e38f) || !(fabsf(b) <= 3.0e38f)) { lo = 0; hi = (int)denom; return; }
    lo = (int)floorf(clampf(fminf(a, b), -1.0f, denom + 1.0f));
    hi = (int)ceilf(clampf(fmaxf(a, b), -1.0f, denom + 1.0f));
    lo = lo < 0 ? 0 : lo;
    hi = hi > (int)denom ? (int)denom : hi;
}

__global__ void k_pusht_shapes(const float4* posLin, const float4* posAng, const PushTDev* envs, uint32_t numEnvs,
                               uint32_t res, float4* shapes) {
    pdl_trigger();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= numEnvs) return;
    const PushTDev env = envs[e];
    float sh[24];
    const float gx = env.frame.z + env.frame.x, gy = env.frame.w + env.frame.y;
    const float gc = env.goalCos, gs = env.goalSin;
    sh[0] = gx + (-gs) * 0.125f; sh[1] = gy + gc * 0.125f;    // goal bar centre
    sh[2] = gx + gs * 0.325f;    sh[3] = gy + (-gc) * 0.325f; // goal stem centre
    sh[4] = gc; sh[5] = gs;
    float cs, sn;
    heading(posAng[env.ids.y], cs, sn);
    sh[6] = posLin[env.ids.y].x; sh[7] = posLin[env.ids.y].y; sh[8] = cs; sh[9] = sn;
    heading(posAng[env.ids.z], cs, sn);
    sh[10] = posLin[env.ids.z].x; sh[11] = posLin[env.ids.z].y; sh[12] = cs; sh[13] = sn;
    sh[14] = posLin[env.ids.x].x; sh[15] = posLin[env.ids.x].y;
    sh[16] = env.frame.x; sh[17] = env.frame.y;
    sh[18] = 2.0f * env.halfWin;
    sh[19] = sh[20] = sh[21] = sh[22] = sh[23] = 0.0f;
    float4* out = shapes + kObsRecord * (size_t)e;
    for (int k = 0; k < 6; k++) out[k] = make_float4(sh[4 * k], sh[4 * k + 1], sh[4 * k + 2], sh[4 * k + 3]);
    // bar (half extents 0.5 x 0.125), stem (0.125 x 0.325) and pusher disc (0.13)
    const float denom = (float)(res - 1u);
    const float cx[5] = {sh[0], sh[2], sh[6], sh[10], sh[14]}, cy[5] = {sh[1], sh[3], sh[7], sh[11], sh[15]};
    const float cc[4] = {gc, gc, sh[8], sh[12]}, ss[4] = {gs, gs, sh[9], sh[13]};
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const float hx = k == 4 ? 0.13f : ((k & 1) ? 0.125f : 0.5f), hy = k == 4 ? 0.13f : ((k & 1) ? 0.325f : 0.125f);
        const float c = k == 4 ? 1.0f : fabsf(cc[k < 4 ? k : 0]), s = k == 4 ? 0.0f : fabsf(ss[k < 4 ? k : 0]);
        int x0, x1, y0, y1;
        pixel_range(cx[k], c * hx + s * hy, sh[16], sh[18], denom, x0, x1);
        pixel_range(cy[k], s * hx + c * hy, sh[17], sh[18], denom, y0, y1);
        out[6 + k] = make_float4(__int_as_float(x0), __int_as_float(x1), __int_as_float(y0), __int_as_float(y1));
    }
}

// rows of a tile: whole rows, about kObsTile bytes
__host__ __device__ __forceinline__ uint32_t obs_rows(uint32_t res) {
    const uint32_t r = kObsTile / (3u * res);
    return r == 0u ? 1u : (r < res ? r : res);
}

__global__ void __launch_bounds__(kObsThreads) k_pusht_obs(const float4* shapes, uint32_t numEnvs, uint32_t res,
                                                           uint8_t* out) {
    extern __shared__ __align__(16) uint8_t img[];   // the tile (from offset 0-15), then the pixel offsets
    __shared__ float4 rec[2][kObsRecord];
    const uint32_t t = threadIdx.x;
    const uint32_t rows = obs_rows(res), perEnv = (res + rows - 1u) / rows;
    float* offs = reinterpret_cast<float*>(img + ((rows * res * 3u + 31u) & ~15u));
    const float denom = (float)(res - 1u);
    for (uint32_t j = t; j < res; j += kObsThreads) offs[j] = (float)j / denom - 0.5f;
    pdl_wait();
    const uint64_t tiles = (uint64_t)numEnvs * perEnv;
    uint32_t buf = 0;
    if (t < kObsRecord && blockIdx.x < tiles) rec[0][t] = shapes[kObsRecord * (size_t)(blockIdx.x / perEnv) + t];
    // the palette entries as bytes
    const uint32_t pal[4][3] = {
        {to_byte(0.06f), to_byte(0.06f), to_byte(0.06f)},
        {to_byte(0.10f), to_byte(0.55f), to_byte(0.12f)},
        {to_byte(0.85f), to_byte(0.15f), to_byte(0.12f)},
        {to_byte(0.2f), to_byte(0.4f), to_byte(0.95f)}};
    const uint32_t bg = pal[0][0] * 0x01010101u;
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1u) {
        const uint32_t e = (uint32_t)(tile / perEnv), row0 = (uint32_t)(tile - (uint64_t)e * perEnv) * rows;
        const uint32_t nr = row0 + rows <= res ? rows : res - row0, bytes = nr * res * 3u;
        uint8_t* dst = out + ((size_t)e * res + row0) * res * 3u;
        const uint32_t skew = (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 15u);
        for (uint32_t v = t; v < (skew + bytes + 15u) / 16u; v += kObsThreads)
            reinterpret_cast<uint4*>(img)[v] = make_uint4(bg, bg, bg, bg);
        if (t < kObsRecord && tile + gridDim.x < tiles)
            rec[buf ^ 1u][t] = shapes[kObsRecord * (size_t)((tile + gridDim.x) / perEnv) + t];
        __syncthreads();
        const float4 s0 = rec[buf][0], s1 = rec[buf][1], s2 = rec[buf][2], s3 = rec[buf][3], s4 = rec[buf][4];
        // the pixels of the five ranges that lie in this tile's rows, one after another
        uint32_t width[5], first[6];
        int x0[5], y0[5];
        first[0] = 0u;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const float4 r = rec[buf][6 + k];
            x0[k] = __float_as_int(r.x);
            const int x1 = __float_as_int(r.y), yb = (int)row0, ye = (int)(row0 + nr) - 1;
            y0[k] = max(__float_as_int(r.z), yb);
            const int y1 = min(__float_as_int(r.w), ye);
            width[k] = x1 >= x0[k] ? (uint32_t)(x1 - x0[k] + 1) : 0u;
            first[k + 1] = first[k] + (y1 >= y0[k] ? width[k] * (uint32_t)(y1 - y0[k] + 1) : 0u);
        }
        for (uint32_t i = t; i < first[5]; i += kObsThreads) {
            uint32_t w = width[0], f = first[0];
            int bx = x0[0], by = y0[0];
#pragma unroll
            for (int k = 1; k < 5; k++)
                if (i >= first[k]) { w = width[k]; f = first[k]; bx = x0[k]; by = y0[k]; }
            const uint32_t q = (i - f) / w;
            const uint32_t py = (uint32_t)by + q, px = (uint32_t)bx + (i - f - q * w);
            const float wx = s4.x + offs[px] * s4.z, wy = s4.y + offs[py] * s4.z;
            uint32_t kind = 0;
            if (in_box(wx, wy, s0.x, s0.y, s1.x, s1.y, 0.5f, 0.125f) ||
                in_box(wx, wy, s0.z, s0.w, s1.x, s1.y, 0.125f, 0.325f))
                kind = 1;
            if (in_box(wx, wy, s1.z, s1.w, s2.x, s2.y, 0.5f, 0.125f)) kind = 2;
            if (in_box(wx, wy, s2.z, s2.w, s3.x, s3.y, 0.125f, 0.325f)) kind = 2;
            const float dx = wx - s3.z, dy = wy - s3.w;
            if (sqrtf(dx * dx + dy * dy) < 0.13f) kind = 3;
            if (kind) {
                uint8_t* o = img + skew + ((py - row0) * res + px) * 3u;
                o[0] = (uint8_t)(kind == 1 ? pal[1][0] : (kind == 2 ? pal[2][0] : pal[3][0]));
                o[1] = (uint8_t)(kind == 1 ? pal[1][1] : (kind == 2 ? pal[2][1] : pal[3][1]));
                o[2] = (uint8_t)(kind == 1 ? pal[1][2] : (kind == 2 ? pal[2][2] : pal[3][2]));
            }
        }
        __syncthreads();
        // whole 16-byte words, then the bytes at the two ends
        const uint32_t head = skew ? min(16u - skew, bytes) : 0u, words = (bytes - head) / 16u;
        const uint32_t tail = bytes - head - 16u * words;
        const uint4* src = reinterpret_cast<const uint4*>(img + skew + head);
        uint4* dv = reinterpret_cast<uint4*>(dst + head);
        for (uint32_t v = t; v < words; v += kObsThreads) dv[v] = src[v];
        if (t < head) dst[t] = img[skew + t];
        else if (t >= 32u && t - 32u < tail) dst[head + 16u * words + t - 32u] = img[skew + head + 16u * words + t - 32u];
        __syncthreads();
    }
}

static uint32_t blocks_for(uint32_t n, uint32_t threads) { return n == 0 ? 1u : (n + threads - 1) / threads; }

void launch_build_instances(const DevPtrs& d, const uint32_t* ids, const float4* colors, uint32_t n,
                            uint32_t colorMode, float* out, cudaStream_t st) {
    if (n) k_build_instances<<<blocks_for(n, 128), 128, 0, st>>>(d, ids, colors, n, colorMode, out);
}

void launch_soft_normals(const DevPtrs& d, const uint32_t* surfVerts, const uint32_t* vtStart, const uint32_t* vtCount,
                         const uint32_t* vtList, uint32_t numSurf, float clothScale, float4* out, cudaStream_t st) {
    if (!numSurf) return;
    k_vertex_normals<<<blocks_for(numSurf, 64), 64, 0, st>>>(d, surfVerts, vtStart, vtCount, vtList, numSurf, clothScale,
                                                             out);
}

void launch_skin_deform(const float4* posLin, const SkinBinding* b, uint32_t n, float4* out, cudaStream_t st) {
    if (n) k_skin_deform<<<blocks_for(n, 256), 256, 0, st>>>(posLin, b, n, out);
}

void launch_pusht_obs(const float4* posLin, const float4* posAng, const PushTDev* envs, uint32_t numEnvs,
                      uint32_t res, float4* shapes, uint8_t* out, cudaStream_t st) {
    if (!numEnvs) return;
    k_pusht_shapes<<<blocks_for(numEnvs, 64), 64, 0, st>>>(posLin, posAng, envs, numEnvs, res, shapes);
    // two waves of blocks walk the tiles (256 threads of 64 registers: four
    // blocks an SM at a time)
    const uint32_t rows = obs_rows(res);
    const uint64_t tiles = (uint64_t)numEnvs * ((res + rows - 1u) / rows);
    const uint32_t grid = (uint32_t)(tiles < 148u * 8u ? tiles : 148u * 8u);
    const size_t smem = ((rows * res * 3u + 31u) & ~15u) + sizeof(float) * res;   // at most 33 KB
    launch_pdl_smem(k_pusht_obs, grid, kObsThreads, smem, st, (const float4*)shapes, numEnvs, res, out);
}

}  // namespace avbd
