// sph_mc.cuh — density grid, grid normals and marching cubes on the device.
//
// Replaces integrate_dens / integrate_normal (SPH-3D-2/sph_system.cu:1842-2351)
// and the host marching cubes SPHSystem::marching_cube(_cell)
// (SPH-3D-2/sph_system.cpp:406-542), which the reference runs on the CPU
// after copying the whole grid back every step.
//
// Grid: ndens[0] x ndens[1] x ndens[2] nodes at (i * den_size), node index
// g = z*R*C + y*R + x.  Cubes are numbered in the reference's loop order
// (x outer, y, z inner): q = (x*(C-1) + y)*(L-1) + z, so the scan over cube
// triangle counts appends triangles in the reference's order.
#pragma once
#include <cstdint>
#include <vector>
#include "../../include/sph/sph.h"
#include "sph_kernels.cuh"
#include "sph_mc_tables.h"

namespace sph {

struct McBuffers {
    uint32_t nodes = 0, cubes = 0, max_tri = 0;
    float *dens = nullptr;        // [nodes]
    float4 *normal = nullptr;     // [nodes]
    uint32_t *cube_cnt = nullptr; // [cubes]
    uint32_t *cube_off = nullptr; // [cubes]
    uint32_t *num_tri = nullptr;  // [1] total triangles of the last extraction
    float *tri = nullptr;         // [6][max_tri][3]: v0 v1 v2 n0 n1 n2
};

inline int mc_alloc(McBuffers &mc, const sph_config &c, std::vector<void *> &allocs)
{
    if (c.dim != 3 || c.ndens[0] < 2 || c.ndens[1] < 2 || c.ndens[2] < 2) return SPH_OK;
    mc.nodes = c.ndens[0] * c.ndens[1] * c.ndens[2];
    mc.cubes = (c.ndens[0] - 1) * (c.ndens[1] - 1) * (c.ndens[2] - 1);
    mc.max_tri = c.max_triangles ? c.max_triangles : 3u * mc.nodes;
    auto alloc = [&](void **p, size_t bytes) {
        if (cudaMalloc(p, bytes ? bytes : 4) != cudaSuccess) return SPH_ERR_CUDA;
        cudaMemset(*p, 0, bytes ? bytes : 4);
        allocs.push_back(*p);
        return SPH_OK;
    };
    int rc = 0;
    rc |= alloc((void **)&mc.dens, sizeof(float) * mc.nodes);
    rc |= alloc((void **)&mc.normal, sizeof(float4) * mc.nodes);
    rc |= alloc((void **)&mc.cube_cnt, sizeof(uint32_t) * mc.cubes);
    rc |= alloc((void **)&mc.cube_off, sizeof(uint32_t) * mc.cubes);
    rc |= alloc((void **)&mc.num_tri, sizeof(uint32_t) * 4);
    rc |= alloc((void **)&mc.tri, sizeof(float) * 18ull * mc.max_tri);
    return rc ? SPH_ERR_CUDA : SPH_OK;
}

// Density splat at every node from the particles of the 27 cells around the
// node's cell, on the given (stale) cell ranges and positions
// (integrate_dens_kernel, SPH-3D-2/sph_system.cu:1905-2183).  Nodes on the
// lower faces stay 0 (the reference's upper-face test never fires).  The
// weight is m * poly6(R) * (R^2 - r^2)^3 with R the particle radius, or the
// kernel length when splat_with_kernel is set.
//
// One thread per two x-adjacent nodes (2m-1, 2m), or (QUAD) per 2 x 2 nodes,
// (2m-1, 2m) in x and in y, where all four lie in one cell.  Nodes of one cell
// have one stencil: each of its candidates is loaded once for all of them.
// Each node still sums exactly its own stencil's particles in its own walk
// order (a node of a pair whose cell differs from its partner's takes the
// candidates of the joint row range that fall in its own range).
//
// Bound by the candidates' loads (lanes of a warp read different cells, so a
// 16-byte load is many L1 requests) and by issue: four nodes per load instead
// of two took 1.24M particles on 3.3M nodes from 414 to 223 us with 256-thread
// blocks; with 128 the heavy groups spread better (surface stage 29.3 -> 28.1
// us a step, built every tenth).
constexpr uint32_t kSplatThreads = 128;

// 2 x 2 nodes a thread where every group lies in one cell and five blocks per
// SM are left (surface stage, x pairs / groups: 2 spacings, 0.1M nodes 37 / 47
// us, 0.3M 57 / 53, 0.8M 107 / 78; 4 spacings, 0.3M 45 / 51, 0.8M 76 / 70, 6.4M
// 315 / 243).  With an even number s of node spacings per cell, cell q holds the
// nodes q s + 1 .. q s + s, whole groups, and FP32 rounding moves none of them up
// to 2^22 nodes an axis: the last one lies a part 1 / (nodes) of its value below
// the next cell, and two roundings add less than a part 2^-23; the first one lies
// (1 - q / ncell) / s above its cell's start, and rounding takes at most
// (1 - q / ncell) ncell 2^-25 more than it would need to land on the start.  Such
// an axis has an odd number of nodes, so no group is cut off.
inline bool splat_quads(const uint32_t *ndens, const uint32_t *ncell, int num_sms)
{
    return (ndens[0] - 1) % (2 * ncell[0]) == 0 && (ndens[1] - 1) % (2 * ncell[1]) == 0 &&
           ndens[0] <= 1u << 22 && ndens[1] <= 1u << 22 &&
           (uint64_t)ndens[0] * ndens[1] * ndens[2] >= 4ull * 5 * kSplatThreads * num_sms;
}

__host__ __device__ inline uint32_t splat_groups(const uint32_t *ndens, bool quads)
{
    return (ndens[0] / 2 + 1) * (quads ? ndens[1] / 2 + 1 : ndens[1]) * ndens[2];   // groups {0}, {1, 2}, {3, 4}, ...
}

template <bool QUAD>
__global__ void __launch_bounds__(kSplatThreads) k_splat(sph_config c, const uint32_t *off,
                                                         const float4 *pos, float *dens)
{
    dependent_entry();
    const uint32_t R = c.ndens[0], Cn = c.ndens[1];
    const uint32_t GX = R / 2 + 1, GY = QUAD ? Cn / 2 + 1 : Cn;
    const uint32_t G = splat_groups(c.ndens, QUAD);
    // per level: the squared splat radius and m * W's coefficient
    const float rad0 = c.splat_with_kernel ? c.kernel[0] : c.radius[0];
    const float rad1 = c.splat_with_kernel ? c.kernel[1] : c.radius[1];
    const float rs0 = __fmul_rn(rad0, rad0), rs1 = __fmul_rn(rad1, rad1);
    const float cf0 = __fmul_rn(c.mass[0], c.splat_with_kernel ? c.poly6[0] : c.poly6_radius[0]);
    const float cf1 = __fmul_rn(c.mass[1], c.splat_with_kernel ? c.poly6[1] : c.poly6_radius[1]);
    for (uint32_t g = grid_stride_start(); g < G; g += grid_stride()) {
        const uint32_t gx = g % GX, gyz = g / GX, gy = gyz % GY, vz = gyz / GY;
        const uint32_t va = 2u * gx - 1u, vb = 2u * gx;   // va is not a node when gx = 0
        auto cell = [&](uint32_t v, int a) {
            return min((uint32_t)floorf(__fmul_rn(__fdiv_rn((float)v, (float)c.ndens[a]), (float)c.ncell[a])),
                       c.ncell[a] - 1);
        };
        const float xa = __fmul_rn((float)va, c.den_size), xb = __fmul_rn((float)vb, c.den_size);
        const float nz = __fmul_rn((float)vz, c.den_size);
        // acc += (m * W) * (rad^2 - r^2)^3 over r^2 < rad^2
        auto add = [&](float &acc, float nx, float ny, const float4 &pj, bool l1) {
            float dx, dyy, dzz;
            const float r2 = r2_of<3>(pj, make_float4(nx, ny, nz, 0.f), dx, dyy, dzz);
            const float rad2 = l1 ? rs0 : rs1;
            const float x = __fsub_rn(rad2, r2);
            if (r2 < rad2) acc = __fmaf_rn(l1 ? cf0 : cf1, __fmul_rn(__fmul_rn(x, x), x), acc);
        };
        const uint32_t ya = QUAD ? 2u * gy - 1u : gy, yb = 2u * gy;   // 2 gy - 1 is not a node when gy = 0
        float *const row_a = dens + ((size_t)vz * Cn + ya) * R;
        if constexpr (QUAD) {
            float *const row_b = dens + ((size_t)vz * Cn + yb) * R;
            float aa = 0.0f, ba = 0.0f, ab = 0.0f, bb = 0.0f;   // 0 on the lower faces
            if (gx > 0 && gy > 0 && vz > 0) {
                const uint3 q = make_uint3(cell(va, 0), cell(ya, 1), cell(vz, 2));
                const float nya = __fmul_rn((float)ya, c.den_size), nyb = __fmul_rn((float)yb, c.den_size);
                for (int dz = -1; dz <= 1; ++dz)
                    for (int dy = -1; dy <= 1; ++dy) {
                        uint32_t b, e;
                        if (!row_range<3>(c, off, q, dy, dz, b, e)) continue;
                        for (uint32_t t = b; t < e; ++t) {
                            const float4 pj = pos[t];
                            const bool l1 = pj.w == 1.0f;
                            add(aa, xa, nya, pj, l1);
                            add(ba, xb, nya, pj, l1);
                            add(ab, xa, nyb, pj, l1);
                            add(bb, xb, nyb, pj, l1);
                        }
                    }
            }
            if (gx > 0 && gy > 0) row_a[va] = aa;
            if (gy > 0) row_a[vb] = ba;
            if (gx > 0) row_b[va] = ab;
            row_b[vb] = bb;
        } else {
            const bool has_b = vb < R;
            float acc_a = 0.0f, acc_b = 0.0f;
            if (gx > 0 && gy > 0 && vz > 0) {
                const uint32_t qax = cell(va, 0), qbx = has_b ? cell(vb, 0) : qax;
                const uint3 qa = make_uint3(qax, cell(gy, 1), cell(vz, 2)), qb = make_uint3(qbx, qa.y, qa.z);
                const float ny = __fmul_rn((float)gy, c.den_size);
                for (int dz = -1; dz <= 1; ++dz)
                    for (int dy = -1; dy <= 1; ++dy) {
                        uint32_t ba, ea;
                        if (!row_range<3>(c, off, qa, dy, dz, ba, ea)) continue;
                        if (qbx == qax) {   // one stencil for both
                            for (uint32_t t = ba; t < ea; ++t) {
                                const float4 pj = pos[t];
                                const bool l1 = pj.w == 1.0f;
                                add(acc_a, xa, ny, pj, l1);
                                add(acc_b, xb, ny, pj, l1);
                            }
                            continue;
                        }
                        // node b's row range starts and ends later in slot order
                        uint32_t bb, eb;
                        row_range<3>(c, off, qb, dy, dz, bb, eb);
                        for (uint32_t t = ba; t < eb; ++t) {
                            const float4 pj = pos[t];
                            const bool l1 = pj.w == 1.0f;
                            if (t < ea) add(acc_a, xa, ny, pj, l1);
                            if (t >= bb) add(acc_b, xb, ny, pj, l1);
                        }
                    }
            }
            if (gx > 0) row_a[va] = acc_a;
            if (has_b) row_a[vb] = acc_b;
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_grid_normals(sph_config c, const float *dens,
                                                          float4 *normal)
{
    dependent_entry();
    const uint32_t R = c.ndens[0], Cn = c.ndens[1], L = c.ndens[2];
    const uint32_t G = R * Cn * L;
    for (uint32_t g = grid_stride_start(); g < G; g += grid_stride()) {
        const uint32_t yz = g / R, vz = yz / Cn;
        const uint32_t v[3] = {g - yz * R, yz - vz * Cn, vz};
        const uint32_t dims[3] = {R, Cn, L};
        const uint32_t stride[3] = {1u, R, R * Cn};
        float n[3];
        for (int a = 0; a < 3; ++a) {
            const float lo = v[a] == 0 ? 0.0f : dens[g - stride[a]];
            const float hi = v[a] == dims[a] - 1 ? 0.0f : dens[g + stride[a]];
            n[a] = lo - hi;
        }
        // no gradient (all of the empty space): what the divisions below give,
        // without their instructions, which bound this kernel (3.3M nodes
        // 38 -> 24 us)
        if (n[0] == 0.0f && n[1] == 0.0f && n[2] == 0.0f && c.den_size > 0.0f) {
            normal[g] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        for (int a = 0; a < 3; ++a) n[a] /= c.den_size;
        const float len = sqrtf(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        normal[g] = len == 0.0f ? make_float4(0.f, 0.f, 0.f, 0.f)
                                : make_float4(n[0] / len, n[1] / len, n[2] / len, 0.f);
    }
}

__device__ __forceinline__ uint32_t mc_cube_case(const sph_config &c, const float *dens, uint32_t x,
                                                 uint32_t y, uint32_t z)
{
    const uint32_t R = c.ndens[0], Cn = c.ndens[1];
    uint32_t flags = 0;
    for (int v = 0; v < 8; ++v) {
        const uint32_t g = (z + kMcCornerOffset[v][2]) * R * Cn + (y + kMcCornerOffset[v][1]) * R +
                           (x + kMcCornerOffset[v][0]);
        if (dens[g] > c.iso_value) flags |= 1u << v;   // SPH-3D-2/sph_system.cpp:459-466
    }
    return flags;
}

__device__ __forceinline__ uint32_t mc_tri_count(uint32_t flags)
{
    uint32_t k = 0;   // triangles fill a row from its start
#pragma unroll
    for (int j = 0; j < 5; ++j) k += kMcTriangles[flags][3 * j] >= 0;
    return k;
}

// Triangle counts.  Cubes are numbered z-innermost, nodes x-innermost: a block
// takes 32 x 32 cubes in x and z and walks ys cubes in y, reads each plane of
// nodes along x, keeps one byte per node of two planes in shared memory, and
// writes the counts along z (a thread per cube read eight scattered lines for
// its corners: 3.2M cubes 41.5 -> 15.5 us, 0.5M cubes 9.7 -> 5.0 us).
constexpr uint32_t kMcTile = 32, kMcSide = kMcTile + 1, kMcPitch = 36;   // a column's bytes: 9 words apart, no bank twice

__global__ void __launch_bounds__(kThreads) k_mc_count(sph_config c, const float *dens,
                                                      uint32_t *cnt, uint32_t ys)
{
    __shared__ uint8_t in[2][kMcSide * kMcPitch], tris[256];
    dependent_entry();
    const uint32_t R = c.ndens[0], Cn = c.ndens[1], L = c.ndens[2];
    const uint32_t Rm = R - 1, Cm = Cn - 1, Lm = L - 1;
    const uint32_t tx = (Rm + kMcTile - 1) / kMcTile, tz = (Lm + kMcTile - 1) / kMcTile;
    const uint32_t bx = blockIdx.x % tx, bzy = blockIdx.x / tx, bz = bzy % tz;   // tiles in x, z, then runs in y
    const uint32_t x0 = bx * kMcTile, z0 = bz * kMcTile;
    const uint32_t y0 = (bzy / tz) * ys, y1 = min(y0 + ys, Cm);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    static_assert(kThreads == 256, "a thread per case, 8 columns of cubes per round");
    tris[tid] = (uint8_t)mc_tri_count(tid);
    // this thread's nodes of a plane: an offset from the plane's first node, or none
    constexpr uint32_t kPer = (kMcSide * kMcSide + kThreads - 1) / kThreads;
    uint32_t node[kPer], at[kPer], b[kPer];
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i) {
        const uint32_t u = tid + i * kThreads, zz = u / kMcSide, xx = u - zz * kMcSide;
        at[i] = zz * kMcPitch + xx;
        node[i] = u < kMcSide * kMcSide && x0 + xx < R && z0 + zz < L ? (z0 + zz) * Cn * R + x0 + xx : ~0u;
        b[i] = node[i] != ~0u && dens[node[i] + y0 * R] > c.iso_value ? 2u : 0u;   // SPH-3D-2/sph_system.cpp:459-466
    }
    for (uint32_t y = y0; y < y1; ++y) {
        uint8_t *const buf = in[y & 1];
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {   // bit 0: the node at y, bit 1: at y + 1
            b[i] = (b[i] >> 1) | (node[i] != ~0u && dens[node[i] + (y + 1) * R] > c.iso_value ? 2u : 0u);
            if (i < kPer - 1 || tid + i * kThreads < kMcSide * kMcSide) buf[at[i]] = (uint8_t)b[i];
        }
        __syncthreads();   // the next plane goes to the other buffer
        if (z0 + lane < Lm) {
            auto face = [](uint32_t lo, uint32_t hi) { return (lo & 1u) | (hi << 1) | ((lo & 2u) << 2); };
            for (uint32_t xx = warp; xx < kMcTile && x0 + xx < Rm; xx += kThreads / 32) {
                const uint8_t *const p = buf + lane * kMcPitch + xx;
                const uint32_t flags = face(p[0], p[1]) | (face(p[kMcPitch], p[kMcPitch + 1]) << 4);
                cnt[((x0 + xx) * Cm + y) * Lm + z0 + lane] = tris[flags];
            }
        }
    }
}

// Triangles of every cube at its scanned offset.  Edge vertices are the edge
// midpoints (a + b) / 2 of the node positions i * den_size, as the reference
// places them (SPH-3D-2/sph_system.cpp:479-480), or linear interpolation at
// the iso value when mc_interpolate is set; vertex normals are the mean of
// the two node normals.
//
// Most cubes have none.  A block's cubes write their triangles' cases to shared
// memory at the scanned offsets; its threads then take one vertex each, so the
// work is even and neighbouring threads write neighbouring vertices.  (With
// 512 or 1,024 cubes a block too few blocks are left on the surface: the
// surface stage of 0.5M cubes 53 -> 59 and 70 us.)
__global__ void __launch_bounds__(kThreads) k_mc_emit(sph_config c, const float *dens,
                                                     const float4 *normal,
                                                     const uint32_t *cnt,
                                                     const uint32_t *off, uint32_t max_tri,
                                                     float *tri)
{
    __shared__ uint32_t list[5 * kThreads];   // per triangle: cube of this block << 16 | which of its own << 8 | its case
    __shared__ uint32_t nlist;
    dependent_entry();
    const uint32_t R = c.ndens[0], Cn = c.ndens[1];
    const uint32_t Cm = Cn - 1, Lm = c.ndens[2] - 1;
    const uint32_t Q = (R - 1) * Cm * Lm;
    auto cube_at = [&](uint32_t q, uint32_t &x, uint32_t &y, uint32_t &z) {
        const uint32_t xy = q / Lm;
        z = q - xy * Lm; x = xy / Cm; y = xy - x * Cm;
    };
    const uint32_t q0 = blockIdx.x * kThreads, q = q0 + threadIdx.x;
    const uint32_t first = off[q0];
    if (q < Q) {
        const uint32_t n = cnt[q], at = off[q] - first;
        if (n) {
            uint32_t x, y, z;
            cube_at(q, x, y, z);
            const uint32_t e = (threadIdx.x << 16) | mc_cube_case(c, dens, x, y, z);
            for (uint32_t k = 0; k < n; ++k) list[at + k] = e | (k << 8);
        }
        if (threadIdx.x == kThreads - 1 || q == Q - 1) nlist = at + n;
    }
    __syncthreads();
    const uint32_t total = 3 * nlist;
    for (uint32_t i = threadIdx.x; i < total; i += kThreads) {
        const uint32_t l = i / 3, j = i - 3 * l, t = first + l;
        if (t >= max_tri) break;
        const uint32_t u = list[l] >> 16, k = (list[l] >> 8) & 0xffu, flags = list[l] & 0xffu;
        uint32_t x, y, z;
        cube_at(q0 + u, x, y, z);
        auto corner = [&](int v) {
            return ((z + kMcCornerOffset[v][2]) * Cn + (y + kMcCornerOffset[v][1])) * R + x + kMcCornerOffset[v][0];
        };
        const int e = kMcTriangles[flags][3 * k + j];
        const int a = kMcEdgeCorner[e][0], b = kMcEdgeCorner[e][1];
        const uint32_t ga = corner(a), gb = corner(b);
        float pa[3] = {__fmul_rn((float)(x + kMcCornerOffset[a][0]), c.den_size),
                       __fmul_rn((float)(y + kMcCornerOffset[a][1]), c.den_size),
                       __fmul_rn((float)(z + kMcCornerOffset[a][2]), c.den_size)};
        float pb[3] = {__fmul_rn((float)(x + kMcCornerOffset[b][0]), c.den_size),
                       __fmul_rn((float)(y + kMcCornerOffset[b][1]), c.den_size),
                       __fmul_rn((float)(z + kMcCornerOffset[b][2]), c.den_size)};
        const float4 na = normal[ga], nb = normal[gb];
        float p[3];
        if (c.mc_interpolate) {
            const float da = dens[ga], db = dens[gb];
            const float s = db != da ? (c.iso_value - da) / (db - da) : 0.5f;
            for (int d = 0; d < 3; ++d) p[d] = pa[d] + s * (pb[d] - pa[d]);
        } else {
            for (int d = 0; d < 3; ++d) p[d] = __fdiv_rn(__fadd_rn(pa[d], pb[d]), 2.0f);
        }
        const float nrm[3] = {__fdiv_rn(__fadd_rn(na.x, nb.x), 2.0f), __fdiv_rn(__fadd_rn(na.y, nb.y), 2.0f),
                              __fdiv_rn(__fadd_rn(na.z, nb.z), 2.0f)};
        float *const vo = tri + 3ull * ((size_t)j * max_tri + t), *const no = vo + 9ull * max_tri;
        for (int d = 0; d < 3; ++d) {
            vo[d] = p[d];
            no[d] = nrm[d];
        }
    }
}

}  // namespace sph
