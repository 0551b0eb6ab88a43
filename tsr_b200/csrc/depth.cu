// depth.cu -- sm_100a triangulation of a depth map into a mesh whose
// vertices become samples: DepthImage::triangulate and createFlexibleMesh
// (Image/DepthImage.cpp:186-461), FlexibleMesh::findVertexNeighbors
// (FlexibleMesh.cpp:137-171) and Mesh::computeVertexScales (Mesh.cpp:63-123).
//
// The reference walks the 2x2 pixel blocks row by row, emits up to two
// triangles per block and numbers a pixel's vertex when a triangle first
// uses it.  Here every block is classified in parallel, the triangle corners
// are written in (block, triangle, corner) order after a scan, a pixel's
// first use is the smallest corner position naming it (atomicMin), and a scan
// over "this corner is its pixel's first use" ranks the first uses: the
// reference's numbering exactly.  A vertex's neighbours are visited in the
// order findVertexNeighbors lists them (first appearance over the triangles'
// edges), so the mean neighbour distance sums in the reference's order.
//
// The camera enters as the two 3x3 matrices the reference computes from its
// PinholeCamera (BaseProject, absent here): hPSToNNRayDirVS = inverse
// viewport x inverse projection, and hPSToNNRayDirWS = that x inverse
// rotation (DepthImage.cpp:189-194).  A homogeneous pixel (x, y, 1) times a
// matrix is taken as a row vector times it.
#include <cub/cub.cuh>

#include "handles.h"

namespace tsr {
namespace {

constexpr unsigned BLK = 256;
constexpr double SQRT_TWO = 1.4142135623730951;     // Math::SQRT_TWO
constexpr double DEPTH_DIFFERENCE_FACTOR = 5.0;     // DepthImage.cpp:25
constexpr uint32_t NONE = 0xFFFFFFFFu;

struct Mat3 {
    double m[9];   // row major: m[3 * i + j]
};

__constant__ uint8_t c_block_tris[4][3] = {{0, 2, 1}, {0, 3, 1}, {0, 2, 3}, {1, 2, 3}};

// (x, y, z) times M: out_j = (x m0j + y m1j) + z m2j
__device__ __forceinline__ void row_times(double x, double y, double z, const Mat3 &M, double *o) {
    for (int j = 0; j < 3; ++j)
        o[j] = __dadd_rn(__dadd_rn(__dmul_rn(x, M.m[j]), __dmul_rn(y, M.m[3 + j])), __dmul_rn(z, M.m[6 + j]));
}

__device__ __forceinline__ double length3(const double *v) {
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(v[0], v[0]), __dmul_rn(v[1], v[1])), __dmul_rn(v[2], v[2])));
}

// DepthImage::triangulateBlock (DepthImage.cpp:218-383) without the output:
// the block's triangles as indices into c_block_tris (0xF: none).
__device__ uint32_t block_triangles(const double *depths, uint32_t W, uint32_t x, uint32_t y, const Mat3 &Mvs) {
    const uint32_t p = W * y + x;
    const double d[4] = {depths[p], depths[p + 1], depths[p + W], depths[p + W + 1]};
    uint32_t mask = 0, avail = 0;
    for (uint32_t i = 0; i < 4; ++i)
        if (!(0.0 >= d[i])) {
            mask |= 1u << i;
            ++avail;
        }
    if (avail < 3) return 0xFFu;
    uint32_t t[2] = {0xFu, 0xFu};
    switch (mask) {
        case 7: t[0] = 0; break;
        case 11: t[0] = 1; break;
        case 13: t[0] = 2; break;
        case 14: t[0] = 3; break;
        case 15:
            if (fabs(__dsub_rn(d[0], d[3])) < fabs(__dsub_rn(d[1], d[2]))) { t[0] = 1; t[1] = 2; }
            else { t[0] = 0; t[1] = 3; }
            break;
        default: return 0xFFu;
    }
    double fp[4] = {0.0, 0.0, 0.0, 0.0};
    for (uint32_t i = 0; i < 4; ++i) {
        if (0.0 >= d[i]) continue;
        double v[3];
        row_times((double)(x + i % 2), (double)(y + i / 2), 1.0, Mvs, v);
        fp[i] = __ddiv_rn(__dmul_rn(Mvs.m[0], d[i]), length3(v));
    }
    for (int k = 0; k < 2; ++k) {
        if (t[k] == 0xFu) continue;
        for (uint32_t e = 0; e < 3; ++e) {   // DepthImage::isDepthDiscontinuity (DepthImage.cpp:385-400)
            const uint32_t v0 = c_block_tris[t[k]][e], v1 = c_block_tris[t[k]][(e + 1) % 3];
            const uint32_t closer = d[v0] < d[v1] ? v0 : v1, further = d[v0] < d[v1] ? v1 : v0;
            const double f = (v0 + v1 == 3) ? __dmul_rn(DEPTH_DIFFERENCE_FACTOR, SQRT_TWO) : DEPTH_DIFFERENCE_FACTOR;
            if (__dsub_rn(d[further], d[closer]) > __dmul_rn(fp[closer], f)) {
                t[k] = 0xFu;
                break;
            }
        }
    }
    return t[0] | (t[1] << 4);
}

__global__ void k_classify_blocks(const double *depths, uint32_t W, uint32_t H, Mat3 Mvs, uint8_t *code,
                                  uint32_t *ntri) {
    const uint32_t bw = W - 1, nb = bw * (H - 1);
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const uint32_t c = block_triangles(depths, W, b % bw, b / bw, Mvs);
    code[b] = (uint8_t)c;
    ntri[b] = ((c & 0xFu) != 0xFu ? 1u : 0u) + ((c >> 4) != 0xFu ? 1u : 0u);
}

// Corner pixels in (block, triangle, corner) order, and every pixel's first
// corner (the smallest corner position naming it).
__global__ void k_emit_corners(uint32_t W, uint32_t H, const uint8_t *code, const uint32_t *toff, uint32_t *corner_pix,
                               uint32_t *first) {
    const uint32_t bw = W - 1, nb = bw * (H - 1);
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const uint32_t c = code[b];
    if (c == 0xFFu) return;
    const uint32_t p = W * (b / bw) + b % bw;
    uint32_t out = 3 * toff[b];
    for (int k = 0; k < 2; ++k) {
        const uint32_t t = (c >> (4 * k)) & 0xFu;
        if (t == 0xFu) continue;
        for (int j = 0; j < 3; ++j) {
            const uint32_t v = c_block_tris[t][j];
            const uint32_t q = p + (v / 2) * W + v % 2;
            corner_pix[out] = q;
            atomicMin(first + q, out);
            ++out;
        }
    }
}

__global__ void k_first_flags(uint32_t nc, const uint32_t *corner_pix, const uint32_t *first, uint32_t *flag) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < nc) flag[c] = first[corner_pix[c]] == c ? 1u : 0u;
}

__global__ void k_pixel_vertices(uint32_t np, const uint32_t *first, const uint32_t *rank, uint32_t *pix2v) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < np) pix2v[p] = first[p] == NONE ? NONE : rank[first[p]];
}

__global__ void k_corner_vertices(uint32_t nc, const uint32_t *corner_pix, const uint32_t *pix2v, uint32_t *tris) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < nc) tris[c] = pix2v[corner_pix[c]];
}

// DepthImage::setVertexPositions / setVertexColors (DepthImage.cpp:402-461)
__global__ void k_depth_vertices(uint32_t W, uint32_t np, const uint32_t *pix2v, const double *depths, Mat3 Mws,
                                 double cx, double cy, double cz, const double *colors, double *pos, double *col) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const uint32_t v = pix2v[p];
    if (v == NONE) return;
    double dir[3];
    row_times((double)(p % W), (double)(p / W), 1.0, Mws, dir);
    const double l = length3(dir);
    if (l > 0.0)
        for (int j = 0; j < 3; ++j) dir[j] = __ddiv_rn(dir[j], l);
    const double dep = depths[p];
    pos[3 * (size_t)v] = __dadd_rn(cx, __dmul_rn(dir[0], dep));
    pos[3 * (size_t)v + 1] = __dadd_rn(cy, __dmul_rn(dir[1], dep));
    pos[3 * (size_t)v + 2] = __dadd_rn(cz, __dmul_rn(dir[2], dep));
    for (int j = 0; j < 3; ++j) col[3 * (size_t)v + j] = colors ? colors[3 * (size_t)p + j] : 0.5;
}

// Mesh::computeAverageDistance (Mesh.cpp:100-123) over the neighbours in the
// order of FlexibleMesh::findVertexNeighbors (FlexibleMesh.cpp:137-171), which
// visits, per triangle (i0, i1, i2), the edges (i0, i1), (i1, i2), (i2, i0) and
// adds each end to the other's list unless present.  A pixel's vertex has its
// triangles in the four blocks around the pixel, and its neighbours among the
// eight pixels around it, so walking those blocks in order, with one bit per
// neighbour, gives the list without building it: the two radix sorts of the six
// directed edge events per triangle took 0.95 of the 1.24 ms of kernels of a
// 1280x960 map, this takes 24 us.
__global__ void k_vertex_scales(uint32_t W, uint32_t H, const uint8_t *code, const uint32_t *pix2v, const double *pos,
                                double *scale) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= W * H) return;
    const uint32_t v = pix2v[p];
    if (v == NONE) return;
    const uint32_t px = p % W, py = p / W;
    const double c[3] = {pos[3 * (size_t)v], pos[3 * (size_t)v + 1], pos[3 * (size_t)v + 2]};
    uint32_t seen = 0, count = 0;   // bit 3 (dy + 1) + dx + 1 of a neighbour at (px + dx, py + dy)
    double sum = 0.0;
    for (int k = 0; k < 4; ++k) {
        // the block whose pixel 3 - k (of 0 1 / 2 3) this is
        const int me = 3 - k, ox = me % 2, oy = me / 2;
        if ((int)px < ox || (int)py < oy || px - ox >= W - 1 || py - oy >= H - 1) continue;
        const uint32_t t2 = code[(W - 1) * (py - oy) + px - ox];
        if (t2 == 0xFFu) continue;
        for (int i = 0; i < 2; ++i) {
            const uint32_t t = (t2 >> (4 * i)) & 0xFu;
            if (t == 0xFu) continue;
            for (int e = 0; e < 3; ++e) {
                const int a = c_block_tris[t][e], b = c_block_tris[t][(e + 1) % 3];
                if (a != me && b != me) continue;
                const int o = a == me ? b : a, dx = o % 2 - ox, dy = o / 2 - oy;
                const uint32_t bit = 1u << (3 * (dy + 1) + dx + 1);
                if (seen & bit) continue;
                seen |= bit;
                ++count;
                const uint32_t q = pix2v[(size_t)(py + dy) * W + px + dx];
                const double d[3] = {__dsub_rn(pos[3 * (size_t)q], c[0]), __dsub_rn(pos[3 * (size_t)q + 1], c[1]),
                                     __dsub_rn(pos[3 * (size_t)q + 2], c[2])};
                sum = __dadd_rn(sum, length3(d));
            }
        }
    }
    scale[v] = count == 0 ? -REAL_MAX : __ddiv_rn(sum, (double)count);
}

template <class T>
void excl_scan(const T *in, T *out, uint32_t n, cudaStream_t st) {
    size_t tmp = 0;
    TSR_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, in, out, n, st));
    DBuf<uint8_t> t(tmp, st);
    TSR_CUDA(cub::DeviceScan::ExclusiveSum(t.p, tmp, in, out, n, st));
}

}  // namespace

void triangulate_depth(const double *depths_host, uint32_t W, uint32_t H, const double *hps_to_ray_vs,
                       const double *hps_to_ray_ws, const double *center, const double *colors_host, tsr_mesh &m) {
    cudaStream_t st = m.stream;
    const uint64_t np64 = (uint64_t)W * H;
    if (W < 2 || H < 2) fail(TSR_ERR_INVALID_ARG, "a depth map needs at least 2 x 2 pixels");
    // up to 2 triangles, so 6 corners, per pixel: their 32-bit indices would hold twice this
    // limit, which is the one that callers know
    if (12 * np64 >= NONE) fail(TSR_ERR_OVERFLOW_U32, "depth map too large: 2^32 / 12 pixels at most");
    const uint32_t np = (uint32_t)np64, nblocks = (W - 1) * (H - 1);
    Mat3 Mvs, Mws;
    for (int i = 0; i < 9; ++i) {
        Mvs.m[i] = hps_to_ray_vs[i];
        Mws.m[i] = hps_to_ray_ws[i];
    }
    DBuf<double> depths(np, st), colors;
    TSR_CUDA(cudaMemcpyAsync(depths.p, depths_host, 8ull * np, cudaMemcpyHostToDevice, st));
    if (colors_host) {
        colors.alloc(3ull * np, st);
        TSR_CUDA(cudaMemcpyAsync(colors.p, colors_host, 24ull * np, cudaMemcpyHostToDevice, st));
    }
    // ---- triangles per block, corners, first uses
    DBuf<uint8_t> code(nblocks, st);
    DBuf<uint32_t> ntri(nblocks + 1, st), toff(nblocks + 1, st), first(np, st);
    TSR_CUDA(cudaMemsetAsync(ntri.p + nblocks, 0, 4, st));
    first.fill_bytes(0xFF);
    k_classify_blocks<<<grid_for(nblocks, BLK), BLK, 0, st>>>(depths.p, W, H, Mvs, code.p, ntri.p); ::tsr::note_launch();
    excl_scan(ntri.p, toff.p, nblocks + 1, st);
    const uint32_t nt = read_scalar(toff.p + nblocks, st), nc = 3 * nt;
    DBuf<uint32_t> corner_pix(nc, st), flag(nc + 1, st), rank(nc + 1, st);
    m.pix2v.alloc(np, st);
    m.width = W;
    m.height = H;
    m.tris.alloc(nc, st);
    if (nt) {
        k_emit_corners<<<grid_for(nblocks, BLK), BLK, 0, st>>>(W, H, code.p, toff.p, corner_pix.p, first.p); ::tsr::note_launch();
        k_first_flags<<<grid_for(nc, BLK), BLK, 0, st>>>(nc, corner_pix.p, first.p, flag.p); ::tsr::note_launch();
    }
    TSR_CUDA(cudaMemsetAsync(flag.p + nc, 0, 4, st));
    excl_scan(flag.p, rank.p, nc + 1, st);
    const uint32_t nv = read_scalar(rank.p + nc, st);
    k_pixel_vertices<<<grid_for(np, BLK), BLK, 0, st>>>(np, first.p, rank.p, m.pix2v.p); ::tsr::note_launch();
    if (nt) k_corner_vertices<<<grid_for(nc, BLK), BLK, 0, st>>>(nc, corner_pix.p, m.pix2v.p, m.tris.p); ::tsr::note_launch();
    m.n_tris = nt;
    m.n_verts = nv;
    m.n_cells = 0;
    // ---- vertex positions and colours
    m.vpos.alloc(3ull * nv, st);
    m.vcol.alloc(3ull * nv, st);
    m.vscale.alloc(nv, st);
    m.vkeys.alloc(2ull * nv, st);
    m.vkeys.fill_bytes(0xFF);
    m.vnrm.alloc(3ull * nv, st);
    m.vnrm.zero();
    k_depth_vertices<<<grid_for(np, BLK), BLK, 0, st>>>(W, np, m.pix2v.p, depths.p, Mws, center[0], center[1], center[2],
                                                        colors.p, m.vpos.p, m.vcol.p); ::tsr::note_launch();
    // ---- normals (createFlexibleMesh: computeNormalsWeightedByAngles)
    angle_weighted_normals(m.tris.p, nt, m.vpos.p, nv, m.vnrm.p, st);
    // ---- scales: the mean distance to the neighbours
    if (nv) {
        k_vertex_scales<<<grid_for(np, BLK), BLK, 0, st>>>(W, H, code.p, m.pix2v.p, m.vpos.p, m.vscale.p);
        ::tsr::note_launch();
    }
    TSR_CUDA(cudaStreamSynchronize(st));
    TSR_CUDA(cudaGetLastError());
}

}  // namespace tsr
