// occupancy.cu -- sm_100a occupancy field of the TSR volumetric core.
//
// Reproduces Occupancy::computeOccupancy (SurfaceExtraction/Occupancy.cpp:
// 105-127): the SAMPLENESS and EMPTINESS cone-kernel passes over every
// camera-to-sample link (updateKernels :138-248, addKernel :279-346), the
// bottom-up SAMPLENESS flag propagation (forwardAnyChildStateFlag :491-516),
// the semi-local Bayesian priors (computePriors :530-568) and the per-leaf
// occupancy value (getOccupancy :570-587).
//
// Precision: the per-link cone set-up, the depth cap, the cone length and the
// cone count are FP64 (as the reference's Real = double); kernel evaluation
// runs in FP32 in a frame centred on the sample, and every per-leaf sum is an
// FP64 accumulator updated by FP64 atomic adds whose result is not used (no
// round trip per accepted pair).  Priors and occupancy are evaluated in FP64.
// Which leaves a prior sums is decided by FP32 distances where those are certain
// (exact on the lattice of box corners, or outside their error bound) and by the
// tree build's FP64 expression everywhere else, so the set is exact.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

#include "handles.h"

namespace tsr {
namespace {

constexpr unsigned BLK = 256;
enum { EMPTINESS = 0, SAMPLENESS = 1 };

struct F3 {
    float x, y, z;
};
__device__ inline F3 f3(float x, float y, float z) { return F3{x, y, z}; }
__device__ inline F3 operator-(F3 a, F3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ inline F3 operator+(F3 a, F3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ inline F3 operator*(F3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ inline float fdot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// Cone in the sample-centred FP32 frame.  t is measured from the end disc:
// te = dot(x - end, m) / denom = tComplete - 1, which keeps the arithmetic
// near the sample (where the kernels are evaluated) well conditioned.
struct ConeF {
    F3 end, axis, m;   // m = end-disc normal
    float radius, full, inv_denom, a_over_l, t_start_e;
    float ray_k;       // 3 / (2 L), L = cone length
    float n1;          // |m|_1
};

struct LinkIn {
    const D3 *pos, *nrm;
    const double *scale, *conf;
    const uint32_t *links;
    const D3 *cams;
    uint32_t k, ncams;
    double h_svo, h_o, rel_cone, root_size;
};

struct TreeIn {
    const D3 *nmin;   // node min corners (FP64), for the start-node descent
};


// Occupancy::addKernel (Occupancy.cpp:279-346) at a leaf centre x, given
// te = dot(x - end, m) / denom (= tComplete - 1) and r2 = |x - PCD centre|^2:
// the confidence-scaled kernel value, or 0 where addKernel adds nothing.
// Straight-line code (no early exits), so that the lanes of a warp testing
// different children stay together.  Which products are fused is written out
// here and below, since it is part of the result: the sums do not change with
// the code around it.
__device__ __forceinline__ float kernel_value(const ConeF &c, float te, float r2, bool sampleness, float conf) {
    const float tcut_m1 = __fmul_rn(te, c.a_over_l);                 // tCut - 1
    const float tcut = __fmaf_rn(te, c.a_over_l, 1.0f);
    const float pr = __fmul_rn(c.radius, __fadd_rn(1.0f, te));       // PCD radius at tComplete
    const float pr2 = __fmul_rn(pr, pr);
    bool ok = (tcut >= 0.0f) & (tcut < 1.0f) & (r2 < pr2);
    float f;   // ray factor: 3/(2Z)(1 - (z/Z)^2) with the 3/(2 L) part in ray_k
    if (sampleness) {
        const float tcen = __fmul_rn(fabsf(__fadd_rn(tcut, -0.5f)), 2.0f);
        f = __fmaf_rn(-tcen, tcen, 1.0f);
        ok &= tcen < 1.0f;
    } else {
        f = __fmul_rn(-tcut_m1, __fadd_rn(1.0f, tcut));              // (1 - tCut)(1 + tCut)
    }
    const float inv = __frcp_rn(pr2);
    const float kv = __fmul_rn(__fmul_rn(__fmul_rn(c.ray_k, f), __fmul_rn(0.63661977236758134f, inv)),
                               __fmaf_rn(-r2, inv, 1.0f));
    const float scaled = __fmul_rn(conf, kv);
    ok &= (kv >= (float)EPS) & (scaled >= (float)EPS);
    return ok ? scaled : 0.0f;
}

// The offset q of u = x - end from the axis point of the same te, and |q|^2.
__device__ __forceinline__ void axis_offset(const ConeF &c, F3 u, float te, F3 &q, float &r2) {
    q = f3(__fmaf_rn(-c.axis.x, te, u.x), __fmaf_rn(-c.axis.y, te, u.y), __fmaf_rn(-c.axis.z, te, u.z));
    r2 = __fmaf_rn(q.z, q.z, __fmaf_rn(q.x, q.x, __fmul_rn(q.y, q.y)));
}

// Cone-frame coordinates of point x: te, the offset q from the axis point of
// the same te, and |q|^2.
__device__ __forceinline__ void cone_coords(const ConeF &c, F3 x, float &te, F3 &q, float &r2) {
    const F3 u = x - c.end;
    te = __fmul_rn(__fmaf_rn(u.z, c.m.z, __fmaf_rn(u.x, c.m.x, __fmul_rn(u.y, c.m.y))), c.inv_denom);
    axis_offset(c, u, te, q, r2);
}

// The same for the centre of child ci of a traversed node.  Unfused products in
// the SAMPLENESS pass, and in the EMPTINESS pass a fused last product for the
// first five children only: no numerical reason, the two are equally accurate,
// but this is how the kernel that defined the field's values was rounded, and a
// field keeps its values, bit for bit per link, from one version to the next.
template <int TYPE>
__device__ __forceinline__ void child_coords_of(const ConeF &c, uint32_t ci, F3 x, float &te, F3 &q, float &r2) {
    const F3 u = x - c.end;
    float dot;
    if (TYPE == SAMPLENESS) {
        dot = __fadd_rn(__fadd_rn(__fmul_rn(u.x, c.m.x), __fmul_rn(u.y, c.m.y)), __fmul_rn(u.z, c.m.z));
    } else {
        const float xy = __fmaf_rn(u.x, c.m.x, __fmul_rn(u.y, c.m.y));
        dot = ci < 5 ? __fmaf_rn(u.z, c.m.z, xy) : __fadd_rn(xy, __fmul_rn(u.z, c.m.z));
    }
    te = __fmul_rn(dot, c.inv_denom);
    axis_offset(c, u, te, q, r2);
}

__device__ inline float eval_kernel(const ConeF &c, F3 x, bool sampleness, float conf) {
    float te, r2;
    F3 q;
    cone_coords(c, x, te, q, r2);
    return kernel_value(c, te, r2, sampleness, conf);
}

__device__ inline F3 rel(const D3 &a, const D3 &origin) {
    return f3((float)(a.x - origin.x), (float)(a.y - origin.y), (float)(a.z - origin.z));
}

// ------------------------------------------------------ cone traversal
// Conservative cone/box rejection (stands in for ObliqueCircularCone::
// haveSeparatingAxis, ConeNodesChecker.cpp:65).  Pruning can only skip boxes
// that contain no point of the cut cone, so the sums do not depend on it.
// Conservative box test with an absolute slack for the FP32 box recurrence.
__device__ inline bool cone_box_separated_pt(const ConeF &c, F3 bmin, float size) {
    float h = 0.5f * size;
    F3 ctr = bmin + f3(h, h, h);
    float mag = fabsf(ctr.x) + fabsf(ctr.y) + fabsf(ctr.z);
    float hs = h + 2e-6f * mag;
    F3 u = ctr - c.end;
    float te = fdot(u, c.m) * c.inv_denom;
    float dt = hs * c.n1 * fabsf(c.inv_denom);
    float slack = 1e-4f * (dt + fabsf(te)) + 1e-6f;
    if (te + dt < c.t_start_e - slack) return true;
    if (te - dt >= slack) return true;
    if (1.0f + te + dt <= 0.0f) return true;
    F3 q = u - c.axis * te;
    float qn = sqrtf(fdot(q, q));
    float tmax = fminf(1.0f + te + dt, 1.0f);
    float bound = qn - hs * 1.7320508f - dt * c.full;
    return bound > tmax * c.radius * 1.0001f + 1e-4f * (qn + hs + dt * c.full);
}

// The same test for a box of centre coordinates (te, q, r2 = |q|^2; q is
// the offset from the axis point of the same te) and half size hs already
// widened by the recurrence slack; dt = hs * |m|_1 * |1/denom|.  A box point
// ctr + d has te + (d.m)/denom and offset q + d - axis (d.m)/denom, whose
// length is at least |q| + d.w with w = (q - (q.axis / denom) m) / |q|, so
// every box point is at least |q| - hs |w|_1 from the axis: the exact
// support of the box in that direction, with the axis shift over the box's
// te range folded in.  Straight-line code; |q| = 0 never separates.
__device__ __forceinline__ bool separated_at(const ConeF &c, float te, F3 q, float r2, float hs, float dt) {
    const float slack = 1e-4f * (dt + fabsf(te)) + 1e-6f;
    bool sep = (te + dt < c.t_start_e - slack) | (te - dt >= slack) | (1.0f + te + dt <= 0.0f);
    const float tmax = fminf(1.0f + te + dt, 1.0f);
    const float inv = rsqrtf(r2);
    const float qn = r2 * inv;
    const F3 v = q - c.m * (fdot(q, c.axis) * c.inv_denom);
    const float v1 = fabsf(v.x) + fabsf(v.y) + fabsf(v.z);
    const float rest = tmax * c.radius * 1.0001f + 1e-4f * (hs + dt * c.full);
    sep |= (qn * 0.9999f - hs * v1 * inv) > rest;
    return sep;
}

// Resident blocks per SM the traversals are compiled for (the register
// budget: 65536 / (128 threads x blocks)).
#ifndef TSR_CONE_BLOCKS
#define TSR_CONE_BLOCKS 8
#endif
#ifndef TSR_PRIOR_BLOCKS
#define TSR_PRIOR_BLOCKS 4
#endif

// Node records: rec[i + 7] = (first child or INVALID, leaf index, with the
// node's SAMPLENESS flag in bit 31).  Children blocks start at 1 + 8k (root 0,
// then whole blocks of 8), so a block's records start on a 64-byte boundary.
// An inner node's second word holds REC_INNER with two bits of what its
// children block has: leaves and inner nodes (flagged ones, once there are
// flags).
constexpr uint32_t REC_FLAG = 0x80000000u, REC_NOLEAF = 0x7FFFFFFFu;
constexpr uint32_t REC_INNER = 0x7FFFFFFCu, REC_HAS_LEAVES = 1u, REC_HAS_INNER = 2u;
constexpr uint32_t REC_OFFSET = 7;

__global__ void k_pack_rec(uint32_t nn, const uint32_t *children, const uint32_t *node_to_leaf,
                           const uint32_t *states, uint2 *rec) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    uint32_t c = children[i];
    uint32_t y = (c == INVALID) ? node_to_leaf[i] : REC_INNER;
    if (states && (states[i] & FLAG_SAMPLENESS)) y |= REC_FLAG;
    if (c != INVALID)
        for (uint32_t k = 0; k < 8; ++k)
            if (!states || (states[c + k] & FLAG_SAMPLENESS))
                y |= children[c + k] == INVALID ? REC_HAS_LEAVES : REC_HAS_INNER;
    rec[i + REC_OFFSET] = make_uint2(c, y);
}

// Pruned field: which leaves need their prior.  Only a reliable leaf
// (E + S >= confidenceThreshold) uses it, and with E == 0 or S == 0 its sign
// is fixed without it (need 0).  A leaf near a predicted sign change
// (PRED_KEEP), or one whose sign the network is unsure of, is queried
// (need 1); any other leaf is a candidate for skipping (need 2): its sign is
// then certified from bounds of its prior (k_certify) or it is queried after
// all.
constexpr uint8_t NEED_NONE = 0, NEED_QUERY = 1, NEED_CERTIFY = 2;


__global__ void k_prior_needed(uint32_t nl, const uint8_t *pred, const double *esum, const double *ssum,
                               double threshold, uint8_t *need) {
    uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    const double e = esum[l], s = ssum[l];
    const uint8_t pr = pred[l];
    uint8_t n = NEED_NONE;
    if (!((e + s) < threshold) && e > 0.0 && s > 0.0)
        n = ((pr & PRED_KEEP) || !(pr & (PRED_POS | PRED_NEG))) ? NEED_QUERY : NEED_CERTIFY;
    else if (!((e + s) < threshold) && (pr & PRED_KEEP))
        n = NEED_QUERY;
    need[l] = n;
}

// The sign of a skip candidate from bounds [lo, hi] of its prior p: the
// occupancy is positive iff (1 - p) S > p E (Occupancy.cpp:570-587; the
// common factor 1 / coneCount dropped), which decreases in p.  Positive when
// it holds at p = hi, negative when it fails at p = lo, each with a relative
// margin of 1e-9 that covers the rounding of the sums and of the exact
// formula; otherwise the leaf is queried (need 1).  A certified leaf's sign
// goes to its PRED_POS / PRED_NEG bits, which the pruned k_finalize uses.
//
// A positive leaf's value (1 - p) S / coneCount - p E / coneCount is also
// placed against EPSILON when the bounds decide it (PRED_HIGH / PRED_LOW,
// same margin): DMC snaps a vertex to the end of an edge whose value is
// within EPSILON of zero, and a negative leaf's value is -EPSILON, so that
// side is all the mesh takes from a positive leaf's value.
__global__ void k_certify(uint32_t nl, const double *esum, const double *ssum, const double2 *bounds,
                          const double *cone_count, uint8_t *pred, uint8_t *need, unsigned long long *certified) {
    const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    bool ok = false;
    if (l < nl && need[l] == NEED_CERTIFY) {
        const double e = esum[l], s = ssum[l];
        const double2 b = bounds[l];
        const double margin = 1e-9 * (s + e);
        const double at_hi = (1.0 - b.y) * s - b.y * e, at_lo = (1.0 - b.x) * s - b.x * e;
        const bool pos = at_hi > margin;
        const bool neg = at_lo < -margin;
        const uint8_t keep = pred[l] & PRED_KEEP;
        const double eps_cc = EPS * *cone_count;
        if (pos) pred[l] = keep | PRED_POS | (at_hi > eps_cc + margin ? PRED_HIGH : 0) |
                           (at_lo < eps_cc - margin ? PRED_LOW : 0);
        else if (neg) pred[l] = keep | PRED_NEG;
        ok = pos || neg;
        need[l] = ok ? NEED_NONE : NEED_QUERY;
    }
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(certified, (unsigned long long)__popc(m));
}

// Per-link set-up of the traversal, precomputed by one thread per link so
// that the persistent traversal below never runs this long FP64 stretch for a
// few lanes of a warp while the others wait.  c0 == INVALID: nothing to
// traverse (no camera, degenerated cone, pruned start, or a start leaf that
// the set-up kernel has already visited).
struct __align__(16) LinkRec {
    float end[3], axis[3], m[3];
    float radius, full, ray_k, inv_denom, a_over_l, t_start_e, n1;
    float smin[3], fconf;     // start node corner in the sample's frame; confidence
    double wlen;              // confidence * cone length
    uint32_t c0;              // children block of the start node
    uint32_t depths;          // depth of those children | max depth << 8
    double spos[3];           // the sample: origin of the FP32 frame
    uint32_t has;             // what the children block has (REC_HAS_LEAVES, REC_HAS_INNER)
    uint32_t pad;
};
static_assert(sizeof(LinkRec) == 128, "copied as eight 16-byte words");

// Set-up of link order[i] (Occupancy.cpp:174-201), FP64, and the start of its
// traversal: the deepest node containing the cut cone's bounding box.
// sign: +1 adds the links' kernels, -1 removes them (Occupancy::updateKernels
// with forRemoval, Occupancy.cpp:138-248: the same acceptance, negated
// values, cone lengths and cone count).
template <int TYPE>
__global__ void __launch_bounds__(128) k_link_setup(uint64_t nlinks, const uint32_t *order, LinkIn in, TreeIn tr,
                                                    const uint2 *rec, LinkRec *out, double *ksum, double *clen,
                                                    double *cone_count, unsigned long long *accepted, double sign) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double count = 0.0;
    unsigned long long acc = 0;
    if (i < nlinks) {
        LinkRec r;
        r.c0 = INVALID;
        r.depths = 0;
        do {
            uint64_t l = order ? order[i] : i;
            uint32_t s = (uint32_t)(l / in.k);
            uint32_t cam = in.links[l];
            if (cam == INVALID || cam >= in.ncams) break;
            D3 p = in.pos[s];
            D3 n = in.nrm[s];
            D3 cwp = in.cams[cam];
            double kernel_r = in.h_o * in.scale[s];
            D3 apex_d{cwp.x - p.x, cwp.y - p.y, cwp.z - p.z};
            D3 end_d{0.0, 0.0, 0.0};
            double cone_len = REAL_MAX;
            if (TYPE == SAMPLENESS) {
                D3 cs{-apex_d.x, -apex_d.y, -apex_d.z};
                double total = sqrt(cs.x * cs.x + cs.y * cs.y + cs.z * cs.z);
                cone_len = kernel_r * in.rel_cone;
                double hh = cone_len * 0.5;
                end_d = D3{cs.x / total * hh, cs.y / total * hh, cs.z / total * hh};
            }
            D3 m{-n.x, -n.y, -n.z};
            D3 axis{end_d.x - apex_d.x, end_d.y - apex_d.y, end_d.z - apex_d.z};
            double full = sqrt(axis.x * axis.x + axis.y * axis.y + axis.z * axis.z);
            double length = cone_len < full ? cone_len : full;
            double denom = axis.x * m.x + axis.y * m.y + axis.z * m.z;
            if (!(full > EPS) || !(kernel_r > 0.0) || fabs(denom) <= EPS * full) break;   // isDegenerated
            double conf = in.conf[s];
            if (TYPE == EMPTINESS) count += sign * conf;
            const double wlen = conf * length;
            const float fconf = (float)conf;
            const uint32_t max_depth =
                (uint32_t)ceil(log2(in.root_size / (in.scale[s] * in.h_svo))) + MAX_DEPTH_DIFFERENCE;
            ConeF c;
            c.end = f3((float)end_d.x, (float)end_d.y, (float)end_d.z);
            c.axis = f3((float)axis.x, (float)axis.y, (float)axis.z);
            c.m = f3((float)m.x, (float)m.y, (float)m.z);
            c.radius = (float)kernel_r;
            c.full = (float)full;
            c.ray_k = (float)(1.5 / length);
            c.inv_denom = (float)(1.0 / denom);
            c.a_over_l = (float)(full / length);
            c.t_start_e = (float)(-length / full);
            c.n1 = fabsf(c.m.x) + fabsf(c.m.y) + fabsf(c.m.z);
            F3 p0 = c.end + c.axis * c.t_start_e;
            F3 lo = f3(fminf(p0.x, c.end.x) - c.radius, fminf(p0.y, c.end.y) - c.radius, fminf(p0.z, c.end.z) - c.radius);
            F3 hi = f3(fmaxf(p0.x, c.end.x) + c.radius, fmaxf(p0.y, c.end.y) + c.radius, fmaxf(p0.z, c.end.z) + c.radius);
            const float root_size_f = (float)in.root_size;
            uint32_t start = 0, base = 0;
            uint2 srec = __ldg(&rec[REC_OFFSET]);
            F3 smin = rel(tr.nmin[0], p);
            float ssize = root_size_f;
            while (srec.x != INVALID && base + 1 <= max_depth) {
                float cs = 0.5f * ssize;
                float margin = 1e-5f * ssize;
                F3 ctr = smin + f3(cs, cs, cs);
                const float l3[3] = {lo.x, lo.y, lo.z}, h3[3] = {hi.x, hi.y, hi.z}, c3[3] = {ctr.x, ctr.y, ctr.z};
                uint32_t digit = 0;
                bool inside = true;
                for (int a = 0; a < 3; ++a) {
                    if (h3[a] < c3[a] - margin) continue;
                    if (l3[a] > c3[a] + margin) { digit |= 1u << a; continue; }
                    inside = false;
                }
                if (!inside) break;
                start = srec.x + digit;
                srec = __ldg(&rec[start + REC_OFFSET]);
                smin = rel(tr.nmin[start], p);
                ssize = cs;
                ++base;
            }
            if (TYPE == EMPTINESS && !(srec.y & REC_FLAG)) break;
            if (cone_box_separated_pt(c, smin, ssize)) break;
            if (srec.x == INVALID) {   // the start is a leaf: visit it here
                float h = 0.5f * ssize;
                float val = eval_kernel(c, smin + f3(h, h, h), TYPE == SAMPLENESS, fconf);
                if (val > 0.0f) {
                    uint32_t leaf = srec.y & REC_NOLEAF;
                    atomicAdd(&ksum[leaf], sign * (double)val);
                    atomicAdd(&clen[leaf], sign * wlen);
                    ++acc;
                }
                break;
            }
            if (base + 1 > max_depth) break;
            r.end[0] = c.end.x; r.end[1] = c.end.y; r.end[2] = c.end.z;
            r.axis[0] = c.axis.x; r.axis[1] = c.axis.y; r.axis[2] = c.axis.z;
            r.m[0] = c.m.x; r.m[1] = c.m.y; r.m[2] = c.m.z;
            r.radius = c.radius; r.full = c.full; r.ray_k = c.ray_k; r.inv_denom = c.inv_denom;
            r.a_over_l = c.a_over_l; r.t_start_e = c.t_start_e; r.n1 = c.n1;
            r.smin[0] = smin.x; r.smin[1] = smin.y; r.smin[2] = smin.z;
            r.fconf = fconf;
            r.wlen = sign * wlen;
            r.c0 = srec.x;
            r.depths = (base + 1) | (max_depth << 8);
            r.spos[0] = p.x; r.spos[1] = p.y; r.spos[2] = p.z;
            r.has = srec.y & (REC_HAS_LEAVES | REC_HAS_INNER);
            r.pad = 0;
        } while (0);
        out[i] = r;
    }
    typedef cub::BlockReduce<double, 128> BR;
    typedef cub::BlockReduce<unsigned long long, 128> BRU;
    __shared__ typename BR::TempStorage tmp;
    __shared__ typename BRU::TempStorage tmpu;
    double bc = BR(tmp).Sum(count);
    unsigned long long ba = BRU(tmpu).Sum(acc);
    if (threadIdx.x == 0) {
        if (TYPE == EMPTINESS && bc != 0.0) atomicAdd(cone_count, bc);
        if (ba) atomicAdd(accepted, ba);
    }
}

// ------------------------------------------- cone traversal
// The links' depth-first traversals (the per-link LeavesIterator with a
// ConeNodesChecker), a warp taking CX_LINKS links at a time.  The blocks of
// children to visit lie on one stack per warp, whichever link they belong to,
// and a step takes four of them, one child a lane: every lane works whatever
// the links' lengths, and one long link is shared by all lanes.  (A lane per
// link left 8 of 32 lanes busy at 300k samples and 21 at 16M, and ended on the
// longest link.)  The links' cones lie in shared memory.  As in the prior
// queries there are two kinds of steps: inner nodes get the box test, and
// their children blocks go on the stack; leaves get the kernel.
//
// Measured, SAMPLENESS + EMPTINESS pass: 14 + 24 -> 2.3 + 5.3 ms at 300k
// held-out samples, 20 + 30 -> 15 + 27 ms at 4M CSG, 99 + 247 -> 59 + 190 ms
// at 16M held-out.  What bounds it is instruction issue (3.2 of 4 a clock).
//
// The FP32 arithmetic of a child's box is part of the result, so it follows
// one rule: the first surviving child's corner comes from its parent's by the
// FP32 recurrence, every other one's from the FP64 tree.  Like the rounding in
// child_coords_of it keeps a link's values what they were; it carries no accuracy.
//
// Leaf flags are not written here: a leaf got a kernel exactly when its sum is
// non-zero (every accepted value is >= EPSILON), so they are set afterwards
// from the sums.
constexpr int CX_LINKS = 8;
constexpr int CX_WIDE = 96;     // from here on a step takes one block, which adds at most 7 a level
constexpr int CX_LEAVES = 64;   // blocks whose leaves wait; worked off when fewer than 32 are free
constexpr int CX_WARPS = 4;

// A warp's stack entries for a tree of that depth: a wide step leaves at most
// CX_WIDE + 28, a narrow one adds 7 a level.
inline uint32_t cone_stack(uint32_t tree_depth) { return (CX_WIDE + 28 + 7 * tree_depth + 8 + 7) & ~7u; }

struct ConeWarp {
    float4 link[CX_LINKS][9];       // LinkRec; the ninth word keeps four links' words in different banks
    float4 leaf_box[CX_LEAVES];     // a block's corner (the link's frame) and index
    uint16_t leaf_tag[CX_LEAVES];   // its link's place, and its nodes' depth << 3
    float4 box[1];                  // the stack, of the tree's depth; its tags follow
};

inline size_t cone_warp_bytes(uint32_t stack) {
    return (offsetof(ConeWarp, box) + stack * (sizeof(float4) + sizeof(uint16_t)) + 15) & ~(size_t)15;
}

__device__ __forceinline__ ConeF cone_of(const float4 *l) {
    const float4 a = l[0], b = l[1], c = l[2], d = l[3];
    ConeF k;
    k.end = f3(a.x, a.y, a.z);
    k.axis = f3(a.w, b.x, b.y);
    k.m = f3(b.z, b.w, c.x);
    k.radius = c.y;
    k.full = c.z;
    k.ray_k = c.w;
    k.inv_denom = d.x;
    k.a_over_l = d.y;
    k.t_start_e = d.z;
    k.n1 = d.w;
    return k;
}

template <int TYPE>
__global__ void __launch_bounds__(32 * CX_WARPS, TSR_CONE_BLOCKS)
    k_cones(uint64_t nlinks, uint32_t per, uint32_t stack, uint32_t warp_bytes, const LinkRec *links, TreeIn tr,
            const uint2 *rec, float root_size_f, double *ksum, double *clen, unsigned long long *accepted,
            unsigned long long *next_link, unsigned long long *visits, int *err, double sign) {
    const unsigned FULL = 0xffffffffu;
    extern __shared__ float4 cone_shared[];
    __shared__ float sizes[64];     // edge length of a node at a depth
    ConeWarp &w =
        *reinterpret_cast<ConeWarp *>(reinterpret_cast<char *>(cone_shared) + (threadIdx.x >> 5) * warp_bytes);
    float4 *const stack_box = w.box;
    uint16_t *const stack_tag = reinterpret_cast<uint16_t *>(w.box + stack);
    const unsigned lane = threadIdx.x & 31, below = (1u << lane) - 1u, ci = lane & 7u;
    const int quarter = (int)(lane >> 3);
    const float bx = (float)(ci & 1u), by = (float)((ci >> 1) & 1u), bz = (float)(ci >> 2), fsign = (float)sign;
    if (threadIdx.x < 64) sizes[threadIdx.x] = ldexpf(root_size_f, -(int)threadIdx.x);
    __syncthreads();
    uint32_t hits = 0, expanded = 0;   // of this lane, since the last links
    unsigned long long acc = 0, nvis = 0;
    int sp = 0, waiting = 0;
    while (true) {
        if (sp == 0 && waiting == 0) {
            acc += hits;
            nvis += 8ull * expanded;
            hits = expanded = 0;
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(next_link, (unsigned long long)per);
            base = __shfl_sync(FULL, base, 0);
            if (base >= nlinks) break;
            const uint32_t n = (uint32_t)min((unsigned long long)per, nlinks - base);
            const float4 *src = reinterpret_cast<const float4 *>(links + base);
            for (uint32_t i = lane; i < 8 * n; i += 32) w.link[i >> 3][i & 7] = __ldg(src + i);
            __syncwarp();
            bool start = false;
            uint32_t has = 0;
            float4 box = make_float4(0.f, 0.f, 0.f, 0.f);
            uint16_t tag = 0;
            if (lane < n) {
                const LinkRec &r = *reinterpret_cast<const LinkRec *>(w.link[lane]);
                if (r.c0 != INVALID) {
                    start = true;
                    has = r.has;
                    box = make_float4(r.smin[0], r.smin[1], r.smin[2], __uint_as_float((r.c0 - 1) >> 3));
                    tag = (uint16_t)(lane | ((r.depths & 0xFFu) << 3));
                }
            }
            const bool push = start && (has & REC_HAS_INNER), wait = start && (has & REC_HAS_LEAVES);
            const unsigned pm = __ballot_sync(FULL, push), wm = __ballot_sync(FULL, wait);
            if (push) {
                const int j = __popc(pm & below);
                stack_box[j] = box;
                stack_tag[j] = tag;
            }
            if (wait) {
                const int j = __popc(wm & below);
                w.leaf_box[j] = box;
                w.leaf_tag[j] = tag;
            }
            sp = __popc(pm);
            waiting = __popc(wm);
            expanded += start;
            __syncwarp();
            continue;
        }
        if (waiting > CX_LEAVES - 32 || sp == 0) {
            // ---- the leaves of the waiting blocks: addKernel's exact test decides, no box test needed
            do {
                const bool valid = quarter < waiting;
                const int at = valid ? waiting - 1 - quarter : 0;
                const float4 b = w.leaf_box[at];
                const uint32_t tag = w.leaf_tag[at];
                const uint2 r = __ldg(&rec[1 + 8 * __float_as_uint(b.w) + ci + REC_OFFSET]);
                const float4 *l = w.link[tag & 7u];
                const ConeF c = cone_of(l);
                const float size = sizes[tag >> 3], h = 0.5f * size;
                const F3 ctr0 = f3(b.x, b.y, b.z) + f3(h, h, h);
                const F3 ctr = f3(fmaf(bx, size, ctr0.x), fmaf(by, size, ctr0.y), fmaf(bz, size, ctr0.z));
                float te, r2;
                F3 q;
                child_coords_of<TYPE>(c, ci, ctr, te, q, r2);
                const float val = kernel_value(c, te, r2, TYPE == SAMPLENESS, l[4].w);
                const bool hit = valid && r.x == INVALID && (TYPE == SAMPLENESS || (r.y & REC_FLAG)) && val > 0.0f;
                if (hit) {
                    const uint32_t lf = r.y & REC_NOLEAF;
                    const double wlen = *reinterpret_cast<const double *>(l + 5);   // carries the sign
                    atomicAdd(&ksum[lf], (double)(fsign * val));
                    atomicAdd(&clen[lf], wlen);
                    ++hits;
                }
                waiting -= 4;
            } while (waiting >= 4 || (waiting > 0 && sp == 0));
            if (waiting < 0) waiting = 0;
            __syncwarp();
            continue;
        }
        // ---- the inner nodes of the blocks on top of the stack
        const int take = sp > CX_WIDE ? 1 : (sp < 4 ? sp : 4);
        const bool valid = quarter < take;
        const int at = sp - 1 - (valid ? quarter : 0);
        const float4 b = stack_box[at];
        const uint32_t tag = stack_tag[at], d = tag >> 3;
        sp -= take;
        const uint32_t node = 1 + 8 * __float_as_uint(b.w) + ci;
        const uint2 r = __ldg(&rec[node + REC_OFFSET]);
        const LinkRec *l = reinterpret_cast<const LinkRec *>(w.link[tag & 7u]);
        const ConeF c = cone_of(w.link[tag & 7u]);
        const float size = sizes[d], h = 0.5f * size;
        const F3 x_min = f3(b.x, b.y, b.z), ctr0 = x_min + f3(h, h, h);
        // one widened half size for all eight boxes: covers the FP32 corner
        // error of every child centre (|centre|_1 <= |x_min|_1 + 4.5 size)
        const float hs = h + 2e-6f * (fabsf(x_min.x) + fabsf(x_min.y) + fabsf(x_min.z) + 4.5f * size);
        const float dt = hs * c.n1 * fabsf(c.inv_denom);
        const F3 ctr = f3(fmaf(bx, size, ctr0.x), fmaf(by, size, ctr0.y), fmaf(bz, size, ctr0.z));
        float te, r2;
        F3 q;
        child_coords_of<TYPE>(c, ci, ctr, te, q, r2);
        const bool sep = separated_at(c, te, q, r2, hs, dt);
        const bool next = valid && r.x != INVALID && (TYPE == SAMPLENESS || (r.y & REC_FLAG)) && !sep &&
                          d + 1 <= (l->depths >> 8);
        const unsigned nm = __ballot_sync(FULL, next);
        float4 box = make_float4(0.f, 0.f, 0.f, 0.f);
        if (next) {
            const bool first = ((nm >> (lane & 24u)) & ((1u << ci) - 1u)) == 0;
            F3 x = f3(fmaf(bx, size, x_min.x), fmaf(by, size, x_min.y), fmaf(bz, size, x_min.z));
            if (!first) x = rel(tr.nmin[node], D3{l->spos[0], l->spos[1], l->spos[2]});
            box = make_float4(x.x, x.y, x.z, __uint_as_float((r.x - 1) >> 3));
        }
        const uint16_t ntag = (uint16_t)(tag + 8);   // one deeper
        const bool push = next && (r.y & REC_HAS_INNER), wait = next && (r.y & REC_HAS_LEAVES);
        const unsigned pm = __ballot_sync(FULL, push), wm = __ballot_sync(FULL, wait);
        if (sp + __popc(pm) > (int)stack) {
            if (lane == 0) atomicExch(err, 1);
        } else {
            if (push) {
                const int j = sp + __popc(pm & below);
                stack_box[j] = box;
                stack_tag[j] = ntag;
            }
            sp += __popc(pm);
        }
        if (wait) {
            const int j = waiting + __popc(wm & below);
            w.leaf_box[j] = box;
            w.leaf_tag[j] = ntag;
        }
        waiting += __popc(wm);
        expanded += next;
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) {
        acc += __shfl_xor_sync(FULL, acc, o);
        nvis += __shfl_xor_sync(FULL, nvis, o);
    }
    if (lane == 0) {
        if (acc) atomicAdd(accepted, acc);
        if (nvis) atomicAdd(visits, nvis);
    }
}

// Pruned field repair: skipped reliable leaves (need == 0, E + S >= the
// threshold) that are positive and share a face with a negative leaf, and
// whose value's side of EPSILON is not proved.  DMC interpolates along
// dual-cell edges, which join face neighbours, so only the two ends of a
// sign change matter; the negative end's value is -EPS whatever its prior
// (Occupancy.cpp:570-587), and with one end at -EPS the vertex snaps to an
// end, decided by whether the positive end's value exceeds EPS
// (DualMarchingCell.cpp:51-71).
__global__ void k_repair_mark(uint32_t nl, const uint32_t *nb_off, const uint32_t *nbs, const double *occ,
                              const uint8_t *need, const uint8_t *pred, const double *esum, const double *ssum,
                              double threshold, uint8_t *mark) {
    uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    auto skipped = [&](uint32_t x) {
        return !need[x] && !((esum[x] + ssum[x]) < threshold) && !(pred[x] & (PRED_HIGH | PRED_LOW));
    };
    const bool pl = occ[l] > 0.0;
    for (uint32_t e = nb_off[l]; e < nb_off[l + 1]; ++e) {
        const uint32_t m = nbs[e];
        if ((occ[m] > 0.0) == pl) continue;
        const uint32_t positive = pl ? l : m;
        if (skipped(positive)) mark[positive] = 1;
    }
}

// The marked leaves become queried ones, counted.
__global__ void k_set_needed(uint32_t nl, const uint8_t *mark, uint8_t *need, uint32_t *count) {
    const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    const bool m = l < nl && mark[l];
    if (m) need[l] = NEED_QUERY;
    const unsigned b = __ballot_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(count, (uint32_t)__popc(b));
}

// A leaf carries a type's flag exactly when it received a kernel of that type.
__global__ void k_leaf_flags(uint32_t nl, const uint32_t *leaf_node, const double *ksum, uint32_t *states,
                             uint32_t flag) {
    uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    if (ksum[l] > 0.0) states[leaf_node[l]] |= flag;
}

// Camera of every listed link (list == null: links 0 .. nlinks-1), as sort keys.
__global__ void k_link_cameras(uint64_t nlinks, const uint32_t *list, const uint32_t *links, uint32_t ncams,
                               uint32_t *keys, uint32_t *vals) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nlinks) return;
    const uint32_t l = list ? list[i] : (uint32_t)i;
    uint32_t c = links[l];
    keys[i] = (c == INVALID || c >= ncams) ? ncams : c;
    vals[i] = l;
}

// The links of the chosen samples: sample s has links s K .. s K + K - 1.
__global__ void k_sample_links(uint32_t count, const uint32_t *samples, uint32_t k, uint32_t *out) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)count * k) return;
    out[i] = samples[i / k] * k + (uint32_t)(i % k);
}

// forwardAnyChildStateFlag, one level bottom-up.
__global__ void k_forward_flag(uint32_t lo, uint32_t hi, const uint32_t *order, const uint32_t *children,
                               uint32_t *states, uint32_t flag) {
    uint32_t i = lo + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= hi) return;
    uint32_t n = order[i];
    uint32_t c0 = children[n];
    if (c0 == INVALID) return;
    uint32_t s = states[n] & ~flag;
    for (uint32_t c = 0; c < 8; ++c)
        if (states[c0 + c] & flag) s |= flag;
    states[n] = s;
}

// Cumulative prior sums per node: psum[k * nn + node] = sum of (emptiness,
// sampleness) cone lengths over SAMPLENESS-flagged leaves of the node's
// subtree at most k levels below the node.  Built bottom-up, one level per
// launch.  Rows are k-major so that the eight siblings of a children block
// share one 128-byte line per k.
constexpr int PK = 8;

__global__ void k_prior_sums(uint32_t lo, uint32_t hi, uint32_t nn, const uint32_t *order,
                             const uint32_t *children, const uint32_t *node_to_leaf, const uint32_t *states,
                             const double *elen, const double *slen, double2 *psum, int *nonfinite) {
    uint32_t i = lo + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= hi) return;
    uint32_t n = order[i];
    uint32_t c0 = children[n];
    if (c0 == INVALID) {
        double2 v = make_double2(0.0, 0.0);
        if (states[n] & FLAG_SAMPLENESS) {
            uint32_t l = node_to_leaf[n];
            v = make_double2(elen[l], slen[l]);
            if (!isfinite(v.x) || !isfinite(v.y)) *nonfinite = 1;
        }
        for (int k = 0; k < PK; ++k) psum[(size_t)k * nn + n] = v;
        return;
    }
    psum[n] = make_double2(0.0, 0.0);
    for (int k = 1; k < PK; ++k) {
        const double2 *row = psum + (size_t)(k - 1) * nn + c0;
        double e = 0.0, s = 0.0;
        for (uint32_t c = 0; c < 8; ++c) {
            double2 v = row[c];
            e += v.x;
            s += v.y;
        }
        psum[(size_t)k * nn + n] = make_double2(e, s);
    }
}

// intersectAABBWithSphere as the tree build evaluates it (aabb_sphere), with
// the per-axis branches turned into selects: an axis where the centre lies
// within the box adds an exact +0, so the sum is bit-identical.
__device__ __forceinline__ bool sphere_meets_box(const D3 &mn, const D3 &mx, const D3 &c, double r) {
    const double tx = c.x < mn.x ? dsub(c.x, mn.x) : (c.x > mx.x ? dsub(c.x, mx.x) : 0.0);
    const double ty = c.y < mn.y ? dsub(c.y, mn.y) : (c.y > mx.y ? dsub(c.y, mx.y) : 0.0);
    const double tz = c.z < mn.z ? dsub(c.z, mn.z) : (c.z > mx.z ? dsub(c.z, mx.z) : 0.0);
    const double d2 = dadd(dadd(dmul(tx, tx), dmul(ty, ty)), dmul(tz, tz));
    return d2 <= dmul(r, r);
}

// Box entirely inside the sphere, with a strict relative margin so that every
// leaf below certainly passes the closed sphere/box test.
__device__ inline bool box_inside_sphere(const D3 &mn, double sz, const D3 &c, double r) {
    double dx = fmax(fabs(c.x - mn.x), fabs(mn.x + sz - c.x));
    double dy = fmax(fabs(c.y - mn.y), fabs(mn.y + sz - c.y));
    double dz = fmax(fabs(c.z - mn.z), fabs(mn.z + sz - c.z));
    return dx * dx + dy * dy + dz * dz <= r * r * (1.0 - 1e-9);
}

// Children block b (nodes 1 + 8b .. 8 + 8b): the parent's corner on the
// lattice of 2^24 cells along the root's edge, and the children's depth.  Any
// corner down to depth 24 is a whole number below 2^24 there, exact in FP32.
constexpr uint32_t LATTICE_DEPTH = 24;

__global__ void k_block_corners(uint32_t nb, const uint32_t *parents, const uint8_t *depth, float4 *out) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const uint32_t first = 1 + 8 * b, d = depth[first];
    uint32_t x = 0, y = 0, z = 0, node = parents[first];
    for (uint32_t k = d - 1; k > 0; --k) {   // the node at depth k is child (node - 1) & 7 of its parent
        const uint32_t c = (node - 1) & 7u;
        if (k <= LATTICE_DEPTH) {
            const uint32_t step = LATTICE_DEPTH - k;
            x |= (c & 1u) << step;
            y |= ((c >> 1) & 1u) << step;
            z |= ((c >> 2) & 1u) << step;
        }
        node = parents[node];
    }
    out[b] = make_float4((float)x, (float)y, (float)z, __uint_as_float(d));
}

// Sort keys of the children blocks: the depth of the block's nodes.
__global__ void k_block_depth_keys(uint32_t nb, const uint8_t *depth, uint32_t *keys, uint32_t *vals) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    keys[b] = depth[1 + 8 * b];
    vals[b] = b;
}

// Blocks of `list` that hold a leaf whose sel[leaf] == value, and how many such leaves there are.
__global__ void k_blocks_with(uint32_t nb, const uint32_t *list, const uint2 *rec, const uint8_t *sel, uint8_t value,
                              uint8_t *flag, uint32_t *leaves) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t count = 0;
    if (i < nb) {
        const uint2 *r = rec + 1 + 8 * list[i] + REC_OFFSET;
        for (int c = 0; c < 8; ++c)
            if (r[c].x == INVALID && sel[r[c].y & REC_NOLEAF] == value) ++count;
        flag[i] = count ? 1 : 0;
    }
    for (int o = 16; o; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
    if ((threadIdx.x & 31) == 0 && count) atomicAdd(leaves, count);
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// What the prior queries read of the tree and the field.
struct PriorIn {
    uint32_t nn;
    const uint32_t *parents;
    const D3 *nmin;             // FP64 corners, for the tests that need them
    const uint2 *rec;
    const float4 *blocks;
    const double2 *psum;
    const int *nonfinite;       // != 0: a leaf's cone length is infinite or NaN
    double root_size, rel_radius;
    double corner_error;        // bound of an FP64 corner's or centre's distance from its lattice point
    bool deep;                  // deeper than the lattice: corners from nmin
    bool whole_radius;          // eight radii are a whole number, small enough for exact FP32 squares
};

// A step pops four blocks and pushes at most 32.  What one step pushed lies below
// only what came of its own blocks, at least a level deeper, so the steps with
// blocks left are at most one a depth; each but the last has lost four of its 32
// to the step right after it.
constexpr int PP_STACK = 28 * MAX_TREE_DEPTH + 32;
constexpr int PP_LEAVES = 64;   // blocks whose leaves wait; worked off when fewer than 32 are free
constexpr int PP_TIES = 96;     // leaves that touch a sphere; worked off when fewer than 64 are free
constexpr int PP_WARPS = 4;

// Occupancy::computePriors (Occupancy.cpp:530-568) with a
// SphereNodeStatesChecker (SphereNodeStatesChecker.cpp:28-36).  The set of
// leaves a query sums is the reference's: SAMPLENESS-flagged leaves at most
// three levels below the query leaf whose box meets the sphere; subtrees
// wholly inside the sphere are added from psum, whose row 0 is a flagged
// leaf's own (emptiness, sampleness) cone-length pair and zero elsewhere.
//
// One warp answers the queries of the up to eight leaves of a children block
// together: they have one size, their centres are one leaf size apart, and
// their radius is 25 of it, so their spheres take in nearly the same nodes.
// Two kinds of steps take four children blocks each, one node a lane, so the
// records, corners and cone lengths of a block arrive in whole lines:
//  * inner nodes are decided for the eight spheres at once: inside all (a row
//    of psum is added), outside all, or their children block is next -- its
//    inner nodes on the stack, its leaves on a second list;
//  * leaves are tested against each of the eight spheres.  Their centres are a
//    2 x 2 x 2 lattice, so the squared distances are sums of two terms per
//    axis, and every lane keeps the eight sums of the leaves it met; they are
//    added across the warp once, at the end.
//
// Lengths are in eighths of the query leaf's size, in the frame of the
// block's centre: every corner is a whole number, and the FP32 distances are
// exact wherever they decide anything.  A distance within `tol` of the radius
// (in practice a box that touches a sphere) is decided by the FP64 boxes, as
// the reference does.
//
// Measured, all queries of the field: 493 -> 164 ms at 16M held-out samples
// (7.6M leaves), 62 -> 28.6 ms at 300k, 34 -> 13.4 ms at 4M CSG samples, 1.5 ->
// 0.5 ms at 4k sphere samples.  A query per lane read eight records and eight
// psum rows of its own per expansion, 128 + 256 cache lines a warp's step, and
// the L1 passed 0.7 child tests a clock and SM; here the lines are shared and a
// test costs 12 of a lane's instructions.  What bounds it is latency at four
// warps a scheduler (128 registers, 32 of them the sums): two leaves a lane at a
// time are 8 % faster than one, three warps 23 % slower, five spill.  The eight
// spheres together open the blocks that any of them needs: 1.6 times the nodes
// are classified for each (23.5k against 14.4k a leaf at 16M held-out samples).
//
// BOUNDS (the pruned field's sign certificates): a node that straddles a
// query's sphere at depth >= the query leaf's depth - coarse_up is not
// descended; its whole subtree row is added to an undecided pair (eU, sU)
// instead, so the query ends early with eL <= E <= eL + eU and
// sL <= S <= sL + sU for the exact sums E, S, and writes
// bounds[leaf] = (eL / (eL + sL + sU), (eL + eU) / (eL + eU + sL)) around the
// prior E / (E + S).
struct Packet {   // the block of queries a warp works on
    float scale, cx, cy, cz;   // lattice cells -> eighths of the query leaf's size, packet frame
    double size;
    float ea;                  // bound of a corner's distance from its lattice point
    uint32_t q0, max_depth;
    // the box of the queries' centres: middle and half extent, 4 where both
    // halves of an axis hold one, 0 at +-4 where one does
    float mid[3], ext[3];
};

struct Box {
    float x, y, z, h;   // centre, half edge length
    float e;            // bound of a corner's error
};

// A node's box from its block's corner and its size.
__device__ __forceinline__ Box box_of(const PriorIn &in, const Packet &P, uint32_t node, float lx, float ly, float lz,
                                      float sz, float bx, float by, float bz) {
    Box b;
    b.h = 0.5f * sz;
    b.e = P.ea;
    if (!in.deep) {
        b.x = fmaf(bx, sz, lx) + b.h;
        b.y = fmaf(by, sz, ly) + b.h;
        b.z = fmaf(bz, sz, lz) + b.h;
    } else {
        const D3 m = in.nmin[node], o = in.nmin[in.parents[P.q0]];
        const double k = 8.0 / P.size;
        b.x = (float)(((m.x - o.x) - P.size) * k) + b.h;
        b.y = (float)(((m.y - o.y) - P.size) * k) + b.h;
        b.z = (float)(((m.z - o.z) - P.size) * k) + b.h;
        b.e += 4e-7f * (fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fabsf(b.z)) + sz);
    }
    return b;
}

// Bound of the FP32 error of a squared distance near the radius.
__device__ __forceinline__ float distance_error(float e, float ru) {
    return e > 0.01f * ru ? INFINITY : 4.0f * ru * e + 4e-7f * ru * ru;
}

// Four times the squared distances of the box from the eight centres (at +-4
// on each axis), less r4 = 4 r^2.  t + |t| = 2 max(t, 0) keeps the work on the
// FMA pipe; the minimum would go to the ALU, which has half its rate.
__device__ __forceinline__ void near_distances(const Box &b, float r4, float *s) {
    auto sq = [&](float c, float less) {
        const float t = fabsf(c) - b.h, u = t + fabsf(t);
        return fmaf(u, u, less);
    };
    const float X0 = sq(b.x + 4.0f, 0.0f), X1 = sq(b.x - 4.0f, 0.0f), Y0 = sq(b.y + 4.0f, -r4),
                Y1 = sq(b.y - 4.0f, -r4), Z0 = sq(b.z + 4.0f, 0.0f), Z1 = sq(b.z - 4.0f, 0.0f);
    const float xy[4] = {X0 + Y0, X1 + Y0, X0 + Y1, X1 + Y1};
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = xy[q & 3] + ((q & 4) ? Z1 : Z0);
}

// The same of the box's far corner.
__device__ __forceinline__ void far_distances(const Box &b, float r4, float *s) {
    auto sq = [&](float c, float less) {
        const float t = 2.0f * (fabsf(c) + b.h);
        return fmaf(t, t, less);
    };
    const float X0 = sq(b.x + 4.0f, 0.0f), X1 = sq(b.x - 4.0f, 0.0f), Y0 = sq(b.y + 4.0f, -r4),
                Y1 = sq(b.y - 4.0f, -r4), Z0 = sq(b.z + 4.0f, 0.0f), Z1 = sq(b.z - 4.0f, 0.0f);
    const float xy[4] = {X0 + Y0, X1 + Y0, X0 + Y1, X1 + Y1};
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = xy[q & 3] + ((q & 4) ? Z1 : Z0);
}

// e += v.x / 128, s += v.y / 128 where d < 0, without a predicate: a predicated
// FP64 addition becomes four selects on the half-rate ALU before it (58 of a
// step's 137 instructions).  sat(-d BIG) is 1.0f or 0.0f, and the bits of
// 1.0f over a zero word are the double 2^-7: an exact product and one rounding.
// The values must be finite.
__device__ __forceinline__ void add_where_negative(float d, const double2 &v, double &e, double &s) {
    const double w = __hiloint2double(__float_as_int(__saturatef(d * -1e30f)), 0);
    e = fma(v.x, w, e);
    s = fma(v.y, w, s);
}
constexpr double PP_UNIT = 128.0;

// The reference's decision of query q of the packet about a node whose FP32
// distance leaves it open: its box and every box above it meet the sphere (1),
// and the box is inside (2).  A box that touches the sphere can pass while the
// box around it, whose far corner is rounded differently, does not; so the
// boxes above are tested too, up to the first that clearly meets.
__device__ __noinline__ int exact_place(const PriorIn *in_p, const Packet *P, uint32_t q, uint32_t node) {
    const PriorIn &in = *in_p;
    const float ru = 8.0f * (float)in.rel_radius;
    const D3 qm = in.nmin[P->q0 + q];
    const double hs = dmul(0.5, P->size), radius = dmul(P->size, in.rel_radius);
    const D3 c{dadd(qm.x, hs), dadd(qm.y, hs), dadd(qm.z, hs)};
    uint32_t n = node;
    bool inside = false;
    while (true) {
        const float4 B = n ? in.blocks[(n - 1) >> 3] : make_float4(0.f, 0.f, 0.f, 0.f);
        const uint32_t d = n ? __float_as_uint(B.w) : 0;
        const D3 mn = in.nmin[n];
        const double sz = ldexp(in.root_size, -(int)d);
        if (!sphere_meets_box(mn, D3{dadd(mn.x, sz), dadd(mn.y, sz), dadd(mn.z, sz)}, c, radius)) return 0;
        if (n == node) inside = box_inside_sphere(mn, sz, c, radius);
        if (d == 0) break;
        n = in.parents[n];
        if (in.deep) continue;
        // the parent's box: corner B, twice the edge length
        const float h = __uint_as_float((127u + P->max_depth - d) << 23);
        const float x = fabsf(fmaf(B.x, P->scale, P->cx) + h + ((q & 1u) ? -4.0f : 4.0f)) - h;
        const float y = fabsf(fmaf(B.y, P->scale, P->cy) + h + ((q & 2u) ? -4.0f : 4.0f)) - h;
        const float z = fabsf(fmaf(B.z, P->scale, P->cz) + h + ((q & 4u) ? -4.0f : 4.0f)) - h;
        const float X = fmaxf(x, 0.0f), Y = fmaxf(y, 0.0f), Z = fmaxf(z, 0.0f);
        if (X * X + Y * Y + Z * Z - ru * ru < -distance_error(P->ea, ru)) break;
    }
    return inside ? 2 : 1;
}

struct PriorWarp {
    Packet packet;
    float4 leaf_box[PP_LEAVES];     // a waiting block's corner (packet frame) and its nodes' size
    uint32_t leaf_block[PP_LEAVES];
    uint32_t tie_node[PP_TIES];     // a leaf, and the queries whose sphere it touches
    uint8_t tie_mask[PP_TIES];
    uint32_t stack[PP_STACK];
};

template <bool BOUNDS>
__global__ void __launch_bounds__(32 * PP_WARPS, BOUNDS ? 3 : TSR_PRIOR_BLOCKS)
    k_priors(uint32_t nblocks, const uint32_t *list, const __grid_constant__ PriorIn in, const uint8_t *sel,
             uint8_t value, double *prior, double2 *bounds, uint32_t coarse_up, unsigned long long *next_block,
             unsigned long long *visits, int *err) {
    const unsigned FULL = 0xffffffffu;
    __shared__ PriorWarp shared[PP_WARPS];
    PriorWarp &w = shared[threadIdx.x >> 5];
    const Packet &P = w.packet;
    const unsigned lane = threadIdx.x & 31, below = (1u << lane) - 1u, ci = lane & 7u;
    const int quarter = (int)(lane >> 3);
    const float bx = (float)(ci & 1u), by = (float)((ci >> 1) & 1u), bz = (float)(ci >> 2);
    const float ru = 8.0f * (float)in.rel_radius, r2 = ru * ru, r4 = 4.0f * r2;
    const bool finite = *in.nonfinite == 0;
    unsigned long long nvis = 0;
    while (true) {
        unsigned long long bi = 0;
        if (lane == 0) bi = atomicAdd(next_block, 1ull);
        bi = __shfl_sync(FULL, bi, 0);
        if (bi >= nblocks) break;
        const uint32_t qb = list[bi];
        const uint2 qrec = __ldg(&in.rec[1 + 8 * qb + ci + REC_OFFSET]);
        const uint32_t qleaf = qrec.y & REC_NOLEAF;
        const bool wanted = qrec.x == INVALID && (!sel || sel[qleaf] == value);
        const unsigned mask = __ballot_sync(FULL, wanted) & 0xFFu;
        if (!mask) continue;
        const float4 Q = __ldg(&in.blocks[qb]);
        const uint32_t pd = __float_as_uint(Q.w);
        const uint2 root = __ldg(&in.rec[REC_OFFSET]);
        int sp = 0, waiting = 0, ties = 0;
        if (lane == 0) {
            Packet k;
            k.q0 = 1 + 8 * qb;
            k.max_depth = pd + MAX_DEPTH_DIFFERENCE;
            k.size = ldexp(in.root_size, -(int)pd);
            k.scale = ldexpf(1.0f, (int)k.max_depth - (int)LATTICE_DEPTH);
            const float half = ldexpf(1.0f, (int)LATTICE_DEPTH - (int)pd);
            k.cx = -(Q.x + half) * k.scale;
            k.cy = -(Q.y + half) * k.scale;
            k.cz = -(Q.z + half) * k.scale;
            k.ea = (float)(in.corner_error / k.size) * 8.0f;
            const unsigned low[3] = {mask & 0x55u, mask & 0x33u, mask & 0x0Fu},
                           high[3] = {mask & 0xAAu, mask & 0xCCu, mask & 0xF0u};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                k.ext[a] = low[a] && high[a] ? 4.0f : 0.0f;
                k.mid[a] = low[a] && high[a] ? 0.0f : (high[a] ? 4.0f : -4.0f);
            }
            w.packet = k;
            w.stack[0] = w.leaf_block[0] = 0;
            w.leaf_box[0] = make_float4(k.cx, k.cy, k.cz, __uint_as_float((126u + k.max_depth) << 23));
        }
        if (root.y & REC_FLAG) {   // the root's children (the root itself holds every centre)
            if (root.y & REC_HAS_INNER) sp = 1;
            if (root.y & REC_HAS_LEAVES) waiting = 1;
        }
        double aE[8], aS[8], uE[BOUNDS ? 8 : 1], uS[BOUNDS ? 8 : 1], allE = 0.0, allS = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) aE[q] = aS[q] = 0.0;
        if (BOUNDS) {
#pragma unroll
            for (int q = 0; q < 8; ++q) uE[q] = uS[q] = 0.0;
        }
        uint32_t opened = sp | waiting;   // children blocks
        __syncwarp();
        // whole-numbered distances: undecided only when zero
        const bool whole = in.whole_radius && !in.deep && 4.0f * ru * P.ea < 0.125f;
        while (sp > 0 || waiting > 0 || ties > 0) {
            if (ties > PP_TIES - 64 || (sp == 0 && waiting == 0)) {
                // ---- leaves that touch a sphere: a lane each
                for (int j = lane; j < ties; j += 32) {
                    const uint32_t node = w.tie_node[j];
                    unsigned met = 0;
                    for (unsigned rest = w.tie_mask[j]; rest; rest &= rest - 1) {
                        const uint32_t q = __ffs(rest) - 1;
                        if (exact_place(&in, &P, q, node)) met |= 1u << q;
                    }
                    const double2 v = __ldg(&in.psum[node]);
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if ((met >> q) & 1u) {
                            aE[q] += v.x / PP_UNIT;
                            aS[q] += v.y / PP_UNIT;
                        }
                }
                ties = 0;
                __syncwarp();
                continue;
            }
            if (waiting > PP_LEAVES - 32 || sp == 0) {
                // ---- the leaves of the waiting blocks, two a lane at a time
                do {
                    uint32_t node[2];
                    float4 B[2];
                    double2 v[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int left = waiting - 4 * k;
                        const bool valid = quarter < left;
                        const int at = valid ? left - 1 - quarter : 0;
                        node[k] = 1 + 8 * w.leaf_block[at] + ci;
                        B[k] = w.leaf_box[at];
                        v[k] = make_double2(0.0, 0.0);
                        if (valid) v[k] = __ldg(&in.psum[node[k]]);
                    }
                    float s[2][8], e[2];
                    bool unsure[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const Box box = box_of(in, P, node[k], B[k].x, B[k].y, B[k].z, B[k].w, bx, by, bz);
                        e[k] = box.e;
                        near_distances(box, r4, s[k]);
                        if (whole) {
                            float product = s[k][0];
#pragma unroll
                            for (int q = 1; q < 8; ++q) product *= s[k][q];
                            unsure[k] = !(fabsf(product) > 0.0f);
                        } else {
                            float least = fabsf(s[k][0]);
#pragma unroll
                            for (int q = 1; q < 8; ++q) least = fminf(least, fabsf(s[k][q]));
                            unsure[k] = !(least > 4.0f * distance_error(box.e, ru));
                        }
                        unsure[k] = unsure[k] && (v[k].x != 0.0 || v[k].y != 0.0);
                    }
                    if (__any_sync(FULL, unsure[0] || unsure[1])) {
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const unsigned um = __ballot_sync(FULL, unsure[k]);
                            if (unsure[k]) {   // decided later, not met here
                                const float tol = 4.0f * distance_error(e[k], ru);
                                unsigned ask = 0;
#pragma unroll
                                for (int q = 0; q < 8; ++q)
                                    if (!(fabsf(s[k][q]) > tol)) {
                                        ask |= 1u << q;
                                        s[k][q] = 1.0f;
                                    }
                                const int j = ties + __popc(um & below);
                                w.tie_node[j] = node[k];
                                w.tie_mask[j] = (uint8_t)(ask & mask);
                            }
                            ties += __popc(um);
                        }
                    }
                    if (finite) {
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            add_where_negative(s[0][q], v[0], aE[q], aS[q]);
                            add_where_negative(s[1][q], v[1], aE[q], aS[q]);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 2; ++k)
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                if (s[k][q] < 0.0f) {
                                    aE[q] += v[k].x / PP_UNIT;
                                    aS[q] += v[k].y / PP_UNIT;
                                }
                    }
                    waiting -= 8;
                } while ((waiting >= 8 || (waiting > 0 && sp == 0)) && ties <= PP_TIES - 64);
                if (waiting < 0) waiting = 0;
                __syncwarp();
                continue;
            }
            // ---- the inner nodes of the blocks on top of the stack
            const int take = sp < 4 ? sp : 4;
            const bool valid = quarter < take;
            const uint32_t b = w.stack[sp - 1 - (valid ? quarter : 0)], node = 1 + 8 * b + ci;
            sp -= take;
            const uint2 r = __ldg(&in.rec[node + REC_OFFSET]);
            const float4 B = __ldg(&in.blocks[b]);
            bool next = false;
            float4 corner = make_float4(0.f, 0.f, 0.f, 0.f);
            if (valid && r.x != INVALID && (r.y & REC_FLAG)) {
                const uint32_t d = __float_as_uint(B.w), k = P.max_depth - d;
                const Box box = box_of(in, P, node, fmaf(B.x, P.scale, P.cx), fmaf(B.y, P.scale, P.cy),
                                       fmaf(B.z, P.scale, P.cz), __uint_as_float((127u + k) << 23), bx, by, bz);
                const float m = box.h + box.e;
                const float dx = fabsf(box.x - P.mid[0]), dy = fabsf(box.y - P.mid[1]), dz = fabsf(box.z - P.mid[2]);
                const float mx = P.ext[0] + m, my = P.ext[1] + m, mz = P.ext[2] + m;
                const float fx = dx + mx, fy = dy + my, fz = dz + mz;
                const float nx = fmaxf(dx - mx, 0.0f), ny = fmaxf(dy - my, 0.0f), nz = fmaxf(dz - mz, 0.0f);
                const bool apart = nx * nx + ny * ny + nz * nz > r2 * (1.0f + 1e-6f);
                const bool inside = fx * fx + fy * fy + fz * fz < r2 * (1.0f - 2e-6f);
                if (inside && k < (uint32_t)PK) {
                    const double2 row = in.psum[(size_t)k * in.nn + node];
                    allE += row.x;
                    allS += row.y;
                } else if (!apart) {
                    if (BOUNDS && d >= (pd > coarse_up + 1 ? pd - coarse_up : 1)) {   // k <= 3 + coarse_up < PK there
                        const double2 row = in.psum[(size_t)k * in.nn + node];
                        const float tol = 4.0f * distance_error(box.e, ru);
                        float s[8], f[8];
                        near_distances(box, r4, s);
                        far_distances(box, r4, f);
                        unsigned ask = 0, met = 0, in_it = 0;
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            if (!(fabsf(s[q]) > tol) || !(fabsf(f[q]) > tol)) ask |= 1u << q;
                            if (s[q] < 0.0f) met |= 1u << q;
                            if (f[q] < 0.0f) in_it |= 1u << q;
                        }
                        for (unsigned rest = ask & mask; rest; rest &= rest - 1) {
                            const uint32_t q = __ffs(rest) - 1;
                            const int place = exact_place(&in, &P, q, node);
                            met = (met & ~(1u << q)) | (place > 0 ? 1u << q : 0u);
                            in_it = (in_it & ~(1u << q)) | (place > 1 ? 1u << q : 0u);
                        }
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            if (!((met >> q) & 1u)) continue;
                            if ((in_it >> q) & 1u) {
                                aE[q] += row.x / PP_UNIT;
                                aS[q] += row.y / PP_UNIT;
                            } else {
                                uE[q] += row.x;
                                uS[q] += row.y;
                            }
                        }
                    } else {
                        next = d < P.max_depth;
                        corner = make_float4(box.x - box.h, box.y - box.h, box.z - box.h, box.h);
                    }
                }
            }
            const uint32_t block = (r.x - 1) >> 3;
            const bool push = next && (r.y & REC_HAS_INNER), wait = next && (r.y & REC_HAS_LEAVES);
            const unsigned pm = __ballot_sync(FULL, push), wm = __ballot_sync(FULL, wait);
            if (sp + __popc(pm) > PP_STACK) {
                if (lane == 0) atomicExch(err, 2);   // deeper than any tree
            } else {
                if (push) w.stack[sp + __popc(pm & below)] = block;
                sp += __popc(pm);
            }
            if (wait) {
                const int j = waiting + __popc(wm & below);
                w.leaf_block[j] = block;
                w.leaf_box[j] = corner;
            }
            waiting += __popc(wm);
            opened += __popc(pm | wm);
            __syncwarp();
        }
        nvis += 8ull * opened * __popc(mask);   // every node of an opened block, for each of the queries
        allE = warp_sum(allE);
        allS = warp_sum(allS);
        double E = 0.0, S = 0.0, UE = 0.0, US = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double te = warp_sum(aE[q]), ts = warp_sum(aS[q]);
            double ue = 0.0, us = 0.0;
            if (BOUNDS) {
                ue = warp_sum(uE[q]);
                us = warp_sum(uS[q]);
            }
            if ((int)lane == q) {
                E = PP_UNIT * te + allE;
                S = PP_UNIT * ts + allS;
                UE = ue;
                US = us;
            }
        }
        if (lane < 8 && wanted) {
            if (BOUNDS)
                bounds[qleaf] = make_double2(E / (E + S + US), (E + UE) / (E + UE + S));
            else
                prior[qleaf] = E / (E + S);
        }
        __syncwarp();   // the packet is done with
    }
    if (lane == 0 && nvis) atomicAdd(visits, nvis);
}

// A tree that is one leaf, the root: its own lengths decide.
__global__ void k_prior_root(const double2 *psum, double *prior, double2 *bounds) {
    const double p = psum->x / (psum->x + psum->y);
    if (bounds) bounds[0] = make_double2(p, p);
    else prior[0] = p;
}

// Occupancy::getOccupancy (Occupancy.cpp:570-587), FP64.  In a pruned field
// (pred != null) a reliable leaf whose prior was not queried (need == 0)
// gets its sign from E == 0 / S == 0 or from the pruner, and the value
// 0.5 (S - E) / coneCount for a positive sign (the value at prior 1/2), so
// only leaves away from a predicted sign change carry an approximate value.
__global__ void k_finalize(uint32_t nl, const double *esum, const double *ssum, const double *elen,
                           const double *slen, const double *prior, double cone_count, double threshold,
                           const uint8_t *pred, const uint8_t *need, double *o_esum, double *o_ssum,
                           double *o_elen, double *o_slen, double *occ) {
    uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    double e = esum[l], s = ssum[l];
    o_esum[l] = e;
    o_ssum[l] = s;
    o_elen[l] = elen[l];
    o_slen[l] = slen[l];
    double v;
    if ((e + s) < threshold) {
        v = -EPS;
    } else if (pred && !need[l]) {
        const bool pos = (e == 0.0) ? true : (s == 0.0) ? false : (pred[l] & PRED_POS) != 0;
        const double approx = 0.5 * (s - e) / cone_count;
        if (pos && (pred[l] & PRED_HIGH))
            v = approx > 2.0 * EPS ? approx : 2.0 * EPS;   // above EPSILON, like the exact value
        else if (pos && (pred[l] & PRED_LOW))
            v = EPS;                                       // at most EPSILON, like the exact value
        else
            v = (pos && approx > 0.0) ? approx : (pos ? EPS : -EPS);
    } else {
        double pr = prior[l];
        double pe = pr * (e / cone_count);
        double ps = (1.0 - pr) * (s / cone_count);
        v = (pe >= ps) ? -EPS : ps - pe;
    }
    occ[l] = v;
}

struct Timer {
    cudaEvent_t a{}, b{};
    cudaStream_t st;
    explicit Timer(cudaStream_t s) : st(s) {
        TSR_CUDA(cudaEventCreate(&a));
        TSR_CUDA(cudaEventCreate(&b));
        TSR_CUDA(cudaEventRecord(a, st));
    }
    float lap() {
        TSR_CUDA(cudaEventRecord(b, st));
        TSR_CUDA(cudaEventSynchronize(b));
        float ms = 0;
        TSR_CUDA(cudaEventElapsedTime(&ms, a, b));
        std::swap(a, b);
        return ms;
    }
    ~Timer() { cudaEventDestroy(a); cudaEventDestroy(b); }
};

// The children blocks in order of depth, coarsest first, tree order within a
// depth (a stable radix sort of 6-bit keys).  A coarse leaf's sphere is wide
// and its query long; taking those first keeps the warps from ending on a
// tail of long queries.
static_assert(MAX_TREE_DEPTH < 64, "depth keys are 6 bits");
DBuf<uint32_t> depth_ordered_blocks(uint32_t nb, const uint8_t *depth, cudaStream_t st) {
    DBuf<uint32_t> out(nb, st);
    if (nb == 0) return out;
    DBuf<uint32_t> k1(nb, st), k2(nb, st), v1(nb, st);
    k_block_depth_keys<<<grid_for(nb, BLK), BLK, 0, st>>>(nb, depth, k1.p, v1.p); ::tsr::note_launch();
    size_t tmp = 0;
    TSR_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, k1.p, k2.p, v1.p, out.p, (int)nb, 0, 6, st));
    DBuf<uint8_t> tb(tmp, st);
    TSR_CUDA(cub::DeviceRadixSort::SortPairs(tb.p, tmp, k1.p, k2.p, v1.p, out.p, (int)nb, 0, 6, st));
    return out;
}

}  // namespace

// The field of all links (update == false), or an update of an existing
// field by the links of `chosen` samples (device indices, tree order) added
// (sign +1) or removed (sign -1): Occupancy::update (Occupancy.h:222-227)
// after onSamplesChanged (Occupancy.cpp:129-136) -- both cone passes over the
// chosen links into the field's sums, node flags set only when adding, then
// the priors and the occupancy of every leaf again.
void compute_occupancy(const tsr_tree &t, const tsr_cameras_view &cv, const tsr_params &p, int mode,
                       tsr_occupancy &o, const tsr_pruner *pruner, const uint32_t *chosen, uint32_t nchosen,
                       double sign, bool update) {
    (void)mode;
    cudaStream_t st = o.stream;
    const uint32_t nl = t.n_leaves, nn = t.n_nodes;
    o.n_leaves = nl;
    o.n_nodes = nn;
    o.confidence_threshold = p.confidence_threshold;
    const uint64_t nlinks = update ? (uint64_t)nchosen * t.k : (uint64_t)t.n_samples * t.k;
    // working set: per link the set-up record, keys and order; per node the
    // traversal records, states and the prior table; per leaf the sums
    reserve_pool((size_t)nlinks * 160 + (size_t)nn * 200 + (size_t)nl * 120 + (64u << 20), o.stream);
    Timer timer(st);
    DBuf<D3> cams(cv.count, st);
    if (cv.count) TSR_CUDA(cudaMemcpyAsync(cams.p, cv.positions, (size_t)cv.count * 24, cudaMemcpyHostToDevice, st));
    DBuf<double> acc;   // esum, ssum, elen, slen of a new field
    double *esum, *ssum, *elen, *slen;
    DBuf<uint32_t> link_list;
    if (update) {
        esum = o.e_sum.p; ssum = o.s_sum.p; elen = o.e_len.p; slen = o.s_len.p;
        link_list.alloc(nlinks, st);
        k_sample_links<<<grid_for(nlinks, BLK), BLK, 0, st>>>(nchosen, chosen, t.k, link_list.p); ::tsr::note_launch();
    } else {
        acc.alloc(4ull * nl, st);
        acc.zero();
        esum = acc.p; ssum = acc.p + nl; elen = acc.p + 2ull * nl; slen = acc.p + 3ull * nl;
        o.states.alloc(nn, st);
        o.states.zero();
    }
    DBuf<double> cone_count(1, st);
    cone_count.zero();
    DBuf<unsigned long long> accepted(5, st);   // accepted E, S; visits E, S; prior visits
    accepted.zero();
    DBuf<int> err(2, st);   // error code, non-finite cone lengths
    err.zero();

    LinkIn in{t.pos.p, t.nrm.p, t.scale.p, t.conf.p, t.links.p, cams.p, t.k, cv.count,
              p.max_relative_sampling_distance, p.bandwidth_factor, p.relative_sample_cone_length, t.root_size};
    TreeIn tr{t.nmin.p};
    if (!update) o.links = nlinks;
    DBuf<unsigned long long> next_link(1, st);
    const uint32_t stack = cone_stack(t.max_depth), warp_bytes = (uint32_t)cone_warp_bytes(stack);
    const size_t cone_smem = (size_t)CX_WARPS * warp_bytes;
    unsigned x_grid = 0, prior_grid = 0, bounds_grid = 0;
    {
        int dev = 0, sms = 0, per_sm = 0;
        TSR_CUDA(cudaGetDevice(&dev));
        TSR_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        TSR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cones<EMPTINESS>, 32 * CX_WARPS, cone_smem));
        x_grid = (unsigned)(sms * (per_sm > 0 ? per_sm : 1));
        TSR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_priors<false>, 32 * PP_WARPS, 0));
        prior_grid = (unsigned)(sms * (per_sm > 0 ? per_sm : 1));
        TSR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_priors<true>, 32 * PP_WARPS, 0));
        bounds_grid = (unsigned)(sms * (per_sm > 0 ? per_sm : 1));
    }
    // links a warp takes at a time: so few that every warp gets some
    const uint32_t links_per_warp =
        (uint32_t)std::min<uint64_t>(CX_LINKS, std::max<uint64_t>(1, nlinks / ((uint64_t)x_grid * CX_WARPS * 2)));
    if (nl > REC_NOLEAF) fail(TSR_ERR_OVERFLOW_U32, "leaf count must stay below 2^31 - 1 for the traversal records");
    DBuf<uint2> recs((size_t)nn + 8, st);
    if (reinterpret_cast<uintptr_t>(recs.p) % 16) fail(TSR_ERR_CUDA, "traversal records are not 16-byte aligned");
    next_link.zero();
    k_pack_rec<<<grid_for(nn, BLK), BLK, 0, st>>>(nn, t.children.p, t.node_to_leaf.p, nullptr, recs.p); ::tsr::note_launch();
    DBuf<LinkRec> lrec((size_t)nlinks, st);
    if (nlinks) {
        k_link_setup<SAMPLENESS><<<grid_for(nlinks, 128), 128, 0, st>>>(nlinks, link_list.p, in, tr, recs.p, lrec.p,
                                                                        ssum, slen, cone_count.p, accepted.p + 1,
                                                                        sign);
        ::tsr::note_launch();
        k_cones<SAMPLENESS><<<x_grid, 32 * CX_WARPS, cone_smem, st>>>(
            nlinks, links_per_warp, stack, warp_bytes, lrec.p, tr, recs.p, (float)t.root_size, ssum, slen,
            accepted.p + 1, next_link.p, accepted.p + 3, err.p, sign);
        ::tsr::note_launch();
    }
    // flags mark leaves that received a kernel; removal leaves them set (Occupancy.cpp:232)
    if (sign > 0.0) {
        k_leaf_flags<<<grid_for(nl, BLK), BLK, 0, st>>>(nl, t.leaf_node.p, ssum, o.states.p, FLAG_SAMPLENESS);
        ::tsr::note_launch();
    }
    o.stage_ms[0] = timer.lap();
    // EMPTINESS links grouped by camera (stable, so sample order is kept
    // within a camera): a warp's cones then share their apex
    DBuf<uint32_t> order((size_t)nlinks, st);
    {
        DBuf<uint32_t> ckeys((size_t)nlinks, st), ckeys2((size_t)nlinks, st), vals((size_t)nlinks, st);
        if (nlinks) {
            k_link_cameras<<<grid_for(nlinks, BLK), BLK, 0, st>>>(nlinks, link_list.p, t.links.p, cv.count, ckeys.p,
                                                                  vals.p); ::tsr::note_launch();
        }
        int bits = 1;
        while ((1u << bits) <= cv.count) ++bits;
        size_t tmp = 0;
        if (nlinks) {
            TSR_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, ckeys.p, ckeys2.p, vals.p, order.p, (int)nlinks, 0,
                                                     bits, st));
            DBuf<uint8_t> tb(tmp, st);
            TSR_CUDA(cub::DeviceRadixSort::SortPairs(tb.p, tmp, ckeys.p, ckeys2.p, vals.p, order.p, (int)nlinks, 0,
                                                     bits, st));
        }
    }
    // forwardAnyChildStateFlag(0, SAMPLENESS) before the EMPTINESS pass (Occupancy.cpp:141-142)
    for (int d = (int)t.level_start.size() - 2; d >= 0; --d) {
        uint32_t lo = t.level_start[d], hi = t.level_start[d + 1];
        k_forward_flag<<<grid_for(hi - lo, BLK), BLK, 0, st>>>(lo, hi, t.level_order.p, t.children.p, o.states.p,
                                                              FLAG_SAMPLENESS); ::tsr::note_launch();
    }
    k_pack_rec<<<grid_for(nn, BLK), BLK, 0, st>>>(nn, t.children.p, t.node_to_leaf.p, o.states.p, recs.p);
    ::tsr::note_launch();
    o.stage_ms[1] = timer.lap();
    next_link.zero();
    if (nlinks) {
        k_link_setup<EMPTINESS><<<grid_for(nlinks, 128), 128, 0, st>>>(nlinks, order.p, in, tr, recs.p, lrec.p, esum,
                                                                       elen, cone_count.p, accepted.p, sign);
        ::tsr::note_launch();
        k_cones<EMPTINESS><<<x_grid, 32 * CX_WARPS, cone_smem, st>>>(
            nlinks, links_per_warp, stack, warp_bytes, lrec.p, tr, recs.p, (float)t.root_size, esum, elen, accepted.p,
            next_link.p, accepted.p + 2, err.p, sign);
        ::tsr::note_launch();
    }
    if (sign > 0.0) {
        k_leaf_flags<<<grid_for(nl, BLK), BLK, 0, st>>>(nl, t.leaf_node.p, esum, o.states.p, FLAG_EMPTINESS);
        ::tsr::note_launch();
    }
    o.stage_ms[2] = timer.lap();
    o.prior.alloc(nl, st);
    DBuf<uint8_t> need;   // pruned field: leaves whose prior is queried
    DBuf<uint8_t> pred_buf;
    if (pruner) pruner_predict(t, *pruner, esum, ssum, p.confidence_threshold, pred_buf, st);
    const uint8_t *pred = pred_buf.p;
    if (pred) {
        o.prior.fill_bytes(0xFF);   // NaN: no prior where the query was skipped
        need.alloc(nl, st);
        k_prior_needed<<<grid_for(nl, BLK), BLK, 0, st>>>(nl, pred, esum, ssum, p.confidence_threshold, need.p);
        ::tsr::note_launch();
    }
    DBuf<double2> psum((size_t)nn * PK, st);   // cumulative prior sums
    for (int d = (int)t.level_start.size() - 2; d >= 0; --d) {
        uint32_t lo = t.level_start[d], hi = t.level_start[d + 1];
        k_prior_sums<<<grid_for(hi - lo, BLK), BLK, 0, st>>>(lo, hi, nn, t.level_order.p, t.children.p,
                                                            t.node_to_leaf.p, o.states.p, elen, slen, psum.p,
                                                            err.p + 1); ::tsr::note_launch();
    }
    const uint32_t nb = (nn - 1) / 8;
    DBuf<float4> block_corners(nb, st);
    DBuf<uint32_t> block_order = depth_ordered_blocks(nb, t.depth.p, st);
    if (nb) {
        k_block_corners<<<grid_for(nb, BLK), BLK, 0, st>>>(nb, t.parents.p, t.depth.p, block_corners.p);
        ::tsr::note_launch();
    }
    PriorIn pin{nn, t.parents.p, t.nmin.p, recs.p, block_corners.p, psum.p, err.p + 1, t.root_size,
                p.relative_radius_for_priors, 0.0, t.max_depth >= LATTICE_DEPTH, false};
    {
        // a corner is a sum of at most MAX_TREE_DEPTH steps, a centre one more, each rounded to half an ulp
        double m = 0.0;
        for (int j = 0; j < 3; ++j) m = std::max(m, std::fabs(t.root_min[j]));
        pin.corner_error = 64.0 * 1.1102230246251565e-16 * (m + t.root_size);
        const double r = 8.0 * p.relative_radius_for_priors;
        pin.whole_radius = r == std::floor(r) && r <= 1024.0;
    }
    // the priors of all leaves (sel == null), or of those with sel[leaf] == value; returns their number
    auto query = [&](const uint8_t *sel, uint8_t value, double2 *bounds) -> uint32_t {
        DBuf<uint32_t> chosen;
        const uint32_t *list = block_order.p;
        uint32_t n = nb, leaves = nl;
        if (nb == 0) {   // the root is the only leaf
            if (sel && read_scalar(sel, st) != value) return 0;
            k_prior_root<<<1, 1, 0, st>>>(psum.p, o.prior.p, bounds); ::tsr::note_launch();
            return 1;
        }
        if (sel) {
            DBuf<uint8_t> flag(nb, st);
            DBuf<uint32_t> counts(2, st);   // blocks, leaves
            counts.zero();
            chosen.alloc(nb, st);
            k_blocks_with<<<grid_for(nb, BLK), BLK, 0, st>>>(nb, list, recs.p, sel, value, flag.p, counts.p + 1);
            ::tsr::note_launch();
            size_t tmp = 0;
            TSR_CUDA(cub::DeviceSelect::Flagged(nullptr, tmp, list, flag.p, chosen.p, counts.p, (int)nb, st));
            DBuf<uint8_t> tb(tmp, st);
            TSR_CUDA(cub::DeviceSelect::Flagged(tb.p, tmp, list, flag.p, chosen.p, counts.p, (int)nb, st));
            uint32_t h[2];
            TSR_CUDA(cudaMemcpyAsync(h, counts.p, 8, cudaMemcpyDeviceToHost, st));
            TSR_CUDA(cudaStreamSynchronize(st));
            n = h[0];
            leaves = h[1];
            list = chosen.p;
        }
        if (n == 0) return leaves;
        next_link.zero();
        if (bounds)
            k_priors<true><<<bounds_grid, 32 * PP_WARPS, 0, st>>>(n, list, pin, sel, value, nullptr, bounds,
                                                                  pruner->bound_levels, next_link.p, accepted.p + 4,
                                                                  err.p);
        else
            k_priors<false><<<prior_grid, 32 * PP_WARPS, 0, st>>>(n, list, pin, sel, value, o.prior.p, nullptr, 0,
                                                                  next_link.p, accepted.p + 4, err.p);
        ::tsr::note_launch();
        return leaves;
    };
    if (pred) {
        // skip candidates: certify their signs from bounds of their priors
        DBuf<unsigned long long> ncert(1, st);
        ncert.zero();
        DBuf<double2> bnd(nl, st);
        if (query(need.p, NEED_CERTIFY, bnd.p)) {
            k_certify<<<grid_for(nl, BLK), BLK, 0, st>>>(nl, esum, ssum, bnd.p, cone_count.p, pred_buf.p, need.p,
                                                        ncert.p); ::tsr::note_launch();
            o.certified = read_scalar(ncert.p, st);
        }
        // every leaf still needing its prior is queried
        o.pruned = nl - query(need.p, NEED_QUERY, nullptr);
    } else {
        query(nullptr, 0, nullptr);
    }
    o.stage_ms[3] = timer.lap();
    if (update) {
        o.cone_count += read_scalar(cone_count.p, st);
    } else {
        o.cone_count = read_scalar(cone_count.p, st);
        o.e_sum.alloc(nl, st); o.s_sum.alloc(nl, st); o.e_len.alloc(nl, st); o.s_len.alloc(nl, st);
        o.occ.alloc(nl, st);
    }
    k_finalize<<<grid_for(nl, BLK), BLK, 0, st>>>(nl, esum, ssum, elen, slen, o.prior.p, o.cone_count,
                                                 p.confidence_threshold, pred, need.p, o.e_sum.p, o.s_sum.p,
                                                 o.e_len.p, o.s_len.p, o.occ.p); ::tsr::note_launch();
    if (pred) {
        // Repair: a skipped positive leaf next to a negative one carries a
        // value the surface uses (the signs themselves are exact); query its
        // prior and recompute it, until no such leaf is left (one round
        // queries them all; the next finds none).
        DBuf<uint8_t> mark(nl, st);
        DBuf<uint32_t> nmark(1, st);
        for (int round = 0; round < 64; ++round) {
            mark.zero();
            nmark.zero();
            k_repair_mark<<<grid_for(nl, BLK), BLK, 0, st>>>(nl, t.nb_off.p, t.nbs.p, o.occ.p, need.p, pred, esum, ssum,
                                                            p.confidence_threshold, mark.p); ::tsr::note_launch();
            k_set_needed<<<grid_for(nl, BLK), BLK, 0, st>>>(nl, mark.p, need.p, nmark.p); ::tsr::note_launch();
            const uint32_t nf = read_scalar(nmark.p, st);
            if (nf == 0) break;
            query(mark.p, 1, nullptr);
            k_finalize<<<grid_for(nl, BLK), BLK, 0, st>>>(nl, esum, ssum, elen, slen, o.prior.p, o.cone_count,
                                                         p.confidence_threshold, pred, need.p, o.e_sum.p, o.s_sum.p,
                                                         o.e_len.p, o.s_len.p, o.occ.p); ::tsr::note_launch();
            o.pruned -= nf;
            o.repaired += nf;
        }
    }
    o.stage_ms[4] = timer.lap();
    unsigned long long a[5];
    TSR_CUDA(cudaMemcpyAsync(a, accepted.p, sizeof(a), cudaMemcpyDeviceToHost, st));
    int e = read_scalar(err.p, st);
    o.accepted[0] = a[0];
    o.accepted[1] = a[1];
    o.visits[0] = a[2];
    o.visits[1] = a[3];
    o.visits[2] = a[4];
    if (e) fail(TSR_ERR_DEVICE_ASSERT, "occupancy traversal exceeded its stack bound");
    TSR_CUDA(cudaGetLastError());
}

// The occupancy of every leaf from sums, cone lengths, priors and cone count
// already in the field's buffers (a field read from a file): the plain
// formula of k_finalize, sums copied onto themselves.
void finalize_field(tsr_occupancy &o, const tsr_params &p) {
    const uint32_t nl = o.n_leaves;
    o.occ.alloc(nl, o.stream);
    if (!nl) return;
    k_finalize<<<grid_for(nl, BLK), BLK, 0, o.stream>>>(nl, o.e_sum.p, o.s_sum.p, o.e_len.p, o.s_len.p, o.prior.p,
                                                       o.cone_count, p.confidence_threshold, nullptr, nullptr,
                                                       o.e_sum.p, o.s_sum.p, o.e_len.p, o.s_len.p, o.occ.p);
    ::tsr::note_launch();
    TSR_CUDA(cudaGetLastError());
}

}  // namespace tsr
