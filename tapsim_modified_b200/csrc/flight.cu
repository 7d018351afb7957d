// Ion flights: one warp per ion.  Restates Trajectory_3d (tapsim/
// trajectory_3d.cpp) in FP64: the embedded Cash-Karp Runge-Kutta step
// (o5_integrator, :583-676, tableau of Cash & Karp 1990), the
// error-restricted step control (errorRestricted_stepper, :358-425), the
// loop that ends when the ion leaves the mesh (integrate, :130-209) and the
// linear extrapolation to the top plane (extrapolate, :303-332).  The field
// at a point is the barycentric interpolation of the per-vertex field_o1 of
// the enclosing tetrahedron (Grid_3d::FastField::compute,
// grid_3d.cpp:1663-1721, with the weights of tetWeights,
// geometry_3d.cpp:916-980); the tetrahedron comes from a visibility walk
// (findTetrahedron, geometry_3d.cpp:988-1044) whose start face rotates
// instead of being drawn with rand().
#include "kernels.cuh"

namespace tgd {
namespace {

constexpr int kBlock = 128;

__constant__ int kFaceDev[4][3] = {{1, 3, 2}, {0, 2, 3}, {0, 3, 1}, {0, 1, 2}};

struct V3 {
    double x, y, z;
};
__device__ __forceinline__ V3 ld3(const float* p, int i) { return {p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }

__device__ __forceinline__ double orient(V3 a, V3 b, V3 c, V3 p) {
    const double ux = b.x - a.x, uy = b.y - a.y, uz = b.z - a.z;
    const double vx = c.x - a.x, vy = c.y - a.y, vz = c.z - a.z;
    const double wx = p.x - a.x, wy = p.y - a.y, wz = p.z - a.z;
    return ux * (vy * wz - vz * wy) - uy * (vx * wz - vz * wx) + uz * (vx * wy - vy * wx);
}

// Sign of orient(a,b,c,p), exact for the points snapped to the power-of-two
// grid the host Delaunay builder uses (|coordinate| <= 2^40 quanta): a double
// evaluation with a forward error bound, and an exact 128-bit integer
// evaluation when the bound does not certify the sign.  The walk thereby
// decides every face consistently (a point on a shared face, such as an ion
// starting at a mesh vertex, is never "beyond" it from both sides), which is
// what makes the visibility walk terminate, as the reference's exact
// Predicates::orient3d does (geometry_3d.cpp:1750-1768).
__device__ int orient_sign(V3 a, V3 b, V3 c, V3 p, double snap) {
    const double ux = b.x - a.x, uy = b.y - a.y, uz = b.z - a.z;
    const double vx = c.x - a.x, vy = c.y - a.y, vz = c.z - a.z;
    const double wx = p.x - a.x, wy = p.y - a.y, wz = p.z - a.z;
    const double m0 = vy * wz - vz * wy, m1 = vx * wz - vz * wx, m2 = vx * wy - vy * wx;
    const double det = ux * m0 - uy * m1 + uz * m2;
    const double perm = fabs(ux) * (fabs(vy * wz) + fabs(vz * wy)) + fabs(uy) * (fabs(vx * wz) + fabs(vz * wx)) +
                        fabs(uz) * (fabs(vx * wy) + fabs(vy * wx));
    const double bound = 16.0 * 1.1102230246251565e-16 * perm;
    if (det > bound) return 1;
    if (det < -bound) return -1;
    const double lim = 1.0995116277760000e12;  // 2^40
    const double px = p.x * snap, py = p.y * snap, pz = p.z * snap;
    if (fabs(px) > lim || fabs(py) > lim || fabs(pz) > lim) return det > 0.0 ? 1 : (det < 0.0 ? -1 : 0);
    const long long ax = __double2ll_rn(a.x * snap), ay = __double2ll_rn(a.y * snap), az = __double2ll_rn(a.z * snap);
    const long long Ux = __double2ll_rn(b.x * snap) - ax, Uy = __double2ll_rn(b.y * snap) - ay, Uz = __double2ll_rn(b.z * snap) - az;
    const long long Vx = __double2ll_rn(c.x * snap) - ax, Vy = __double2ll_rn(c.y * snap) - ay, Vz = __double2ll_rn(c.z * snap) - az;
    const long long Wx = __double2ll_rn(px) - ax, Wy = __double2ll_rn(py) - ay, Wz = __double2ll_rn(pz) - az;
    const __int128 M0 = (__int128)Vy * Wz - (__int128)Vz * Wy;
    const __int128 M1 = (__int128)Vx * Wz - (__int128)Vz * Wx;
    const __int128 M2 = (__int128)Vx * Wy - (__int128)Vy * Wx;
    const __int128 e = (__int128)Ux * M0 - (__int128)Uy * M1 + (__int128)Uz * M2;
    return e > 0 ? 1 : (e < 0 ? -1 : 0);
}

// Returns the tetrahedron holding p, -1 when p is outside the mesh, -2 when
// the walk exceeded `limit` steps.
__device__ int locate(const DevMesh& m, V3 p, int t, int limit, unsigned& rot) {
    if (t < 0) return -1;
    for (int step = 0; step < limit; step++) {
        const int* v = m.tet_v + 4 * t;
        int next = -1;
        bool moved = false;
        const unsigned r = rot++;
        for (int j = 0; j < 4; j++) {
            const int k = (int)((r + j) & 3);
            const V3 a = ld3(m.xyz, v[kFaceDev[k][0]]), b = ld3(m.xyz, v[kFaceDev[k][1]]), c = ld3(m.xyz, v[kFaceDev[k][2]]);
            if (orient_sign(a, b, c, p, m.snap) < 0) {
                next = m.tet_n[4 * t + k];
                moved = true;
                break;
            }
        }
        if (!moved) return t;
        if (next < 0) return -1;
        t = next;
    }
    return -2;
}

// Barycentric weights (tetWeights): |sub-volume| / |volume|, 1/4 each for a
// flat tetrahedron.
__device__ void weights(const DevMesh& m, int t, V3 p, double w[4]) {
    const int* v = m.tet_v + 4 * t;
    const V3 P[4] = {ld3(m.xyz, v[0]), ld3(m.xyz, v[1]), ld3(m.xyz, v[2]), ld3(m.xyz, v[3])};
    const double vol = fabs(orient(P[0], P[1], P[2], P[3]));
    if (vol == 0.0) {
        w[0] = w[1] = w[2] = w[3] = 0.25;
        return;
    }
    w[0] = fabs(orient(p, P[1], P[2], P[3])) / vol;
    w[1] = fabs(orient(P[0], p, P[2], P[3])) / vol;
    w[2] = fabs(orient(P[0], P[1], p, P[3])) / vol;
    w[3] = fabs(orient(P[0], P[1], P[2], p)) / vol;
}

// Vertex fields of one flight call: every node's field_o1 is computed once,
// in bulk, from the current potentials before the flights start, and the
// potentials are copied beside them (the flights read only these two
// snapshots, so a flight may overlap the next event's relaxation) (the
// FastField buffer of the reference, grid_3d.cpp:1672-1702, filled for all
// vertices at once instead of on first use).  Four lanes share a row; a
// singular node stores NaN in x, which the flight reports as S_SINGULAR when
// it interpolates from that vertex, as the on-demand computation would.
// With a cell list, only the listed cells are computed: the event loop lists
// the cells that are free or have a free neighbour, since the field of a
// Dirichlet cell among Dirichlet cells depends only on potentials and
// couplings that never change.
constexpr int kLanesPerRow = 4;
__global__ void k_vertex_fields(DevMesh m, const int32_t* __restrict__ cells, int count) {
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = gid / kLanesPerRow;
    const int lane = gid % kLanesPerRow;
    const bool live = t < (cells ? count : m.n);
    const int ii = live ? (cells ? cells[t] : t) : m.n - 1;
    const int i = ii;
    const bool hull = (m.flags[ii] & F_HULL) != 0;
    const double xi = m.xyz[3 * ii], yi = m.xyz[3 * ii + 1], zi = m.xyz[3 * ii + 2];
    const double pi = m.phi64[ii];
    double a00 = 0, a01 = 0, a02 = 0, a11 = 0, a12 = 0, a22 = 0, b0 = 0, b1 = 0, b2 = 0;
    const int q1 = hull ? 0 : m.row_ptr[ii + 1];
    for (int q = (hull ? 0 : m.row_ptr[ii]) + lane; q < q1; q += kLanesPerRow) {
        if (m.cnz[q] == 0) continue;
        const int j = m.col[q];
        const double dx = (double)m.xyz[3 * j] - xi, dy = (double)m.xyz[3 * j + 1] - yi, dz = (double)m.xyz[3 * j + 2] - zi;
        const double dp = m.phi64[j] - pi;
        a00 += dx * dx; a01 += dx * dy; a02 += dx * dz;
        a11 += dy * dy; a12 += dy * dz; a22 += dz * dz;
        b0 += dp * dx; b1 += dp * dy; b2 += dp * dz;
    }
    for (int o = kLanesPerRow / 2; o > 0; o >>= 1) {
        a00 += __shfl_xor_sync(0xffffffffu, a00, o); a01 += __shfl_xor_sync(0xffffffffu, a01, o);
        a02 += __shfl_xor_sync(0xffffffffu, a02, o); a11 += __shfl_xor_sync(0xffffffffu, a11, o);
        a12 += __shfl_xor_sync(0xffffffffu, a12, o); a22 += __shfl_xor_sync(0xffffffffu, a22, o);
        b0 += __shfl_xor_sync(0xffffffffu, b0, o); b1 += __shfl_xor_sync(0xffffffffu, b1, o);
        b2 += __shfl_xor_sync(0xffffffffu, b2, o);
    }
    if (!live || lane != 0) return;
    if (m.phiTrace != m.phi64) m.phiTrace[i] = pi;
    double* out = m.vfield + 3 * (size_t)i;
    if (hull) {
        out[0] = out[1] = out[2] = 0.0;
        return;
    }
    const double c00 = a11 * a22 - a12 * a12, c01 = a02 * a12 - a01 * a22, c02 = a01 * a12 - a02 * a11;
    const double det = a00 * c00 + a01 * c01 + a02 * c02;
    if (det == 0.0 || !(det == det)) {
        out[0] = __longlong_as_double(0x7ff8000000000000ll);
        out[1] = out[2] = 0.0;
        return;
    }
    const double c11 = a00 * a22 - a02 * a02, c12 = a01 * a02 - a00 * a12, c22 = a00 * a11 - a01 * a01;
    const double inv = 1.0 / det;
    out[0] = -(c00 * b0 + c01 * b1 + c02 * b2) * inv;
    out[1] = -(c01 * b0 + c11 * b1 + c12 * b2) * inv;
    out[2] = -(c02 * b0 + c12 * b1 + c22 * b2) * inv;
}

// Packed tetrahedron records, 128 bytes each: vertex 0 (3 floats) and the
// six-fold volume (float), the gradients n1, n2, n3 of the barycentric
// coordinates of vertices 1..3 (9 doubles: lambda_k(p) = n_k.(p - v0),
// lambda_0 = 1 - lambda_1 - lambda_2 - lambda_3), the neighbours (4 ints)
// the vertex ids (4 ints) and 3e-13 times the largest gradient component
// (double).  A walk step then tests the four faces with three dot products, and the same lambdas are the interpolation weights
// |sub-volume| / volume of tetWeights (geometry_3d.cpp:916-980).  A flat
// tetrahedron stores zero gradients and volume 0.
constexpr int kTetWords = 32;
__global__ void k_pack_tets(DevMesh m, float* pack) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m.ntets) return;
    float* o = pack + kTetWords * (size_t)t;
    int v[4];
    V3 P[4];
    for (int k = 0; k < 4; k++) {
        v[k] = m.tet_v[4 * t + k];
        P[k] = ld3(m.xyz, v[k]);
    }
    const V3 e1{P[1].x - P[0].x, P[1].y - P[0].y, P[1].z - P[0].z};
    const V3 e2{P[2].x - P[0].x, P[2].y - P[0].y, P[2].z - P[0].z};
    const V3 e3{P[3].x - P[0].x, P[3].y - P[0].y, P[3].z - P[0].z};
    const V3 c23{e2.y * e3.z - e2.z * e3.y, e2.z * e3.x - e2.x * e3.z, e2.x * e3.y - e2.y * e3.x};
    const V3 c31{e3.y * e1.z - e3.z * e1.y, e3.z * e1.x - e3.x * e1.z, e3.x * e1.y - e3.y * e1.x};
    const V3 c12{e1.y * e2.z - e1.z * e2.y, e1.z * e2.x - e1.x * e2.z, e1.x * e2.y - e1.y * e2.x};
    const double vol6 = e1.x * c23.x + e1.y * c23.y + e1.z * c23.z;
    const double inv = vol6 != 0.0 ? 1.0 / vol6 : 0.0;
    o[0] = m.xyz[3 * v[0]];
    o[1] = m.xyz[3 * v[0] + 1];
    o[2] = m.xyz[3 * v[0] + 2];
    o[3] = (float)vol6;
    if (vol6 != 0.0 && o[3] == 0.0f) o[3] = 1e-38f;  // keep "not flat" when the float underflows
    double* g = reinterpret_cast<double*>(o + 4);
    g[0] = c23.x * inv; g[1] = c23.y * inv; g[2] = c23.z * inv;
    g[3] = c31.x * inv; g[4] = c31.y * inv; g[5] = c31.z * inv;
    g[6] = c12.x * inv; g[7] = c12.y * inv; g[8] = c12.z * inv;
    int* oi = reinterpret_cast<int*>(o);
    for (int k = 0; k < 4; k++) {
        oi[22 + k] = m.tet_n[4 * t + k];
        oi[26 + k] = v[k];
    }
    double gmax = 0.0;
    for (int k = 0; k < 9; k++) gmax = fmax(gmax, fabs(g[k]));
    reinterpret_cast<double*>(o)[15] = 3e-13 * gmax;
}

__device__ V3 vertex_field(const DevMesh& m, int i) {
    const V3 E{m.vfield[3 * (size_t)i], m.vfield[3 * (size_t)i + 1], m.vfield[3 * (size_t)i + 2]};
    if (E.x != E.x) {
        atomicOr(m.status, S_SINGULAR);
        return V3{0, 0, 0};
    }
    return E;
}

// One lane's slot of the warp's tetrahedra (see trace_ion): a packed record,
// and the vertex fields once interpolated from.  Every member is addressed
// with compile-time indices so that the slot lives in registers.  An empty
// slot has t = -1 and zero gradients, which hold no point.
struct LaneTet {
    int t;
    int nb0, nb1, nb2, nb3;
    int v0, v1, v2, v3;
    float vol6;
    bool hasF;
    V3 P0;
    V3 G1, G2, G3;
    double gmax;  // 3e-13 times the largest gradient component
    V3 F0, F1, F2, F3;
};

__device__ __forceinline__ int pick4(int k, int x0, int x1, int x2, int x3) {
    return k == 0 ? x0 : (k == 1 ? x1 : (k == 2 ? x2 : x3));
}

__device__ __forceinline__ void load_slot(const DevMesh& m, LaneTet& s, int t) {
    const float4* p = reinterpret_cast<const float4*>(m.tetpack + kTetWords * (size_t)t);
    const float4 q0 = __ldg(p);
    const double2 g0 = __ldg(reinterpret_cast<const double2*>(p + 1));
    const double2 g1 = __ldg(reinterpret_cast<const double2*>(p + 2));
    const double2 g2 = __ldg(reinterpret_cast<const double2*>(p + 3));
    const double2 g3 = __ldg(reinterpret_cast<const double2*>(p + 4));
    const double2 g4 = __ldg(reinterpret_cast<const double2*>(p + 5));  // g[8], neighbours 0, 1
    const int4 q6 = __ldg(reinterpret_cast<const int4*>(p + 6));       // neighbours 2, 3, vertices 0, 1
    const int4 q7 = __ldg(reinterpret_cast<const int4*>(p + 7));       // vertices 2, 3, gmax
    s.t = t;
    s.P0 = V3{q0.x, q0.y, q0.z};
    s.vol6 = q0.w;
    s.G1 = V3{g0.x, g0.y, g1.x};
    s.G2 = V3{g1.y, g2.x, g2.y};
    s.G3 = V3{g3.x, g3.y, g4.x};
    s.gmax = __hiloint2double(q7.w, q7.z);
    const long long nb01 = __double_as_longlong(g4.y);
    s.nb0 = (int)(unsigned)(nb01 & 0xffffffffll);
    s.nb1 = (int)(unsigned)((unsigned long long)nb01 >> 32);
    s.nb2 = q6.x;
    s.nb3 = q6.y;
    s.v0 = q6.z;
    s.v1 = q6.w;
    s.v2 = q7.x;
    s.v3 = q7.y;
    s.hasF = false;
}

// Products and sums unfused, and in lane_field fused in a stated order: the
// step control's decisions turn on the last digit of the fields, so the
// arithmetic must not change with what the compiler finds to share.
__device__ __forceinline__ double dot_rn(V3 g, double x, double y, double z) {
    return __dadd_rn(__dadd_rn(__dmul_rn(g.x, x), __dmul_rn(g.y, y)), __dmul_rn(g.z, z));
}

// Barycentric coordinates of p in this lane's tetrahedron.  *inside: p lies
// inside for certain, every coordinate above a bound that is at least the
// rounding bounds the walk works with (1e-13 times the absolute sums of the
// products), so that the walk could end in no other tetrahedron.
struct Bary {
    double l0, l1, l2, l3;
};
__device__ __forceinline__ Bary lane_bary(const LaneTet& S, V3 p, bool* inside) {
    const double dx = p.x - S.P0.x, dy = p.y - S.P0.y, dz = p.z - S.P0.z;
    Bary b;
    b.l1 = dot_rn(S.G1, dx, dy, dz);
    b.l2 = dot_rn(S.G2, dx, dy, dz);
    b.l3 = dot_rn(S.G3, dx, dy, dz);
    b.l0 = 1.0 - b.l1 - b.l2 - b.l3;
    const double thr = S.gmax * (fabs(dx) + fabs(dy) + fabs(dz)) + 1e-13;
    *inside = b.l0 > thr && b.l1 > thr && b.l2 > thr && b.l3 > thr;
    return b;
}

// Sign of the side of face k (opposite vertex k) that p lies on, from the
// exact predicate on the vertex coordinates (as Predicates::orient3d decides
// in the reference).
__device__ __noinline__ int face_side_exact(const float* xyz, double snap, int i0, int i1, int i2, V3 p) {
    return orient_sign(ld3(xyz, i0), ld3(xyz, i1), ld3(xyz, i2), p, snap);
}

// The neighbour through which a walk to p leaves this lane's tetrahedron
// (-1: the hull), kHere when p lies beyond none of its faces.  Mostly every
// coordinate is clear of lane_bary's bound, and the walk takes the face that
// p is furthest beyond (in coordinates), the faces beyond which it lies in
// an order rotating from step to step once the walk is long.  Otherwise a
// coordinate decides its face unless it is within its own rounding bound of
// zero (about a thousand ulps of the terms summed), or the tetrahedron is
// flat; then the exact predicate decides.
// For a point within a mesh quantum of a face, the coordinates may put it on
// the other side than the predicate, which snaps the point to the mesh's
// grid, and tetrahedra that decide differently can send a walk round in
// circles.  A walk of kSnapStep steps goes on by the predicate on the snapped
// point alone, whose decisions agree, so that it ends.
constexpr int kSnapStep = 256;
constexpr int kHere = -3;
__device__ __forceinline__ int walk_exit(const DevMesh& m, const LaneTet& S, V3 p, const Bary& b, int step,
                                         unsigned rot) {
    const double dx = p.x - S.P0.x, dy = p.y - S.P0.y, dz = p.z - S.P0.z;
    const double thr = S.gmax * (fabs(dx) + fabs(dy) + fabs(dz)) + 1e-13;
    unsigned out = (b.l0 < -thr ? 1u : 0u) | (b.l1 < -thr ? 2u : 0u) | (b.l2 < -thr ? 4u : 0u) |
                   (b.l3 < -thr ? 8u : 0u);
    const bool clear = fabs(b.l0) > thr && fabs(b.l1) > thr && fabs(b.l2) > thr && fabs(b.l3) > thr;
    const bool exact = S.vol6 == 0.0f || step >= kSnapStep;
    if (clear && !exact && step < 24) {
        if (out == 0u) return kHere;
        double low = b.l0;
        int to = S.nb0;
        if (b.l1 < low) { low = b.l1; to = S.nb1; }
        if (b.l2 < low) { low = b.l2; to = S.nb2; }
        if (b.l3 < low) to = S.nb3;
        return to;
    }
    if (!clear || exact) {
        const double a1 = fabs(S.G1.x * dx) + fabs(S.G1.y * dy) + fabs(S.G1.z * dz);
        const double a2 = fabs(S.G2.x * dx) + fabs(S.G2.y * dy) + fabs(S.G2.z * dz);
        const double a3 = fabs(S.G3.x * dx) + fabs(S.G3.y * dy) + fabs(S.G3.z * dz);
        const double e1 = 1e-13 * a1, e2 = 1e-13 * a2, e3 = 1e-13 * a3, e0 = 1e-13 * (1.0 + a1 + a2 + a3);
        out = (b.l0 < -e0 ? 1u : 0u) | (b.l1 < -e1 ? 2u : 0u) | (b.l2 < -e2 ? 4u : 0u) | (b.l3 < -e3 ? 8u : 0u);
        unsigned sure = out | (b.l0 > e0 ? 1u : 0u) | (b.l1 > e1 ? 2u : 0u) | (b.l2 > e2 ? 4u : 0u) |
                        (b.l3 > e3 ? 8u : 0u);
        V3 q = p;
        if (exact) out = sure = 0u;
        if (step >= kSnapStep) q = V3{rint(p.x * m.snap) / m.snap, rint(p.y * m.snap) / m.snap, rint(p.z * m.snap) / m.snap};
        for (unsigned left = ~sure & 15u; left; left &= left - 1u) {
            const int k = __ffs((int)left) - 1;
            const int i0 = pick4(kFaceDev[k][0], S.v0, S.v1, S.v2, S.v3);
            const int i1 = pick4(kFaceDev[k][1], S.v0, S.v1, S.v2, S.v3);
            const int i2 = pick4(kFaceDev[k][2], S.v0, S.v1, S.v2, S.v3);
            if (face_side_exact(m.xyz, m.snap, i0, i1, i2, q) < 0) out |= 1u << k;
        }
    }
    if (out == 0u) return kHere;
    const unsigned r = rot & 3u;
    const unsigned turned = (out >> r) | (out << (4u - r));  // bit j: face (r + j) & 3
    const int k = (int)((r + (unsigned)__ffs((int)turned) - 1u) & 3u);
    return pick4(k, S.nb0, S.nb1, S.nb2, S.nb3);
}

// findTetrahedron over the warp's tetrahedra.  On entry S is the lane whose
// tetrahedron the walk starts from, b every lane's coordinates of p and bo
// those of a second point (other), which a slot loaded on the way gets as
// well.  Returns 0 with S the lane holding p's tetrahedron, -1 when p is
// outside the mesh, -2 when the walk exceeded its bound.  `next` is the slot
// that the next new record goes to, in turn; the slot `keep` stays.
__device__ __forceinline__ int warp_walk(const DevMesh& m, LaneTet& T, int lane, int& S, int& next, int keep, V3 p,
                                         Bary& b, V3 other, Bary& bo, bool& inOther, int limit, unsigned& rot) {
    for (int step = 0; step < limit; step++) {
        int to = kHere;
        if (lane == S) to = walk_exit(m, T, p, b, step, rot);
        rot++;
        to = __shfl_sync(0xffffffffu, to, S);
        if (to == kHere) {
            // a flat tetrahedron weights its vertices alike
            if (lane == S && T.vol6 == 0.0f) b.l0 = b.l1 = b.l2 = b.l3 = 0.25;
            return 0;
        }
        if (to < 0) return -1;
        const unsigned have = __ballot_sync(0xffffffffu, T.t == to);
        if (have) {
            S = __ffs((int)have) - 1;
            continue;
        }
        next = (next + 1) & 31;
        if (next == keep) next = (next + 1) & 31;
        if (lane == next) {
            load_slot(m, T, to);
            bool in;
            b = lane_bary(T, p, &in);
            bo = lane_bary(T, other, &inOther);
        }
        S = next;
    }
    return -2;
}

// The vertex fields of this lane's tetrahedron, once per record
__device__ __forceinline__ void lane_load_fields(const DevMesh& m, LaneTet& T) {
    if (T.hasF) return;
    T.F0 = vertex_field(m, T.v0);
    T.F1 = vertex_field(m, T.v1);
    T.F2 = vertex_field(m, T.v2);
    T.F3 = vertex_field(m, T.v3);
    T.hasF = true;
}

__device__ __forceinline__ double weighted(const Bary& b, double f0, double f1, double f2, double f3) {
    return fma(fabs(b.l3), f3, fma(fabs(b.l2), f2, fma(fabs(b.l0), f0, __dmul_rn(fabs(b.l1), f1))));
}

// Component c of the field interpolated in lane S's tetrahedron with the
// weights |b| (FastField::compute).
__device__ __forceinline__ double lane_field(const LaneTet& T, const Bary& b, int S, int c) {
    const double x = __shfl_sync(0xffffffffu, weighted(b, T.F0.x, T.F1.x, T.F2.x, T.F3.x), S);
    const double y = __shfl_sync(0xffffffffu, weighted(b, T.F0.y, T.F1.y, T.F2.y, T.F3.y), S);
    const double z = __shfl_sync(0xffffffffu, weighted(b, T.F0.z, T.F1.z, T.F2.z, T.F3.z), S);
    return c == 0 ? x : (c == 1 ? y : z);
}

// A vector whose component c the lanes with that component hold
__device__ __forceinline__ V3 gather3(double v) {
    return V3{__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 1), __shfl_sync(0xffffffffu, v, 2)};
}

__device__ double potential_at(const DevMesh& m, const double* phi, V3 p, int t) {
    const int* v = m.tet_v + 4 * t;
    double w[4];
    weights(m, t, p, w);
    return w[0] * phi[v[0]] + w[1] * phi[v[1]] + w[2] * phi[v[2]] + w[3] * phi[v[3]];
}

// Tetrahedron t2 shares a vertex with t1 and is not t1: membership of the
// set Geometry_3d::Table::adjacentTetrahedra (geometry_3d.cpp:1046-1096)
// builds for t1 by a walk over face neighbours.
__device__ bool shares_vertex(const DevMesh& m, int t1, int t2) {
    if (t2 < 0 || t2 == t1) return false;
    for (int a = 0; a < 4; a++) {
        const int va = m.tet_v[4 * t1 + a];
        for (int b = 0; b < 4; b++)
            if (va == m.tet_v[4 * t2 + b]) return true;
    }
    return false;
}

// Geometry_3d::Table::isBoundaryTetrahedron (geometry_3d.cpp:819-828)
__device__ bool boundary_tet(const DevMesh& m, int t) {
    for (int a = 0; a < 4; a++)
        if (m.flags[m.tet_v[4 * t + a]] & F_HULL) return true;
    return false;
}

// The accept / retry rule of the steppers other than the error-restricted
// one of the main path, for a trial point located in tetrahedron nt (< 0:
// outside the mesh): 0 NONE takes every step; 2 geometryRestricted_stepper
// (trajectory_3d.cpp:427-452) accepts a point in a tetrahedron sharing a
// vertex with the current one (or outside the mesh from a boundary
// tetrahedron), grows dt by 1.1 while the point stays in the current
// tetrahedron and shrinks it by 0.9 otherwise; 3 adaptive_stepper
// (:454-532) shrinks dt by 0.1 when the point leaves that set, then applies
// the error rule.  Returns true to accept, false to retry with the updated
// dt.
__device__ __forceinline__ bool stepper_verdict(const DevMesh& m, const TraceParams& tp, int tet, int nt, double rel,
                                                double* dt) {
    if (tp.stepper == 0) return true;
    if (tp.stepper == 2) {
        if (nt < 0 && boundary_tet(m, tet)) return true;
        if (shares_vertex(m, tet, nt)) return true;
        if (nt == tet) {
            *dt *= 1.1;
        } else {
            if (*dt == tp.dt_min) return true;
            *dt *= 0.9;
        }
        return false;
    }
    if (tp.stepper == 3 && nt >= 0 && nt != tet && !shares_vertex(m, tet, nt)) {
        *dt *= 0.1;
        return false;
    }
    if (rel < tp.tol || *dt == tp.dt_min) {
        if (rel != 0.0) {
            const double tmp = *dt * pow(tp.tol / rel, 0.25) * 0.9;
            if (tmp < *dt) *dt *= 1.1; else *dt = tmp;
        }
        return true;
    }
    const double tmp = *dt * pow(tp.tol / rel, 0.25) * 0.9;
    if (tmp > *dt) *dt *= 0.9; else *dt = tmp;
    return false;
}

// Point idx of the path of ion `slot` (Trajectory_3d::phaseVector,
// trajectory_3d.h:40-80), dropped beyond the path's capacity.
__device__ __forceinline__ void path_point(const TraceParams& tp, int slot, int idx, double t, V3 x, V3 v, int tet) {
    if (idx >= tp.path_cap) return;
    float4* p = reinterpret_cast<float4*>(tp.path + ((size_t)slot * tp.path_cap + idx) * 8);
    p[0] = make_float4((float)t, (float)x.x, (float)x.y, (float)x.z);
    p[1] = make_float4((float)v.x, (float)v.y, (float)v.z, __int_as_float(tet < 0 ? -1 : tet));
}

// The Cash-Karp tableau (Cash & Karp 1990) by rounds of two stages (see
// ck_trial): for the stages a = 2r and b = 2r + 1 of round r, the weight of
// a in b, those of a and of b in the next four stages (0 past the sixth),
// the fifth-order weights of a and b, and their differences to the
// fourth-order ones.
constexpr double kC5[6] = {37.0 / 378.0, 0.0, 250.0 / 621.0, 125.0 / 594.0, 0.0, 512.0 / 1771.0};
constexpr double kC4[6] = {2825.0 / 27648.0, 0.0, 18575.0 / 48384.0, 13525.0 / 55296.0, 277.0 / 14336.0, 1.0 / 4.0};
constexpr double kB20 = 3.0 / 40.0, kB21 = 9.0 / 40.0, kB30 = 3.0 / 10.0, kB31 = -9.0 / 10.0, kB32 = 6.0 / 5.0,
                 kB40 = -11.0 / 54.0, kB41 = 5.0 / 2.0, kB42 = -70.0 / 27.0, kB43 = 35.0 / 27.0,
                 kB50 = 1631.0 / 55296.0, kB51 = 175.0 / 512.0, kB52 = 575.0 / 13824.0, kB53 = 44275.0 / 110592.0,
                 kB54 = 253.0 / 4096.0;
#define TG_CK_ROUNDS(R)                                                                                            \
    {{(R)(1.0 / 5.0), (R)kB20, (R)kB30, (R)kB40, (R)kB50, (R)kB21, (R)kB31, (R)kB41, (R)kB51, (R)kC5[0],           \
      (R)kC5[1], (R)(kC5[0] - kC4[0]), (R)(kC5[1] - kC4[1])},                                                      \
     {(R)kB32, (R)kB42, (R)kB52, (R)0, (R)0, (R)kB43, (R)kB53, (R)0, (R)0, (R)kC5[2], (R)kC5[3],                   \
      (R)(kC5[2] - kC4[2]), (R)(kC5[3] - kC4[3])},                                                                 \
     {(R)kB54, (R)0, (R)0, (R)0, (R)0, (R)0, (R)0, (R)0, (R)0, (R)kC5[4], (R)kC5[5], (R)(kC5[4] - kC4[4]),         \
      (R)(kC5[5] - kC4[5])}}
__constant__ double kCk64[3][13] = TG_CK_ROUNDS(double);
__constant__ float kCk32[3][13] = TG_CK_ROUNDS(float);
template <typename R>
__device__ __forceinline__ R ck_coef(int r, int i) {
    if constexpr (sizeof(R) == 8) return kCk64[r][i];
    else return kCk32[r][i];
}

// The field of the current state: 2 its component is known (E), 1 the state
// is located (lane S holds its tetrahedron, b the coordinates), 0 neither.
// Every trial of a step evaluates its first stage at the same point, so a
// retried trial takes the field from here, and the first trial takes the
// location from the one that accepted the state.
struct Stage0 {
    double E;
    int tet;
    int mode;
};

// One Cash-Karp trial step (o5_integrator, trajectory_3d.cpp:583-676) of
// length dt from (x, v), its arithmetic in R: FP64, or FP32 as the reference
// integrates.  The state enters and leaves in double (rounded to R on the
// way in, so in FP32 it is the float state); the points of the stages are
// located and their fields interpolated as in FP64, then rounded to R.
// *rel: the largest relative error of a position or velocity component (as
// errorRestricted_stepper forms it, trajectory_3d.cpp:366-387).  Returns
// false when a walk exceeded its bound.
// A lane holds one component (c) of every vector.  The position of stage b
// takes the increments h v_j of the stages before it, and v_j the fields of
// the stages before j: so position b does not wait for the field of stage
// b - 1, and the stages go in three rounds of two whose points are located
// and interpolated together.  Each later stage's sums take the increments as
// they come, in stage order, as one sum over them would.
template <typename R>
__device__ __forceinline__ bool ck_trial(const DevMesh& m, LaneTet& T, int lane, int c, int& S, int& next, Bary& b,
                                         const TraceParams& tp, unsigned& rot, bool direct, double xc, double vc,
                                         double k, double dt, double* nxo, double* nvo, double* exo, double* evo,
                                         double* relo, Stage0& s0) {
    const R xx = (R)xc, vv = (R)vc, kk = (R)k, h = (R)dt;
    R sx[6] = {xx, xx, xx, xx, xx, xx}, sv[6] = {vv, vv, vv, vv, vv, vv};
    R nx = xx, nv = vv, ex = 0, ev = 0;
    bool walkOk = true;
#pragma unroll 1
    for (int r = 0; r < 3; r++) {
        const R dxa = sv[0] * h;
        const R wab = ck_coef<R>(r, 0);
        const V3 pa = gather3((double)sx[0]);
        const V3 pb = gather3((double)(sx[1] + wab * dxa));
        const int known = r == 0 ? s0.mode : 0;
        int ra = 0, rb = 0;
        bool ina = false, inb = false;
        if (known == 2) {
            // the walk to b starts from the state's tetrahedron, also after a
            // trial whose stages ended in others: where b lies on a vertex or
            // a face, as all-FP32 positions do for many trials, the start
            // decides which tetrahedron holds it
            const unsigned have = __ballot_sync(0xffffffffu, T.t == s0.tet);
            if (have) {
                S = __ffs((int)have) - 1;
            } else {
                S = next = (next + 1) & 31;
                if (lane == S) load_slot(m, T, s0.tet);
            }
        }
        int Sa = S;
        Bary bb = lane_bary(T, pb, &inb);
        if (known == 0) {
            b = lane_bary(T, pa, &ina);
            const unsigned hit = direct ? 0u : __ballot_sync(0xffffffffu, ina);
            if (hit) {
                S = __ffs((int)hit) - 1;
            } else {
                const int from = S;
                ra = warp_walk(m, T, lane, S, next, -1, pa, b, pb, bb, inb, tp.walk_limit, rot);
                if (ra < 0) S = from;
            }
            Sa = S;
        }
        {
            const unsigned hit = direct ? 0u : __ballot_sync(0xffffffffu, inb);
            if (hit) {
                S = __ffs((int)hit) - 1;
            } else {
                const int from = S;
                rb = warp_walk(m, T, lane, S, next, Sa, pb, bb, pa, b, ina, tp.walk_limit, rot);
                if (rb < 0) S = from;
            }
        }
        walkOk = walkOk && ra != -2 && rb != -2;
        if ((lane == Sa && ra == 0 && known != 2) || (lane == S && rb == 0)) lane_load_fields(m, T);
        double Ea = s0.E;
        if (known != 2) {
            Ea = lane_field(T, b, Sa, c);
            if (ra < 0) Ea = 0.0;
        }
        double Eb = lane_field(T, bb, S, c);
        if (rb < 0) Eb = 0.0;
        if (r == 0) {
            s0.tet = __shfl_sync(0xffffffffu, T.t, Sa);
            s0.E = Ea;
            s0.mode = 2;
        }
        const R dva = (R)Ea * kk * h, dvb = (R)Eb * kk * h;
        const R dxb = (sv[1] + wab * dva) * h;
        const R c5a = ck_coef<R>(r, 9), c5b = ck_coef<R>(r, 10), dca = ck_coef<R>(r, 11), dcb = ck_coef<R>(r, 12);
        nx += c5a * dxa; nv += c5a * dva; ex += dca * dxa; ev += dca * dva;
        nx += c5b * dxb; nv += c5b * dvb; ex += dcb * dxb; ev += dcb * dvb;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const R wa = ck_coef<R>(r, 1 + j), wb = ck_coef<R>(r, 5 + j);
            sx[j] = sx[j + 2] + wa * dxa;
            sv[j] = sv[j + 2] + wa * dva;
            sx[j] += wb * dxb;
            sv[j] += wb * dvb;
        }
    }
    // lanes 0..3 of every eight take the position's quotient, the others the
    // velocity's
    const R num = (lane & 4) ? ev : ex, den = (lane & 4) ? nv : nx;
    R rel = 0;
    if (den != (R)0) rel = fmax(rel, fabs(num / den));
    rel = fmax(rel, __shfl_xor_sync(0xffffffffu, rel, 1));
    rel = fmax(rel, __shfl_xor_sync(0xffffffffu, rel, 2));
    rel = fmax(rel, __shfl_xor_sync(0xffffffffu, rel, 4));
    *nxo = (double)nx;
    *nvo = (double)nv;
    *exo = (double)ex;
    *evo = (double)ev;
    *relo = (double)rel;
    return walkOk;
}

// errorRestricted_stepper's rule (trajectory_3d.cpp:396-421) in R: accept
// when rel is below the threshold or the step is at its floor, and adjust
// dt by (tol / rel)^(1/4) with the safety factor 0.9, growing by at most
// 1.1 and shrinking by at least 0.9.  Returns true to accept.
template <typename R>
__device__ __forceinline__ bool error_rule(double relIn, const TraceParams& tp, double* dtIo) {
    const R rel = (R)relIn, tol = (R)tp.tol;
    R dt = (R)*dtIo;
    const bool accept = rel < tol || dt == (R)tp.dt_min;
    // the fourth root of a quotient below 0.9^-4 = 1.5242 leaves tmp below
    // dt, so that an accepted step's dt grows by 1.1 whatever the root
    if (accept && rel != (R)0 && tol < rel * (R)1.52) {
        dt = dt * (R)1.1;
    } else if (!accept || rel != (R)0) {
        const R tmp = dt * (R)pow(tol / rel, (R)0.25) * (R)0.9;
        if (accept) dt = tmp < dt ? dt * (R)1.1 : tmp;
        else dt = tmp > dt ? dt * (R)0.9 : tmp;
    }
    *dtIo = (double)dt;
    return accept;
}

// One ion from x (velocity v, charge/mass k) into *out, by one warp; with
// kPath its path and error estimate go to slot `slot` of tp's path buffers
// (a separate instantiation, so that the flights without a path keep their
// registers).
// kPrec: the arithmetic of the Cash-Karp steps (TraceParams::precision),
// fixed per instantiation so that each kernel holds only its own registers.
//
// A flight is a chain of trial steps, each a chain of point locations and
// interpolations, so what counts is the length of that chain.  Every lane
// keeps the record (and vertex fields) of one of the last 32 tetrahedra the
// flight came through, and a point is located by all lanes testing theirs at
// once: 60% of the trials are retries with a smaller step, whose points lie
// in tetrahedra already there, and so do most points of a step that is not
// the first through a region.  Only a point in none of them walks on
// (warp_walk), over the lanes' records where the walk crosses them.
// Measured on the B200: 1000 mixed-precision ions on a 307k-cell tip 15.2 ms
// with one thread per ion, 6.1 ms so; 4096 FP64 ions on a 514k-cell alloy tip
// 40.4 and 10.4 ms (13.2 before the ions beside a coordinate plane started
// first); impacts and trials of both, and of 7,096 all-FP32 ions, the same to
// the bit.  About 1300 warp instructions per trial at 5 cycles each (2.2 of
// them waits on the fixed latency of dependent FP64 arithmetic), instead of
// 3400.  At 240 registers eight warps fit an SM; in the first version of this
// kernel (7.4 ms for the 1000 ions) 12 or 16 spilled and took 8.6 and 10.4 ms.
template <bool kPath, int kPrec>
__device__ __forceinline__ void trace_ion(const DevMesh& m, V3 x, V3 v, double k, int guessTet, const TraceParams& tp,
                                          unsigned rot, int slot, ImpactOut* out) {
    const int lane = threadIdx.x & 31;
    const int c = min(lane & 3, 2);  // the lane's component of the state
    const V3 x0 = x;
    ImpactOut res;
    double time = 0.0;
    int tet = locate(m, x, guessTet, tp.walk_limit, rot);
    res.steps = 0;
    res.trials = 0;
    res.last_tet = tet;
    res.last_pos[0] = (float)x.x; res.last_pos[1] = (float)x.y; res.last_pos[2] = (float)x.z;
    res.last_phi = 0.0f;
    if (kPath) {
        float* e = tp.path_err + 12 * (size_t)slot;
        if (lane < 12) e[lane] = 0.0f;
        if (lane == 0 && tet >= 0) path_point(tp, slot, 0, 0.0, x, v, tet);  // Trajectory_3d::init (:99-123)
        __syncwarp();
    }
    if (tet < 0) {
        if (tet == -2) atomicOr(m.status, S_WALK_LIMIT);
        res.status = -1;  // Trajectory_3d::init: initial point is outside
        res.stop[0] = (float)x.x; res.stop[1] = (float)x.y; res.stop[2] = (float)x.z;
        res.stop_time = 0.0f;
        if (lane == 0) *out = res;
        return;
    }
    // a short bound on the walks keeps them as they are: each from the last
    // located point's tetrahedron
    const bool direct = tp.walk_limit < kSnapStep;
    LaneTet T{};
    T.t = -1;
    int S = 0;     // the lane holding the last located point's tetrahedron
    int next = 0;  // the slot filled last
    Bary b{};      // every lane's coordinates of the current state, once it is located
    if (lane == 0) {
        load_slot(m, T, tet);
        bool in;
        b = lane_bary(T, x, &in);
        if (T.vol6 == 0.0f) b.l0 = b.l1 = b.l2 = b.l3 = 0.25;
        lane_load_fields(m, T);
    }
    double xc = c == 0 ? x.x : (c == 1 ? x.y : x.z), vc = c == 0 ? v.x : (c == 1 ? v.y : v.z);
    Stage0 s0;
    s0.E = lane_field(T, b, S, c);
    s0.tet = tet;
    s0.mode = 2;
    int status;
    if (!__any_sync(0xffffffffu, s0.E != 0.0)) {
        status = 1;  // NO_FIELD
    } else {
        status = 3;  // ITERATION_LIMIT_PASSED unless another exit is taken
        double dt = tp.dt0;
        bool loBefore = kPrec == 1;
        for (int it = 0; it < tp.max_steps; it++) {
            double nxc = 0.0, nvc = 0.0;
            double used = dt;
            bool accepted = false;
            int nt = -1;
            V3 nx{};
            // FP32 arithmetic for this step: always with precision 1, and
            // with precision 2 once the ion is beyond fp64_radius of its start
            const double ddx = x.x - x0.x, ddy = x.y - x0.y, ddz = x.z - x0.z;
            const bool lo = kPrec != 0 && tp.integrator == 1 &&
                            (kPrec == 1 || ddx * ddx + ddy * ddy + ddz * ddz > tp.fp64_radius2);
            // the first step in FP32 starts from the state rounded to float
            if (kPrec == 2 && lo != loBefore) s0.mode = 0;
            loBefore = lo;
            for (int tries = 0; tries < tp.stepper_limit; tries++) {
                res.trials++;
                if (lo) {
                    if ((float)dt < (float)tp.dt_min) dt = (double)(float)tp.dt_min;
                } else if (dt < tp.dt_min) {
                    dt = tp.dt_min;
                }
                used = dt;
                double rel = 0.0, exc = 0.0, evc = 0.0;
                bool take = false;
                if (tp.integrator == 0) {
                    // o1_integrator (trajectory_3d.cpp:560-581): Euler; the
                    // error estimate is the next state times dt^2
                    if (s0.mode == 1) {
                        if (lane == S) lane_load_fields(m, T);
                        s0.E = lane_field(T, b, S, c);
                        s0.mode = 2;
                    }
                    nvc = vc + dt * s0.E * k;
                    nxc = xc + dt * vc;
                    rel = __any_sync(0xffffffffu, nxc != 0.0 || nvc != 0.0) ? dt * dt : 0.0;
                    exc = nxc * (used * used);
                    evc = nvc * (used * used);
                } else {
                    bool walkOk;
                    if (kPrec == 1 || (kPrec == 2 && lo))
                        walkOk = ck_trial<float>(m, T, lane, c, S, next, b, tp, rot, direct, xc, vc, k, dt, &nxc, &nvc,
                                                 &exc, &evc, &rel, s0);
                    else
                        walkOk = ck_trial<double>(m, T, lane, c, S, next, b, tp, rot, direct, xc, vc, k, dt, &nxc,
                                                  &nvc, &exc, &evc, &rel, s0);
                    if (!walkOk && lane == 0) atomicOr(m.status, S_WALK_LIMIT);
                }
                if (kPath && lane < 3) {
                    // the latest trial's error vector
                    float* e = tp.path_err + 12 * (size_t)slot + 6;
                    e[c] = (float)exc;
                    e[3 + c] = (float)evc;
                }
                const bool errorRule = tp.stepper == 1 && tp.integrator != 0;
                const bool byTet = tp.stepper == 2 || tp.stepper == 3;  // verdicts that look at the tetrahedron
                if (!byTet) {
                    if (!errorRule) take = stepper_verdict(m, tp, tet, -1, rel, &dt);
                    else if (kPrec == 0) take = error_rule<double>(rel, tp, &dt);
                    else take = lo ? error_rule<float>(rel, tp, &dt) : error_rule<double>(rel, tp, &dt);
                    if (!take) continue;
                }
                // the trial point located, for the verdict or the next step
                nx = gather3(nxc);
                bool in;
                b = lane_bary(T, nx, &in);
                const unsigned hit = direct ? 0u : __ballot_sync(0xffffffffu, in);
                if (hit) {
                    S = __ffs((int)hit) - 1;
                    nt = 0;
                } else {
                    const int from = S;
                    Bary bo;
                    nt = warp_walk(m, T, lane, S, next, -1, nx, b, nx, bo, in, tp.walk_limit, rot);
                    if (nt < 0) S = from;
                }
                if (nt == -2 && lane == 0) atomicOr(m.status, S_WALK_LIMIT);
                if (nt == 0) nt = __shfl_sync(0xffffffffu, T.t, S);
                if (byTet) take = stepper_verdict(m, tp, tet, nt, rel, &dt);
                if (take) {
                    accepted = true;
                    break;
                }
            }
            if (!accepted) {
                status = 2;  // STEPPER_LIMIT_PASSED
                break;
            }
            res.steps++;
            if (kPath) {
                // Trajectory_3d::cumulative_error (trajectory_3d.cpp:683-700)
                // with the accepted step's error: each of the six components
                // becomes sqrt(current^2 + step^2), in float as the reference
                // keeps it
                __syncwarp();
                if (lane < 6) {
                    float* e = tp.path_err + 12 * (size_t)slot;
                    e[lane] = sqrtf(e[lane] * e[lane] + e[6 + lane] * e[6 + lane]);
                }
                const V3 nv = gather3(nvc);
                if (lane == 0) path_point(tp, slot, res.steps, time + used, nx, nv, nt);
                __syncwarp();
            }
            const double tnext = lo ? (double)((float)time + (float)used) : time + used;
            if (nt < 0) {
                // left the mesh: the previous point is the last inside it
                res.last_tet = tet;
                res.last_pos[0] = (float)x.x; res.last_pos[1] = (float)x.y; res.last_pos[2] = (float)x.z;
            }
            x = nx;
            xc = nxc;
            vc = nvc;
            time = tnext;
            tet = nt;
            if (nt < 0) {
                tet = -1;
                status = 5;  // SYSTEM_LIMIT_PASSED
                break;
            }
            s0.tet = nt;
            s0.mode = 1;
        }
    }
    v = gather3(vc);
    if (tet >= 0) {
        res.last_tet = tet;
        res.last_pos[0] = (float)x.x; res.last_pos[1] = (float)x.y; res.last_pos[2] = (float)x.z;
    }
    res.last_phi = res.last_tet >= 0 ? (float)potential_at(m, m.phiTrace, V3{res.last_pos[0], res.last_pos[1],
                                                                              res.last_pos[2]},
                                                           res.last_tet)
                                     : 0.0f;
    // extrapolate to the top plane along the last velocity
    const double dtz = (tp.top_z - x.z) / v.z;
    res.stop[0] = (float)(x.x + dtz * v.x);
    res.stop[1] = (float)(x.y + dtz * v.y);
    res.stop[2] = (float)(x.z + dtz * v.z);
    res.stop_time = (float)(time + dtz);
    res.status = status;
    if (kPath) {
        // Trajectory_3d::extrapolate (trajectory_3d.cpp:303-332): the last
        // point, located from the last tetrahedron (outside stays outside;
        // a flight at rest, NO_FIELD, extrapolates to a non-finite point)
        const V3 p{x.x + dtz * v.x, x.y + dtz * v.y, x.z + dtz * v.z};
        int pt = -1;
        if (tet >= 0 && isfinite(p.x) && isfinite(p.y) && isfinite(p.z)) {
            pt = locate(m, p, tet, tp.walk_limit, rot);
            if (pt == -2 && lane == 0) atomicOr(m.status, S_WALK_LIMIT);
        }
        if (lane == 0) path_point(tp, slot, res.steps + 1, time + dtz, p, v, pt);
        const float fdt = (float)dtz;
        if (fdt > 0.0f && lane == 0) {
            float* e = tp.path_err + 12 * (size_t)slot;
#pragma unroll
            for (int j = 0; j < 3; j++) e[j] += fdt * e[3 + j];
        }
    }
    if (lane == 0) *out = res;
}

// One ion per warp, one warp per block: as the flights' lengths differ by an
// order of magnitude, the blocks waiting take the place of each that ends.
// order (may be null): the ions in the order of their blocks.
template <bool kPath, int kPrec>
__global__ void __launch_bounds__(32) k_trace(DevMesh m, int nIons, const float* start, const float* vel,
                                              const float* qm, const int32_t* guess, const int32_t* order,
                                              TraceParams tp, ImpactOut* out) {
    if ((int)blockIdx.x >= nIons) return;
    const int ion = order ? order[blockIdx.x] : (int)blockIdx.x;
    const V3 x{start[3 * (size_t)ion], start[3 * (size_t)ion + 1], start[3 * (size_t)ion + 2]};
    const V3 v = vel ? V3{vel[3 * (size_t)ion], vel[3 * (size_t)ion + 1], vel[3 * (size_t)ion + 2]} : V3{0, 0, 0};
    trace_ion<kPath, kPrec>(m, x, v, qm[ion], guess ? guess[ion] : 0, tp, (unsigned)ion * 7u, ion, out + ion);
}

// A single ion, its start passed by value (no staging copy)
template <bool kPath, int kPrec>
__global__ void __launch_bounds__(32) k_trace_one(DevMesh m, float x, float y, float z, float vx, float vy, float vz,
                                                  float qm, int guess, TraceParams tp, ImpactOut* out) {
    trace_ion<kPath, kPrec>(m, V3{x, y, z}, V3{vx, vy, vz}, qm, guess, tp, 0u, 0, out);
}

__global__ void k_potential_at(DevMesh m, int n, const float* xyz, const int32_t* guess, int limit, float* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned rot = (unsigned)i;
    const V3 p{xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
    const int t = locate(m, p, guess ? guess[i] : 0, limit, rot);
    if (t == -2) atomicOr(m.status, S_WALK_LIMIT);
    out[i] = t >= 0 ? (float)potential_at(m, m.phi64, p, t) : 0.0f;
}

}  // namespace

int trace_resident() {
    static const int n = [] {  // initialised once, also under concurrent host threads
        int dev = 0, sms = 148, perSM = 8;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_trace<false, 0>, 32, 0) != cudaSuccess) perSM = 8;
        return (sms > 0 ? sms : 148) * (perSM > 0 ? perSM : 8);
    }();
    return n;
}
void launch_trace(const DevMesh& m, int nIons, const float* start, const float* vel, const float* qm,
                  const int32_t* guess, const int32_t* order, TraceParams tp, ImpactOut* out, cudaStream_t s) {
    if (nIons <= 0) return;
    count_launch();
    auto go = [&](auto kernel) { kernel<<<nIons, 32, 0, s>>>(m, nIons, start, vel, qm, guess, order, tp, out); };
    const int prec = tp.precision == 1 ? 1 : (tp.precision == 2 ? 2 : 0);
    if (tp.path) {
        if (prec == 0) go(k_trace<true, 0>); else if (prec == 1) go(k_trace<true, 1>); else go(k_trace<true, 2>);
    } else {
        if (prec == 0) go(k_trace<false, 0>); else if (prec == 1) go(k_trace<false, 1>); else go(k_trace<false, 2>);
    }
}
void launch_pack_tets(const DevMesh& m, float* pack, cudaStream_t s) {
    if (m.ntets > 0) { count_launch(); k_pack_tets<<<(m.ntets + kBlock - 1) / kBlock, kBlock, 0, s>>>(m, pack); }
}
void launch_vertex_fields(const DevMesh& m, cudaStream_t s, const int32_t* cells, int count) {
    const long long items = cells ? count : m.n;
    if (m.n > 0 && items > 0) {
        count_launch();
        const long long threads = items * kLanesPerRow;
        k_vertex_fields<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(m, cells, (int)items);
    }
}
void launch_trace_one(const DevMesh& m, const float start[3], const float vel[3], float qm, int guess, TraceParams tp,
                      ImpactOut* out, cudaStream_t s) {
    count_launch();
    auto go = [&](auto kernel) {
        kernel<<<1, 32, 0, s>>>(m, start[0], start[1], start[2], vel[0], vel[1], vel[2], qm, guess, tp, out);
    };
    const int prec = tp.precision == 1 ? 1 : (tp.precision == 2 ? 2 : 0);
    if (tp.path) {
        if (prec == 0) go(k_trace_one<true, 0>); else if (prec == 1) go(k_trace_one<true, 1>); else go(k_trace_one<true, 2>);
    } else {
        if (prec == 0) go(k_trace_one<false, 0>); else if (prec == 1) go(k_trace_one<false, 1>);
        else go(k_trace_one<false, 2>);
    }
}
void launch_potential_at(const DevMesh& m, int n, const float* xyz, const int32_t* guess, int walkLimit, float* out,
                         cudaStream_t s) {
    if (n > 0) { count_launch(); k_potential_at<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(m, n, xyz, guess, walkLimit, out); }
}

}  // namespace tgd
