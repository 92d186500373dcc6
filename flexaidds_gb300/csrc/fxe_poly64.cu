// fxe_poly64.cu — Voronoi contact surfaces and complementarity scoring in double precision
// (reference precision; fxe_voronoi.cu holds the single-precision form). The candidate lists come
// from contacts_kernel (fxe_contacts.cu).
//
// pose_kernel      one warp per pose: calc_region's loop over the scorable atoms in Calclist
//                  order (LIB/Vcontacts.cpp:74-139) — each atom's list without the saved atoms
//                  that kept no contact with it, its extended-radical-plane polyhedron started
//                  from the seed an earlier atom left (voronoi_poly2, :147-490), faces
//                  (order_faces, :699-831) and spherical areas (calc_areas, :838-1044), the
//                  contacts it keeps (save_areas) and the seeds it leaves (save_seeds) —
//                  then vcfunction's walk over the kept contacts (LIB/vcfunction.cpp:14-574).
//
// Compiled with --fmad=false and the reference's own expressions, so that every operation rounds
// as in the reference's double arithmetic.
//
// The atoms of one pose stay in order because the reference's results depend on it: which
// earlier atom seeds a hull decides the walk's start vertex, and with engulfing planes the
// atom centre lies outside its own cell, so a start from the closest plane can lie outside the
// cell and trace another polyhedron. Parallelism is across poses (one warp each), across the
// planes, edges, vertices and faces of each polyhedron (the 32 lanes), and, for the triangles and
// arcs of the areas, across a group of warps: the poses of a group step through their atoms together
// and pool those items. Stepping together also keeps the group's warps at the same place of 170 KB of
// code, more than the instruction caches hold: sixteen warps each on its own took 11.1 ms where the
// lockstep took 8.0 (2,000 poses of the benchmark's system).
//
// What bounds it: the FP64 unit, which takes one warp instruction per 64 cycles and SM quarter
// whatever its active lanes. Hence
//   * quotients in five FP64 instructions and roots in four (fxe_dmath.cuh);
//   * comparisons on the integer units (the bit patterns of doubles order like the doubles);
//   * the three coordinates of a vertex or a direction on three lanes, one instruction for all;
//   * the triangles and arcs of all the group's poses packed into full warps (25 and 7 per atom on
//     the benchmark's systems, of a warp's 32 lanes);
//   * plane tests decided in single precision with an error bound wherever that is certain.
#include <algorithm>
#include <cfloat>
#include <climits>

#include "fxe_common.cuh"
#include "fxe_dmath.cuh"

namespace fxe {
namespace f64 {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kFaceWords = (kMaxCand + 31) / 32;
constexpr uint8_t kNone = 255;
constexpr int kAtomNone = 5;     // an atom without contacts
constexpr int kAtomWalking = 4;  // the hull walk goes on in the group's next step
constexpr int kAtomRetry = 3;    // the atom outgrew this shape's capacities: score the pose with the large one

// Warps of a block, one block per SM, in groups that step through their poses' atoms together.
constexpr int kWarps = 16;
// Batches of edges a hull walk may step before its warp meets its group (it goes on in the group's
// next step): a walk takes 5.4 on average, many more when it fails. 2,000 poses of the benchmark's system
// take 7.77 ms with 8, 7.59 with 10, 7.40 with 12, 7.37 with 16, 7.36 with 20.
constexpr int kWalkBudget = 16;

// Capacities of one polyhedron. The compact shape holds the polyhedra of ordinary poses (on the
// benchmark's systems at most 44 vertices inside the sphere, 125 face points and 125 area items over
// 2,300 atoms; means 17, 43 and 33) and any hull walk and its arc points (176 vertices: those past
// `verts` lie in storage the faces use later), in 14.5 KB per pose, so that sixteen poses fit an SM. A
// pose one of whose atoms outgrows it is scored again, from its start, in the large shape when its
// group has no other pose.
// (With 256 items one pose of the benchmark's in 8,000 was: 3.2 ms more for its launch. With 290 none of
// 130,000.)
template <int kV, int kX, int kP, int kI, int kN>
struct Shape {
    static constexpr int verts = kV;         // of the faces; vertex indices are bytes (255 means "none")
    static constexpr int walk_verts = kX;    // of the hull walk and its arc points
    static constexpr int pts = kP;
    static constexpr int items = kI;
    static constexpr int poses = kN;         // of a block at a time
    static constexpr int vwords = (kV + 31) / 32;
    static constexpr int over = kV >= kMaxVerts ? kAtomCapacity : kAtomRetry;
};
using Compact = Shape<104, kMaxVerts, 352, 290, kWarps>;
using Large = Shape<kMaxVerts, kMaxVerts, kMaxFacePts, 3 * kMaxFacePts + 8, 5>;

struct __align__(32) real4 {
    double x, y, z, w;
};
__device__ __forceinline__ real4 make_real4(double x, double y, double z, double w) { return real4{x, y, z, w}; }
__device__ __forceinline__ double comp(const real4& v, int c) { return reinterpret_cast<const double*>(&v)[c]; }

// Quotients, roots and arc tangents out of line: the kernel's code outgrows the instruction caches (with
// quotients and roots in line 2,000 poses of the benchmark's system take 8.27 ms instead of 7.49).
__device__ __noinline__ double ddiv(double a, double b) {
    bool slow;
    double q = div_short(a, b, &slow);
    if (slow) q = plain_div(a, b);
    return q;
}
__device__ __noinline__ double dsqrt(double x) {
    bool slow;
    double g = sqrt_short(x, &slow);
    if (slow) g = plain_sqrt(x);
    return g;
}
__device__ __noinline__ double datan(double x) { return atan(x); }

// --- warp helpers -------------------------------------------------------------------------------
__device__ __forceinline__ int warp_sum(int v) { return __reduce_add_sync(kFull, v); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

__device__ __forceinline__ int warp_excl_scan(int v, int lane, int* total) {
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    *total = __shfl_sync(kFull, x, 31);
    return x - v;
}

// The smallest key (bit pattern of a double that is not negative) and, of the lanes that hold it,
// the smallest index.
__device__ __forceinline__ void warp_argmin(long long& key, int& i) {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_min_sync(kFull, hi);
    const unsigned ml = __reduce_min_sync(kFull, hi == mh ? lo : 0xffffffffu);
    i = __reduce_min_sync(kFull, hi == mh && lo == ml ? i : INT_MAX);
    key = (long long)(((unsigned long long)mh << 32) | ml);
}

// ------------------------------------------------------------------------------------------
// per-warp workspace of one polyhedron
// ------------------------------------------------------------------------------------------
template <class Sh>
struct Vor {
    real4 pl[kMaxPlanes];              // plane A.x + D = 0 (A unit normal, D = -plane distance)
    union {
        float4 plf[kMaxPlanes];        // the planes rounded to single precision, for pre-tests
        uint32_t vmask[kMaxPlanes * Sh::vwords];   // after the walk: per plane, its vertices
    };
    // vertex x, y, z, distance to the atom centre; then the two points of the lens two engulfing
    // planes cut
    real4 vx[Sh::verts + 2];
    union {
        struct {
            real4 vx[Sh::walk_verts - Sh::verts + 1];   // the walk's vertices and arc points from Sh::verts on
            // (two spare slots: the step that reaches the 200-edge limit writes up to two edges)
            uchar4 ep[kMaxEdges + 2];      // plane0, plane1, start plane, end plane
            uchar2 es[kMaxEdges + 2];      // start vertex, end vertex
            uint8_t flip[kMaxEdges + 2];   // the direction is minus the planes' cross product
        } e;
        struct {
            double val[Sh::items];            // test points; cosine keys; the area items' values
            uint32_t item[Sh::items];         // the area items: triangles, then arcs
            uint8_t pt[Sh::pts];
        } f;
    } u;
    float4 centre;                     // project_points' fallback centre
    double rado;
    float rr;                          // rado squared in single precision, as the reference squares it
    uchar4 vp[Sh::walk_verts];         // the vertex's planes (kNone = sphere)
    int cidx[kMaxCand];                // Calc index of each contact
    uint16_t foff[kMaxCand + 1];
    union {
        struct {
            uint16_t toff[kMaxCand + 1];   // per face: first triangle / arc item
            uint16_t aoff[kMaxCand + 1];
        };
        uint8_t elist[kMaxEdges + 8];      // before the faces: the hull edges with an end outside the sphere
    };
    uint8_t cslot[kMaxCand];           // the contact's slot in the atom's candidate list
    uint8_t fnp[kMaxCand];
    uint8_t fseed[kMaxCand];           // the face's first vertex of three contact planes (kNone: none)
    uint8_t flag[kMaxPlanes];
    union {
        uint8_t sprev[kMaxCand];       // per face: point 1 before a replayed stale read (kNone: none)
        uint8_t flist[kMaxCand];       // before and after: faces whose test point is checked
    };
    uint32_t excl[kFaceWords];         // candidates left out of the atom's list
    uint32_t cmask[kFaceWords];        // faces with a test point
    uint32_t bad[kFaceWords];          // faces whose test point lies in front of another plane
    int eng[4];
    int epi;
    int nt, na, ne;                    // triangle items, the faces' own arcs, credited arcs
};

template <class Sh>
struct PoseShared {
    Vor<Sh> v;
    uint8_t order[kMaxLig];            // mobile atoms in Calclist order
    uint32_t done[kMaskWords];         // mobile atoms whose contacts are saved
};

__device__ __forceinline__ double dot3(const real4& a, double x, double y, double z) {
    return a.x * x + a.y * y + a.z * z;
}

// solve_3x3 (LIB/Vcontacts.cpp:1384-1414).
__device__ __noinline__ bool solve3(const real4& e0, const real4& e1, const real4& e2, double* pt) {
    const double c00 = e1.y * e2.z - e2.y * e1.z;
    const double c01 = -e1.x * e2.z + e2.x * e1.z;
    const double c02 = e1.x * e2.y - e2.x * e1.y;
    const double c10 = -e0.y * e2.z + e2.y * e0.z;
    const double c11 = e0.x * e2.z - e2.x * e0.z;
    const double c12 = -e0.x * e2.y + e2.x * e0.y;
    const double c20 = e0.y * e1.z - e1.y * e0.z;
    const double c21 = -e0.x * e1.z + e1.x * e0.z;
    const double c22 = e0.x * e1.y - e1.x * e0.y;
    const double det = e0.x * c00 + e0.y * c01 + e0.z * c02;
    if (is0(det)) return false;
    pt[0] = ddiv(-(e0.w * c00 + e1.w * c10 + e2.w * c20), det);
    pt[1] = ddiv(-(e0.w * c01 + e1.w * c11 + e2.w * c21), det);
    pt[2] = ddiv(-(e0.w * c02 + e1.w * c12 + e2.w * c22), det);
    return true;
}

// Coordinate i (0..2) of solve3's solution, with the same operations in the same order: each
// lane of a warp can take one coordinate with one instruction stream (the cofactors of column i
// as P*Q - R*S on operands chosen per lane; -a*b + c*d is that value exactly). 0 when det is 0.
__device__ __forceinline__ double solve3_coord(const real4& e0, const real4& e1, const real4& e2, int i) {
    const double c00 = e1.y * e2.z - e2.y * e1.z;
    const double c01 = -e1.x * e2.z + e2.x * e1.z;
    const double c02 = e1.x * e2.y - e2.x * e1.y;
    const double det = e0.x * c00 + e0.y * c01 + e0.z * c02;
    // column i of the cofactors of rows 1 and 2
    const double p1 = i == 0 ? e2.y : i == 1 ? e0.x : e2.x, q1 = i == 0 ? e0.z : i == 1 ? e2.z : e0.y;
    const double r1 = i == 0 ? e0.y : i == 1 ? e2.x : e0.x, s1 = i == 0 ? e2.z : i == 1 ? e0.z : e2.y;
    const double p2 = i == 0 ? e0.y : i == 1 ? e1.x : e0.x, q2 = i == 0 ? e1.z : i == 1 ? e0.z : e1.y;
    const double r2 = i == 0 ? e1.y : i == 1 ? e0.x : e1.x, s2 = i == 0 ? e0.z : i == 1 ? e1.z : e0.y;
    const double c0i = i == 0 ? c00 : i == 1 ? c01 : c02;
    const double c1i = p1 * q1 - r1 * s1;
    const double c2i = p2 * q2 - r2 * s2;
    if (is0(det)) return 0.0;
    return ddiv(-(e0.w * c0i + e1.w * c1i + e2.w * c2i), det);
}

// solve_2xS (LIB/Vcontacts.cpp:1427-1476).
// rr is the square of the radius as the reference forms it: a single-precision product.
__device__ __noinline__ bool solve2s(const real4& a, const real4& b, double rr, double* p0, double* p1) {
    const double e2x = a.y * b.z - a.z * b.y;
    const double e2y = a.z * b.x - a.x * b.z;
    const double e2z = a.x * b.y - a.y * b.x;
    const double c00 = b.y * e2z - e2y * b.z;
    const double c01 = -b.x * e2z + e2x * b.z;
    const double c02 = b.x * e2y - e2x * b.y;
    const double c10 = -a.y * e2z + e2y * a.z;
    const double c11 = a.x * e2z - e2x * a.z;
    const double c12 = -a.x * e2y + e2x * a.y;
    const double det = e2x * e2x + e2y * e2y + e2z * e2z;
    if (is0(det)) return false;
    const double ax = ddiv(-(a.w * c00 + b.w * c10), det);
    const double ay = ddiv(-(a.w * c01 + b.w * c11), det);
    const double az = ddiv(-(a.w * c02 + b.w * c12), det);
    double t = ddiv(rr - ax * ax - ay * ay - az * az, det);
    if (lt0(t)) return false;
    t = dsqrt(t);
    const double tx = t * e2x, ty = t * e2y, tz = t * e2z;
    p0[0] = ax + tx; p0[1] = ay + ty; p0[2] = az + tz;
    p1[0] = ax - tx; p1[1] = ay - ty; p1[2] = az - tz;
    return true;
}

// The cosine at q of the angle p q r.
__device__ __forceinline__ double cos_pqr(const real4& p, const real4& q, const real4& r) {
    const double ax = p.x - q.x, ay = p.y - q.y, az = p.z - q.z;
    const double bx = r.x - q.x, by = r.y - q.y, bz = r.z - q.z;
    return ddiv(ax * bx + ay * by + az * bz, dsqrt((ax * ax + ay * ay + az * az) * (bx * bx + by * by + bz * bz)));
}

// A cosine's sort key: keys compare as signed integers in the order the values compare, the two
// zeros sharing one; a NaN gets the smallest (key_less is false whenever one is involved).
__device__ __forceinline__ long long cos_key(double c) {
    long long b = bits(c);
    if ((b & LLONG_MAX) > kInfBits) return LLONG_MIN;
    if ((b << 1) == 0) b = 0;
    return b < 0 ? b ^ LLONG_MAX : b;
}
__device__ __forceinline__ bool key_less(long long a, long long b) { return a < b && a != LLONG_MIN; }

// spherical_arc (LIB/Vcontacts.cpp:1518-1557): the cap sector between B and C about the
// contact centre Ao minus a spherical triangle, the reference's own expression.
__device__ __forceinline__ double sph_arc(const real4& ao, const real4& b, const real4& c, double rado) {
    const double cosAOB = ddiv(ao.x * b.x + ao.y * b.y + ao.z * b.z, ao.w * b.w);
    const double cosBOC = ddiv(b.x * c.x + b.y * c.y + b.z * c.z, b.w * c.w);
    // (x / 8 and x * 0.125 are the same correctly rounded value: the multiply is the cheaper)
    const double h = dsqrt((1 + cosBOC) * 0.125);
    const double U = (1 + cosAOB) * h;
    const double V = (1 - cosAOB) * h;
    const double W = dsqrt((1 - cosAOB) * (1 + cosAOB) * (1 - cosBOC) * 0.125);
    const double tS = ddiv(1 - U + V + W + W, 1 + U - V - W - W);
    const double tSB = ddiv(1 - U - V, 1 + U + V);
    const double tSA = ddiv(1 - U + V - W - W, 1 + U - V + W + W);
    double tanprod = 0.0;
    if (gt0(tS * tSA)) tanprod = dsqrt(tSB * tSB * tS * tSA);
    const double px = b.x - ao.x, py = b.y - ao.y, pz = b.z - ao.z;
    const double qx = c.x - ao.x, qy = c.y - ao.y, qz = c.z - ao.z;
    const double cosBAC = ddiv(px * qx + py * qy + pz * qz,
                               dsqrt((px * px + py * py + pz * pz) * (qx * qx + qy * qy + qz * qz)));
    double angBAC;
    if (cosBAC > 1.0) angBAC = 0.0;
    else if (cosBAC < -1.0) angBAC = kPi;
    else angBAC = acos(cosBAC);
    return rado * (angBAC * (rado - ao.w) - 4.0 * rado * datan(dsqrt(tanprod)));
}

// Area of the fan triangle v0 va vb on the sphere of radius rado: L'Huilier-type tangent products
// as the reference writes them (LIB/Vcontacts.cpp:927-940).
__device__ __forceinline__ double fan_triangle(const real4& v0, const real4& va, const real4& vb, double rado) {
    const double cNN1 = ddiv(va.x * vb.x + va.y * vb.y + va.z * vb.z, va.w * vb.w);
    const double cN0a = ddiv(v0.x * va.x + v0.y * va.y + v0.z * va.z, v0.w * va.w);
    const double cN0b = ddiv(v0.x * vb.x + v0.y * vb.y + v0.z * vb.z, v0.w * vb.w);
    const double U = dsqrt((1 + cN0a) * (1 + cNN1) * (1 + cN0b) * 0.125);
    const double V = dsqrt((1 - cN0a) * (1 - cNN1) * (1 + cN0b) * 0.125);
    const double W = dsqrt((1 - cN0a) * (1 + cNN1) * (1 - cN0b) * 0.125);
    const double Xv = dsqrt((1 + cN0a) * (1 - cNN1) * (1 - cN0b) * 0.125);
    const double tS = ddiv(1 - U + V + W + Xv, 1 + U - V - W - Xv);
    const double tSA = ddiv(1 - U - V - W + Xv, 1 + U + V + W - Xv);
    const double tSB = ddiv(1 - U - V + W - Xv, 1 + U + V - W + Xv);
    const double tSC = ddiv(1 - U + V - W - Xv, 1 + U - V + W + Xv);
    const double tanprod = dsqrt(tS * tSA * tSB * tSC);
    return gt0(tanprod) ? 4.0 * rado * rado * datan(dsqrt(tanprod)) : 0.0;
}

__device__ __forceinline__ real4 centre_of(const real4& pl) {
    return make_real4(-pl.x * pl.w, -pl.y * pl.w, -pl.z * pl.w, fabs(pl.w));
}

// Test point i of the faces' inside tests (faces_inside): in double in the first half of sh.u.f.val,
// truncated to single precision in the second (test_point_f).
template <class Sh>
__device__ __forceinline__ float* test_point_f(Vor<Sh>& sh, int i) { return reinterpret_cast<float*>(&sh.u.f.val[Sh::items / 2]) + 3 * i; }
template <class Sh>
__device__ __forceinline__ void put_test_point(Vor<Sh>& sh, int i, double x, double y, double z) {
    double* q = &sh.u.f.val[3 * i];
    q[0] = x;
    q[1] = y;
    q[2] = z;
    float* f = test_point_f(sh, i);
    f[0] = d2f_trunc(x);
    f[1] = d2f_trunc(y);
    f[2] = d2f_trunc(z);
}

template <class Sh>
__device__ __noinline__ bool in_front_exact(const Vor<Sh>& sh, int k, const double* q) {
    return gt0(dot3(sh.pl[k], q[0], q[1], q[2]) + sh.pl[k].w);
}

// test_point (LIB/Vcontacts.cpp:1357-1372) for several faces at once: face X = sh.flist[i], i < nf, keeps its test
// point i when the point lies behind every flagged contact plane other than X; a face with a plane
// in front of its point gets its bit in sh.bad. One plane per lane, decided in single precision
// unless the value is within its error bound (as in `behind`).
template <class Sh>
__device__ __noinline__ void faces_inside(Vor<Sh>& sh, int NC, int nf, int lane) {
    uint32_t bad[kFaceWords] = {0u, 0u, 0u};
    #pragma unroll 1
    for (int c0 = 0; nf > 0 && c0 < NC; c0 += 32) {
        const int cp = c0 + lane;
        const bool on = cp < NC && sh.flag[cp] != 0;
        const real4 P = sh.pl[on ? cp : 0];
        const float Px = d2f_trunc(P.x), Py = d2f_trunc(P.y), Pz = d2f_trunc(P.z), Pw = d2f_trunc(P.w);
        #pragma unroll 1
        for (int i = 0; i < nf; ++i) {
            const int X = sh.flist[i];
            const float* f = test_point_f(sh, i);
            const float x = f[0], y = f[1], z = f[2];
            const float v = fmaf(Px, x, fmaf(Py, y, fmaf(Pz, z, Pw)));
            const float e = 0x1.0p-20f * (fabsf(Px * x) + fabsf(Py * y) + fabsf(Pz * z) + fabsf(Pw));
            bool front = false;
            if (on && cp != X) front = fabsf(v) > e ? v > 0.0f : in_front_exact(sh, cp, &sh.u.f.val[3 * i]);
            if (__any_sync(kFull, front)) {
                const uint32_t b = 1u << (X & 31);
                if (X < 32) bad[0] |= b;
                else if (X < 64) bad[1] |= b;
                else bad[2] |= b;
            }
        }
    }
    if (lane == 0) {
        sh.bad[0] = bad[0];
        sh.bad[1] = bad[1];
        sh.bad[2] = bad[2];
    }
    __syncwarp();
}

// The walk's vertex i.
template <class Sh>
__device__ __forceinline__ real4* walk_vertex(Vor<Sh>& sh, int i) { return i < Sh::verts ? &sh.vx[i] : &sh.u.e.vx[i - Sh::verts]; }
template <class Sh>
__device__ __forceinline__ const real4* walk_vertex(const Vor<Sh>& sh, int i) {
    return i < Sh::verts ? &sh.vx[i] : &sh.u.e.vx[i - Sh::verts];
}

// Coordinate c of the cross product of planes p0's and p1's normals.
template <class Sh>
__device__ __forceinline__ double cross_coord(const Vor<Sh>& sh, int p0, int p1, int c) {
    const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
    return comp(sh.pl[p0], c1) * comp(sh.pl[p1], c2) - comp(sh.pl[p0], c2) * comp(sh.pl[p1], c1);
}

// The same in single precision from the truncated planes: each coordinate within 2^-20 of it (the
// normals are unit vectors, the bounding planes' 1.23 long).
__device__ __forceinline__ float3 cross_f(const float4& a, const float4& b) {
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// The sign of t.(r + v) + t.w in double: whether add_vedge reverses the direction.
template <class Sh>
__device__ __noinline__ bool edge_flip_exact(const Vor<Sh>& sh, int p0, int p1, int tp, double pos, int c, int base) {
    const double q = comp(sh.pl[tp], c) * (pos + cross_coord(sh, p0, p1, c));
    const double q0 = __shfl_sync(kFull, q, base), q1 = __shfl_sync(kFull, q, base + 1), q2 = __shfl_sync(kFull, q, base + 2);
    return gt0(q0 + q1 + q2 + sh.pl[tp].w);
}

// Whether the edge along planes p0 and p1 from the vertex whose coordinate c this lane holds (pos;
// lanes base + 0..2 hold the three) runs against the planes' cross product, so that it points away
// from plane tp (add_vedge, LIB/Vcontacts.cpp:633-660). Decided in single precision where its error
// bound allows (any lane with `active` set and unsure sends the warp to the double form).
template <class Sh>
__device__ __forceinline__ bool edge_flip(const Vor<Sh>& sh, int p0, int p1, int tp, double pos, int c, int base, bool active) {
    const float rf = d2f_trunc(pos);
    const float rx = __shfl_sync(kFull, rf, base), ry = __shfl_sync(kFull, rf, base + 1), rz = __shfl_sync(kFull, rf, base + 2);
    const float3 v = cross_f(sh.plf[p0], sh.plf[p1]);
    const float4 t = sh.plf[tp];
    const float tv = t.x * (rx + v.x) + t.y * (ry + v.y) + t.z * (rz + v.z) + t.w;
    const float err = 1.9073486328125e-06f * (fabsf(t.x) * (fabsf(rx) + 1.5f) + fabsf(t.y) * (fabsf(ry) + 1.5f) +
                                              fabsf(t.z) * (fabsf(rz) + 1.5f) + fabsf(t.w));   // 2^-19
    bool flip = tv > 0.0f;
    if (__any_sync(kFull, active && !(fabsf(tv) > err))) flip = edge_flip_exact(sh, p0, p1, tp, pos, c, base);
    return flip;
}

// Single-precision value of vt = -(P.s + w) / (P.V) and a bound on its distance from the same
// expression evaluated in double. With inputs truncated to float (2^-23 of them), V's coordinates
// within 2^-20, unit normals (the bounding planes' are 1.23 long) and roundings of 2^-24, P.V is
// within 2.1 * 2^-20 (kDenErr: 2.5 * 2^-20) and P.s + w within 2^-20 (1.25 |s|_1 + |w|), es being
// its first part; with |P.V| above 16 kDenErr the quotient's denominator is known to a sixteenth, and
// the reciprocal and the two products round by less than 4 units of |vt|. *ok is false below that
// (the double test also skips P.V == 0 exactly).
constexpr float kDenErr = 2.5f * 0x1.0p-20f;
__device__ __forceinline__ float start_err(float sx, float sy, float sz) {
    return 1.25f * 0x1.0p-20f * (fabsf(sx) + fabsf(sy) + fabsf(sz));
}
__device__ __forceinline__ float vt_pretest(const float4& P, float sx, float sy, float sz, float Vx,
                                            float Vy, float Vz, float es, float* err, bool* ok) {
    const float den = fmaf(P.x, Vx, fmaf(P.y, Vy, P.z * Vz));
    const float num = fmaf(P.x, sx, fmaf(P.y, sy, fmaf(P.z, sz, P.w)));
    const float rd = rcp_approx(den);
    const float vt = -num * rd, av = fabsf(vt);
    *ok = fabsf(den) > 16.0f * kDenErr;
    *err = fmaf(av, 4.8e-7f, fmaf(av, kDenErr, fmaf(fabsf(P.w), 0x1.0p-20f, es)) * (1.08f * fabsf(rd)));
    return vt;
}

// A step's result: the closing plane (-1 if none) and the coordinate of the new vertex this lane
// holds (coordinate min(lane & 3, 2)).
struct WalkStep {
    double pos;
    int pc;
};

// The candidate vt of plane k for the edge from s along V: its bit pattern when positive and below
// cur, else cur.
template <class Sh>
__device__ __forceinline__ bool step_key(const Vor<Sh>& sh, int k, const double* s, const double* V, long long cur,
                                         long long* key) {
    const real4 P = sh.pl[k];
    const double den = P.x * V[0] + P.y * V[1] + P.z * V[2];
    if (is0(den)) return false;
    const long long b = bits(ddiv(-(P.x * s[0] + P.y * s[1] + P.z * s[2] + P.w), den));
    if (!(b > 0 && b < cur)) return false;
    *key = b;
    return true;
}

// The vertex that ends edge e (LIB/Vcontacts.cpp:283-330), in full precision: the plane with
// the smallest positive vt along the edge (planes spread over the lanes) and, when that point
// lies outside the sphere, the bounding planes too. The result is uniform across the warp.
template <class Sh>
__device__ __noinline__ WalkStep walk_step_exact(const Vor<Sh>& sh, int NC, int e, double rr, int lane) {
    const uchar4 ep = sh.u.e.ep[e];
    const double* s = reinterpret_cast<const double*>(walk_vertex(sh, sh.u.e.es[e].x));
    const int pA = ep.x, pB = ep.y, oldC = ep.z;
    const int c = min(lane & 3, 2), base = lane & ~3;
    double Vc = cross_coord(sh, pA, pB, c);
    if (sh.u.e.flip[e]) Vc = -Vc;
    const double V[3] = {__shfl_sync(kFull, Vc, base), __shfl_sync(kFull, Vc, base + 1), __shfl_sync(kFull, Vc, base + 2)};
    long long key = bits(9.9e9);
    int pC = INT_MAX;
    #pragma unroll 1
    for (int k = lane; k < NC; k += 32) {
        if (k == pA || k == pB || k == oldC) continue;
        if (step_key(sh, k, s, V, key, &key)) pC = k;
    }
    warp_argmin(key, pC);
    const double sc = s[c];
    WalkStep r;
    r.pos = sc + __longlong_as_double(key) * Vc;
    const double q = r.pos * r.pos;
    const double q0 = __shfl_sync(kFull, q, base), q1 = __shfl_sync(kFull, q, base + 1), q2 = __shfl_sync(kFull, q, base + 2);
    if (lt_nn(rr, q0 + q1 + q2)) {
        const int k = NC + lane;
        if (lane < 4 && k != pA && k != pB && k != oldC && step_key(sh, k, s, V, key, &key)) pC = k;
        warp_argmin(key, pC);
        r.pos = sc + __longlong_as_double(key) * Vc;
    }
    r.pc = pC == INT_MAX ? -1 : pC;
    return r;
}

// The hull walk steps several open edges at once: a step's result depends only on its edge (start
// vertex, direction, planes), all fixed when the edge was made, and the reference takes every edge
// that is open now, in index order, before any edge the steps append (those get higher indices).
// So the first kWalkGroups open edges are stepped together, one group of kWalkLanes lanes each, and
// their results are booked one after another in index order, skipping an edge an earlier one closed.
constexpr int kWalkGroups = 4;
constexpr int kWalkLanes = 32 / kWalkGroups;

// One step for the group's edge e (e < 0: the group idles; every lane still joins the shuffles).
// gmask: the group's lanes. *unsure: the single-precision pre-tests did not decide it (redo with
// walk_step_exact). In a group of eight lanes the first half takes the coordinates of P.V, the
// second those of P.s; both halves end with the new vertex's coordinates.
template <class Sh>
__device__ __forceinline__ WalkStep walk_step_group(const Vor<Sh>& sh, int NC, int e, float rrf, int lane, unsigned gmask,
                                                    bool* unsure_out) {
    const bool has = e >= 0;
    const int sub = lane & (kWalkLanes - 1), c = min(lane & 3, 2), base = lane & ~3, gbase = lane & ~(kWalkLanes - 1);
    uchar4 ep = make_uchar4(kNone, kNone, kNone, kNone);
    const double* s = reinterpret_cast<const double*>(&sh.vx[0]);
    bool flip = false;
    if (has) {
        ep = sh.u.e.ep[e];
        flip = sh.u.e.flip[e] != 0;
        s = reinterpret_cast<const double*>(walk_vertex(sh, sh.u.e.es[e].x));
    }
    const int pA = ep.x, pB = ep.y, oldC = ep.z;
    // this lane's coordinate of the direction in double (used after the pre-tests, which hide it)
    const double sc = s[c];
    double Vc = cross_coord(sh, has ? pA : 0, has ? pB : 0, c);
    if (flip) Vc = -Vc;
    // planes pre-tested in single precision; when the winner is surely positive and every other
    // plane surely not positive or surely farther, only the winner's vt is evaluated in double
    const float3 Vf = cross_f(sh.plf[has ? pA : 0], sh.plf[has ? pB : 0]);
    const float Vx = flip ? -Vf.x : Vf.x, Vy = flip ? -Vf.y : Vf.y, Vz = flip ? -Vf.z : Vf.z;
    const float sf = d2f_trunc(sc);
    const float sx = __shfl_sync(kFull, sf, base), sy = __shfl_sync(kFull, sf, base + 1), sz = __shfl_sync(kFull, sf, base + 2);
    const float es = start_err(sx, sy, sz);
    float best = 9.9e9f, beste = 0.0f;
    int bi = INT_MAX;
    // and the two smallest lower bounds (vt - err) over the planes whose vt may be positive: every
    // plane but the winner must be surely not positive or surely farther
    float lo1 = 3.0e38f, lo2 = 3.0e38f;
    int lo1i = INT_MAX;
    bool unsure = false;
    if (has) {
        #pragma unroll 1
        for (int k = sub; k < NC; k += kWalkLanes) {
            if (k == pA || k == pB || k == oldC) continue;
            float er;
            bool ok;
            const float vt = vt_pretest(sh.plf[k], sx, sy, sz, Vx, Vy, Vz, es, &er, &ok);
            if (!ok) {
                unsure = true;
                continue;
            }
            if (vt > 0.0f && vt < best) { best = vt; beste = er; bi = k; }
            if (vt + er > 0.0f) {
                const float lo = vt - er;
                if (lo < lo1) { lo2 = lo1; lo1 = lo; lo1i = k; }
                else if (lo < lo2) lo2 = lo;
            }
        }
    }
#pragma unroll
    for (int o = kWalkLanes / 2; o > 0; o >>= 1) {
        const float b2 = __shfl_xor_sync(kFull, best, o);
        const float e2 = __shfl_xor_sync(kFull, beste, o);
        const int i2 = __shfl_xor_sync(kFull, bi, o);
        if (b2 < best || (b2 == best && i2 < bi)) { best = b2; beste = e2; bi = i2; }
    }
    const bool won = bi != INT_MAX;
    if (won && !(best - beste > 0.0f)) unsure = true;
    const float mylo = lo1i == bi ? lo2 : lo1;
    if (mylo < 3.0e38f && !(won && mylo > best + beste)) unsure = true;
    if (has && !won) unsure = true;   // (no plane: the bounding planes decide)
    // the winner's vt and the vertex, one coordinate per lane
    const real4& P = sh.pl[won ? bi : 0];
    const double m = comp(P, c) * (sub < 4 ? Vc : sc);
    const double m0 = __shfl_sync(kFull, m, base), m1 = __shfl_sync(kFull, m, base + 1), m2 = __shfl_sync(kFull, m, base + 2);
    const double t = m0 + m1 + m2;
    double den = __shfl_sync(kFull, t, gbase);
    const double num = __shfl_sync(kFull, t + P.w, gbase + 4);
    if (!won) den = 1.0;
    const double vt = ddiv(-num, den);
    WalkStep r;
    r.pos = sc + vt * Vc;
    // perhaps outside the sphere (the reference then tries the bounding planes too): those, 10 A
    // out, are most of the time surely farther
    const float vtf = d2f_trunc(vt);
    const float ax = vtf * Vx, ay = vtf * Vy, az = vtf * Vz, av = 2e-6f * fabsf(vtf);
    const float fx = fabsf(sx + ax) + 2e-6f * (fabsf(sx) + fabsf(ax)) + av, fy = fabsf(sy + ay) + 2e-6f * (fabsf(sy) + fabsf(ay)) + av,
                fz = fabsf(sz + az) + 2e-6f * (fabsf(sz) + fabsf(az)) + av;
    bool need = false;
    if (has && won && sub < 4 && !(fx * fx + fy * fy + fz * fz < rrf * 0.99999f)) {
        const int k = NC + sub;
        if (k != pA && k != pB && k != oldC) {
            float er;
            bool ok;
            const float bt = vt_pretest(sh.plf[k], sx, sy, sz, Vx, Vy, Vz, es, &er, &ok);
            need = !(ok && (bt + er <= 0.0f || bt - er > vtf * 1.0000005f));   // (vtf: truncated, 2^-23 of it)
        }
    }
    *unsure_out = (__ballot_sync(kFull, unsure || need) & gmask) != 0u;
    r.pc = won ? bi : -1;
    return r;
}

// The face that the arc between points cur and nxt of engulfed face X is credited to
// (LIB/Vcontacts.cpp:971-1000): the plane the two points share besides X, when it is neither the
// sphere nor an engulfing plane; -1 when the reference moves on without crediting anything.
template <class Sh>
__device__ __forceinline__ int engulf_comm(const Vor<Sh>& sh, int NC, int X, int cur, int nxt) {
    const uchar4 qc = sh.vp[cur], qn = sh.vp[nxt];
    int pa1, pa2;
    if (qc.x == X) { pa1 = qc.y; pa2 = qc.z; }
    else { pa1 = qc.x; pa2 = (qc.y == X) ? qc.z : qc.y; }
    int comm;
    if (pa1 == qn.x || pa1 == qn.y || pa1 == qn.z) comm = pa1;
    else if (pa2 == qn.x || pa2 == qn.y || pa2 == qn.z) comm = pa2;
    else return -1;
    return (comm != kNone && !(comm < NC && (sh.flag[comm] & kEngulf))) ? comm : -1;
}

// Face history of one pose (reference face order): order_faces leaves each contact's point list
// in ptorder[X].pt[] (LIB/Vcontacts.cpp:726-831), a workspace that outlives the atom, and reads
// ptorder[X].pt[numpts] — a slot past the face's own list — when no point shares the first
// point's second plane (:800-812). That slot holds what an earlier atom of the pose left there
// (zero at the start of the pose). The history keeps those lists per contact index X, rows of
// kHistPts entries, followed by the pre-extra contents of the vertex slots the antipodal points
// take (the reference appends them one face at a time, so a face's read of a later face's slot
// still sees the old vertex there).
constexpr int kHistPts = 64;
constexpr int kHistBytes = kMaxCand * kHistPts;
constexpr size_t kHistStride = kHistBytes + kMaxCand * (sizeof(real4) + sizeof(uchar4));
static_assert(kHistBytes % 32 == 0 && kHistStride % 32 == 0, "history rows keep 32-byte alignment");

__device__ __forceinline__ real4* hist_vx(uint8_t* h) { return reinterpret_cast<real4*>(h + kHistBytes); }
__device__ __forceinline__ uchar4* hist_vp(uint8_t* h) {
    return reinterpret_cast<uchar4*>(h + kHistBytes + kMaxCand * sizeof(real4));
}

// The smallest of the lanes' values (not negative), with the lowest index among equal ones and its
// upper bound; false when another entry's lower bound (lo1 / lo2: each lane's two smallest, lo1i the
// first's index) does not lie above that, or a lane is undecided.
__device__ __forceinline__ bool certain_min(float best, float hi, int bi, float lo1, float lo2, int lo1i, bool undecided, int* at) {
    const unsigned b = __float_as_uint(best), m = __reduce_min_sync(kFull, b);
    const int i = __reduce_min_sync(kFull, b == m ? bi : INT_MAX);
    const unsigned own = __ballot_sync(kFull, b == m && bi == i);
    const float h = __shfl_sync(kFull, hi, __ffs(own) - 1);
    *at = i;
    return !__any_sync(kFull, undecided || !((lo1i == i ? lo2 : lo1) > h)) && i != INT_MAX;
}

// get_firstvert's search (see first_planes_exact) decided in single precision, false when an error
// bound does not allow it (3 % of the searches). The search starts a fifth of the atoms, so nearly
// every step of a group waited for one: 25,000 - 38,000 cycles in double precision of some 230,000.
//  Two planes' line lies at d^2 = (wa^2 + wb^2 - 2 wa wb cos) / sin^2 of unit
// normals with cosine cos; inputs truncated by 2^-23 of them leave cos within 6e-7, so the numerator
// within 3e-6 (|wa| + |wb|)^2 and the denominator within 1.5e-6.
template <class Sh>
__device__ __noinline__ bool first_planes_fast(const Vor<Sh>& sh, int NC, int lane, int* pA, int* pB, int* pC) {
    constexpr float kBig = 3.0e38f;
    long long bv = bits(9.9e9);
    int iA = INT_MAX;
    #pragma unroll 1
    for (int c = lane; c < NC; c += 32) {
        const long long d = bits(fabs(sh.pl[c].w));
        if (d < bv) { bv = d; iA = c; }
    }
    warp_argmin(bv, iA);
    if (iA == INT_MAX) return false;
    const float4 A = sh.plf[iA];
    float best = kBig, hi = kBig, lo1 = kBig, lo2 = kBig;
    int bi = INT_MAX, lo1i = INT_MAX;
    bool undecided = false;
    #pragma unroll 1
    for (int c = lane; c < NC + 4; c += 32) {
        if (c == iA) continue;
        float4 C = sh.plf[c];
        if (c >= NC) {   // the bounding planes' normals are 1.224683 long
            C.x *= 0.816538f; C.y *= 0.816538f; C.z *= 0.816538f; C.w *= 0.816538f;
        }
        const float cs = A.x * C.x + A.y * C.y + A.z * C.z, s2 = 1.0f - cs * cs;
        const float w2 = (fabsf(A.w) + fabsf(C.w)) * (fabsf(A.w) + fabsf(C.w));
        const float n = fmaxf(A.w * A.w + C.w * C.w - 2.0f * A.w * C.w * cs, 0.0f), en = 3e-6f * w2;
        if (!(s2 > 1e-4f)) {
            undecided = true;
            continue;
        }
        const float d2 = n / s2, h = (n + en) / (s2 - 1.5e-6f) * 1.000001f, l = (n - en) / (s2 + 1.5e-6f) * 0.999999f - 1e-12f;
        if (d2 < best) { best = d2; hi = h; bi = c; }
        if (l < lo1) { lo2 = lo1; lo1 = l; lo1i = c; }
        else if (l < lo2) lo2 = l;
    }
    int iB;
    if (!certain_min(best, hi, bi, lo1, lo2, lo1i, undecided, &iB)) return false;
    // the point of the line closest to the centre, and the plane the line meets first
    float4 B = sh.plf[iB];
    if (iB >= NC) {
        B.x *= 0.816538f; B.y *= 0.816538f; B.z *= 0.816538f; B.w *= 0.816538f;
    }
    const float cs = A.x * B.x + A.y * B.y + A.z * B.z, is2 = 1.0f / (1.0f - cs * cs);
    const float ka = -(A.w - B.w * cs) * is2, kb = -(B.w - A.w * cs) * is2;
    const float px = ka * A.x + kb * B.x, py = ka * A.y + kb * B.y, pz = ka * A.z + kb * B.z;
    const float es = start_err(px, py, pz) + 8e-6f * (fabsf(A.w) + fabsf(B.w)) * is2 * is2;
    const float3 v = cross_f(A, B);
    best = hi = lo1 = lo2 = kBig;
    bi = lo1i = INT_MAX;
    #pragma unroll 1
    for (int c = lane; c < NC + 4; c += 32) {
        if (c == iA || c == iB) continue;
        const float4 C = sh.plf[c];
        float er;
        bool ok;
        const float vt = fabsf(vt_pretest(C, px, py, pz, v.x, v.y, v.z, es, &er, &ok));
        float l = vt - er;
        if (ok) {
            if (vt < best) { best = vt; hi = vt + er; bi = c; }
        } else {
            // nearly parallel to the line: beyond |numerator| over the largest such denominator
            const float num = fabsf(fmaf(C.x, px, fmaf(C.y, py, fmaf(C.z, pz, C.w))));
            const float left = num - fmaf(fabsf(C.w), 0x1.0p-20f, es);
            if (!(left > 0.0f)) undecided = true;
            l = left * (0.9f / (17.0f * kDenErr));
        }
        if (l < lo1) { lo2 = lo1; lo1 = l; lo1i = c; }
        else if (l < lo2) lo2 = l;
    }
    int iC;
    if (!certain_min(best, hi, bi, lo1, lo2, lo1i, undecided, &iC)) return false;
    *pA = iA;
    *pB = iB;
    *pC = iC;
    return true;
}

// get_firstvert's search from the plane closest to the centre (LIB/Vcontacts.cpp:498-592): the
// first vertex's planes, false when a step finds none.
template <class Sh>
__device__ __noinline__ bool first_planes_exact(const Vor<Sh>& sh, int NC, int lane, int* pA, int* pB, int* pC) {
    long long bv = bits(9.9e9);
    int bi = INT_MAX;
    #pragma unroll 1
    for (int c = lane; c < NC; c += 32) {
        const long long d = bits(fabs(sh.pl[c].w));
        if (d < bv) { bv = d; bi = c; }
    }
    warp_argmin(bv, bi);
    const int pA0 = bi;
    if (pA0 == INT_MAX) return false;
    const real4 A = sh.pl[pA0];
    bv = bits(9.9e9);
    bi = INT_MAX;
    #pragma unroll 1
    for (int c = lane; c < NC + 4; c += 32) {
        if (c == pA0) continue;
        const real4 C = sh.pl[c];
        const real4 v = make_real4(A.y * C.z - A.z * C.y, A.z * C.x - A.x * C.z, A.x * C.y - A.y * C.x, 0.0);
        double t[3];
        if (solve3(A, C, v, t)) {
            const long long d = bits(fabs(dsqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2])));
            if (d < bv) { bv = d; bi = c; }
        }
    }
    warp_argmin(bv, bi);
    const int pB0 = bi;
    if (pB0 == INT_MAX) return false;
    const real4 B = sh.pl[pB0];
    const real4 v = make_real4(A.y * B.z - A.z * B.y, A.z * B.x - A.x * B.z, A.x * B.y - A.y * B.x, 0.0);
    double ptA[3];
    solve3(A, B, v, ptA);
    bv = bits(9.9e9);
    bi = INT_MAX;
    #pragma unroll 1
    for (int c = lane; c < NC + 4; c += 32) {
        if (c == pA0 || c == pB0) continue;
        const real4 C = sh.pl[c];
        const double den = C.x * v.x + C.y * v.y + C.z * v.z;
        if (!is0(den)) {
            const long long vt = bits(fabs(ddiv(-(C.x * ptA[0] + C.y * ptA[1] + C.z * ptA[2] + C.w), den)));
            if (vt < bv) { bv = vt; bi = c; }
        }
    }
    warp_argmin(bv, bi);
    if (bi == INT_MAX) return false;
    *pA = pA0;
    *pB = pB0;
    *pC = bi;
    return true;
}

// The hull walk's progress: vertices and edges so far, and the first edge that may be open.
struct Walk {
    int vn, edges, start;
};

// The first vertex and its three edges.
template <class Sh>
__device__ __forceinline__ void walk_start(Vor<Sh>& sh, int lane, int pA0, int pB0, int pC0, Walk& walk) {
    const int c = min(lane & 3, 2), base = lane & ~3;
    {
        // the vertex's coordinates one per lane, then its three edges at once, four lanes each
        const double tc = solve3_coord(sh.pl[pA0], sh.pl[pB0], sh.pl[pC0], c);
        const int g = min(lane >> 2, 2);
        const int p0 = g == 0 ? pA0 : g == 1 ? pB0 : pC0;
        const int p1 = g == 0 ? pB0 : g == 1 ? pC0 : pA0;
        const int tp = g == 0 ? pC0 : g == 1 ? pA0 : pB0;
        const bool flip = edge_flip(sh, p0, p1, tp, tc, c, base, true);
        if (lane < 3) reinterpret_cast<double*>(&sh.vx[0])[lane] = tc;   // (its distance comes with the others')
        if (lane < 12 && (lane & 3) == 3) {
            sh.u.e.ep[g] = make_uchar4((uint8_t)p0, (uint8_t)p1, (uint8_t)tp, kNone);
            sh.u.e.es[g] = make_uchar2(0, kNone);
            sh.u.e.flip[g] = flip;
            sh.flag[p0] |= kOnHull;
        }
        if (lane == 0) sh.vp[0] = make_uchar4((uint8_t)pA0, (uint8_t)pB0, (uint8_t)pC0, 0);
    }
    __syncwarp();
    walk = Walk{1, 3, 0};
}

// The hull walk (LIB/Vcontacts.cpp:262-410), the open edges stepped kWalkGroups at a time, at most
// kWalkBudget times: kAtomOk when no edge is open, kAtomWalking when there are more. Vertices in
// walk_vertex / sh.vp, edges in sh.u.e.
template <class Sh>
__device__ __forceinline__ int hull_walk(Vor<Sh>& sh, int NC, double rr, int lane, Walk& walk) {
    const int c = min(lane & 3, 2), base = lane & ~3;
    int edgenum = walk.edges, startedge = walk.start, vn = walk.vn;
    const int grp = lane / kWalkLanes;
    const unsigned gmask = ((1u << kWalkLanes) - 1u) << (lane & ~(kWalkLanes - 1));
    const bool second = (lane & 4) != 0;   // this lane's half takes the step's second new edge
    const float rrf = d2f_trunc(rr);
    int left = kWalkBudget;
    #pragma unroll 1
    for (;;) {
        // the first kWalkGroups open edges, in index order (one byte each)
        unsigned batch = 0u;
        int nb = 0;
        #pragma unroll 1
        for (int e0 = startedge & ~31; e0 < edgenum && nb < kWalkGroups; e0 += 32) {
            const int f = e0 + lane;
            unsigned m = __ballot_sync(kFull, f < edgenum && sh.u.e.es[f].y == kNone);
            while (m && nb < kWalkGroups) {
                batch |= (unsigned)(e0 + __ffs(m) - 1) << (8 * nb);
                m &= m - 1;
                ++nb;
            }
        }
        if (nb == 0) break;
        startedge = batch & 0xffu;
        if (left-- == 0) {
            walk = Walk{vn, edgenum, startedge};
            return kAtomWalking;
        }
        bool unsure_g;
        const WalkStep gs = walk_step_group(sh, NC, grp < nb ? (int)((batch >> (8 * grp)) & 0xffu) : -1, rrf, lane, gmask, &unsure_g);
        const int mine = (gs.pc << 1) | (int)unsure_g;
        // book the steps in index order; a new vertex's coordinates are stored by its group after
        // the batch, and so are the directions of its (at most two) new edges: slot, planes
        double pos = gs.pos;
        int my_vn = -1, pe = -1, p0e = 0, pce = 0, tpe = 0;
        #pragma unroll 1
        for (int g = 0; g < nb; ++g) {
            const int e = (batch >> (8 * g)) & 0xffu;
            const int pu = __shfl_sync(kFull, mine, g * kWalkLanes);
            int pC = pu >> 1;   // (an arithmetic shift keeps -1)
            if (sh.u.e.es[e].y != kNone) continue;   // closed by an earlier edge of the batch
            if (pu & 1) {
                const WalkStep w = walk_step_exact(sh, NC, e, rr, lane);
                if (grp == g) pos = w.pos;
                pC = w.pc;
            }
            if (pC < 0) return kAtomHullFail;
            if (vn >= kMaxVerts - 1) return kAtomCapacity;
            const uchar4 ep = sh.u.e.ep[e];
            const int pA = ep.x, pB = ep.y;
            // edges (pA, pC) and (pB, pC): the first match after this edge, else a new edge
            int mAC = INT_MAX, mBC = INT_MAX;
            #pragma unroll 1
            for (int e0 = e + 1; e0 < edgenum; e0 += 32) {
                const int f = e0 + lane;
                bool ac = false, bc = false;
                if (f < edgenum) {
                    const uchar4 q = sh.u.e.ep[f];
                    ac = (q.x == pA && q.y == pC) || (q.x == pC && q.y == pA);
                    bc = (q.x == pB && q.y == pC) || (q.x == pC && q.y == pB);
                }
                const unsigned ma = __ballot_sync(kFull, ac), mb = __ballot_sync(kFull, bc);
                if (ma && mAC == INT_MAX) mAC = e0 + __ffs(ma) - 1;
                if (mb && mBC == INT_MAX) mBC = e0 + __ffs(mb) - 1;
                if (mAC != INT_MAX && mBC != INT_MAX) break;
            }
            __syncwarp();
            // a walk that keeps opening edges past the reference's 200-edge check ends here: as a hull
            // failure when the reference's check fails it at this step, else over capacity
            const int n_new = (mAC == INT_MAX) + (mBC == INT_MAX);
            if (edgenum + n_new > kMaxEdges + 2) return mBC == INT_MAX ? kAtomHullFail : kAtomCapacity;
            const int eAC = mAC != INT_MAX ? mAC : edgenum;
            const int eBC = mBC != INT_MAX ? mBC : edgenum + (mAC == INT_MAX ? 1 : 0);
            if (lane == 0) {
                sh.vp[vn] = make_uchar4((uint8_t)pA, (uint8_t)pB, (uint8_t)pC, 0);
                sh.u.e.es[e].y = (uint8_t)vn;
                sh.u.e.ep[e].w = (uint8_t)pC;
                sh.flag[pC] |= kOnHull;
            }
            if (lane < 2) {
                const bool match = lane == 0 ? mAC != INT_MAX : mBC != INT_MAX;
                const int ee = lane == 0 ? eAC : eBC;
                const int p0 = lane == 0 ? pA : pB, tp = lane == 0 ? pB : pA;
                if (match) {
                    sh.u.e.es[ee].y = (uint8_t)vn;
                    sh.u.e.ep[ee].w = (uint8_t)tp;
                } else {
                    sh.u.e.ep[ee] = make_uchar4((uint8_t)p0, (uint8_t)pC, (uint8_t)tp, kNone);
                    sh.u.e.es[ee] = make_uchar2((uint8_t)vn, kNone);
                }
            }
            if (grp == g) {
                my_vn = vn;
                pe = second ? (mBC == INT_MAX ? eBC : -1) : (mAC == INT_MAX ? eAC : -1);
                p0e = second ? pB : pA;
                tpe = second ? pA : pB;
                pce = pC;
            }
            edgenum += n_new;
            if (mBC == INT_MAX && edgenum >= kMaxEdges) return kAtomHullFail;
            ++vn;
            __syncwarp();
        }
        // the new vertices, and the sense of the new edges, away from their third plane
        const bool flip = edge_flip(sh, p0e, pce, tpe, pos, c, base, pe >= 0);
        if ((lane & 3) < 3 && my_vn >= 0 && !second) reinterpret_cast<double*>(walk_vertex(sh, my_vn))[c] = pos;
        if ((lane & 3) == 3 && pe >= 0) sh.u.e.flip[pe] = flip;
        __syncwarp();
    }
    walk = Walk{vn, edgenum, startedge};
    return kAtomOk;
}

// Whether point x lies behind plane k (a negative value of the plane's equation), decided in single
// precision unless the value is within its error bound (inputs truncated by 2^-23 of them, sums
// rounded by 2^-24: 2^-20 of the sum of absolute terms covers both).
template <class Sh>
__device__ __noinline__ bool behind_exact(const Vor<Sh>& sh, int k, const double* x) {
    return lt0(dot3(sh.pl[k], x[0], x[1], x[2]) + sh.pl[k].w);
}
template <class Sh>
__device__ __forceinline__ bool behind(const Vor<Sh>& sh, int k, const double* x) {
    const float4 P = sh.plf[k];
    const float fx = d2f_trunc(x[0]), fy = d2f_trunc(x[1]), fz = d2f_trunc(x[2]);
    const float v = fmaf(P.x, fx, fmaf(P.y, fy, fmaf(P.z, fz, P.w)));
    const float e = 0x1.0p-20f * (fabsf(P.x * fx) + fabsf(P.y * fy) + fabsf(P.z * fz) + fabsf(P.w));
    return fabsf(v) > e ? v < 0.0f : behind_exact(sh, k, x);
}

// Arc points where edges leave the sphere (LIB/Vcontacts.cpp:418-462), then the vertices inside it,
// in order; *nv_out their count.
template <class Sh>
__device__ __forceinline__ int arc_points(Vor<Sh>& sh, double rado, double rr, int lane, int vn, int edgenum, int* nv_out) {
    // vertex distances to the centre, all at once
    #pragma unroll 1
    for (int vi = lane; vi < vn; vi += 32) {
        real4& X = *walk_vertex(sh, vi);
        X.w = dsqrt(X.x * X.x + X.y * X.y + X.z * X.z);
    }
    __syncwarp();
    // the edges with an end outside the sphere listed in order, then their sphere intersections a
    // warp at a time
    int n_out = 0;
    #pragma unroll 1
    for (int e0 = 0; e0 < edgenum; e0 += 32) {
        const int e = e0 + lane;
        bool out = false;
        if (e < edgenum) {
            const uchar2 se = sh.u.e.es[e];
            out = lt_nn(rado, walk_vertex(sh, se.x)->w) || lt_nn(rado, walk_vertex(sh, se.y)->w);
        }
        const unsigned m = __ballot_sync(kFull, out);
        if (out) sh.elist[n_out + __popc(m & lanemask_lt())] = (uint8_t)e;
        n_out += __popc(m);
    }
    __syncwarp();
    #pragma unroll 1
    for (int k0 = 0; k0 < n_out; k0 += 32) {
        const int k = k0 + lane;
        int cnt = 0;
        double a0[3], a1[3];
        bool k0v = false, k1v = false;
        uchar4 q = make_uchar4(0, 0, 0, 0);
        if (k < n_out) {
            q = sh.u.e.ep[sh.elist[k]];
            if (solve2s(sh.pl[q.x], sh.pl[q.y], rr, a0, a1)) {
                k0v = behind(sh, q.z, a0) && behind(sh, q.w, a0);
                k1v = behind(sh, q.z, a1) && behind(sh, q.w, a1);
                cnt = (int)k0v + (int)k1v;
            }
        }
        int tot;
        const int off = warp_excl_scan(cnt, lane, &tot);
        if (vn + tot > kMaxVerts - 1) return kAtomCapacity;
        int w = vn + off;
        if (k0v) {
            *walk_vertex(sh, w) = make_real4(a0[0], a0[1], a0[2], rado);
            sh.vp[w] = make_uchar4(q.x, q.y, kNone, 0);
            ++w;
        }
        if (k1v) {
            *walk_vertex(sh, w) = make_real4(a1[0], a1[1], a1[2], rado);
            sh.vp[w] = make_uchar4(q.x, q.y, kNone, 0);
        }
        vn += tot;
        __syncwarp();
    }
    int nv = 0;
    #pragma unroll 1
    for (int v0 = 0; v0 < vn; v0 += 32) {
        const int vi = v0 + lane;
        real4 X = make_real4(0, 0, 0, 0);
        uchar4 P = make_uchar4(0, 0, 0, 0);
        bool keep = false;
        if (vi < vn) {
            X = *walk_vertex(sh, vi);
            P = sh.vp[vi];
            keep = le_nn(X.w, rado);
        }
        const unsigned m = __ballot_sync(kFull, keep);
        __syncwarp();
        if (keep) {
            const int w = nv + __popc(m & lanemask_lt());
            if (w < Sh::verts) sh.vx[w] = X;
            sh.vp[w] = P;
        }
        nv += __popc(m);
        __syncwarp();
    }
    *nv_out = nv;
    return nv > Sh::verts - 1 ? Sh::over : kAtomOk;
}

// The first set bit at or after bit `from` of the vertex mask a & b, or -1.
template <class Sh>
__device__ __forceinline__ int first_vertex(const uint32_t* a, const uint32_t* b, int from) {
    #pragma unroll 1
    for (int w = from >> 5; w < Sh::vwords; ++w) {
        uint32_t m = a[w] & b[w];
        if (w == from >> 5) m &= 0xffffffffu << (from & 31);
        if (m) return 32 * w + __ffs(m) - 1;
    }
    return -1;
}

// Faces (order_faces, LIB/Vcontacts.cpp:699-831): points per plane in vertex order, plus an
// antipodal arc point, ordered around the face. The edge arrays are dead from here on; their
// storage holds the face lists. Sets sh.foff / fnp / pt, sh.toff (the triangles before each face:
// two fewer than its points) and sh.nt.
template <class Sh>
__device__ __forceinline__ int order_faces(Vor<Sh>& sh, int NC, int NV, double rado, int lane, uint8_t* hist, int& miss,
                                           int& lost) {
    constexpr int NW = Sh::vwords;
    // per plane (contacts and bounding planes), its vertices as a bit mask
    #pragma unroll 1
    for (int k = lane; k < (NC + 4) * NW; k += 32) sh.vmask[k] = 0u;
    __syncwarp();
    uint32_t arcm[NW], regm[NW];   // vertices on the sphere; vertices of three contact planes
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        bool arc = false, reg = false;
        const int vi = 32 * w + lane;
        if (vi < NV) {
            const uchar4 P = sh.vp[vi];
            arc = P.z == kNone;
            reg = P.x < NC && P.y < NC && P.z < NC;
            const uint32_t b = 1u << lane;
            if (P.x < NC + 4) atomicOr(&sh.vmask[P.x * NW + w], b);
            if (P.y < NC + 4) atomicOr(&sh.vmask[P.y * NW + w], b);
            if (P.z < NC + 4) atomicOr(&sh.vmask[P.z * NW + w], b);
        }
        arcm[w] = __ballot_sync(kFull, arc);
        regm[w] = __ballot_sync(kFull, reg);
    }
    __syncwarp();
    // the faces' point lists and, for a face of more than two points, the antipode of its first
    // sphere point, which joins the face when it lies behind every other plane (test_point)
    int tot_pts = 0, nf = 0;
    #pragma unroll 1
    for (int x0 = 0; x0 < NC; x0 += 32) {
        const int X = x0 + lane;
        int cnt = 0;
        const bool face = X < NC && sh.flag[X] != 0;
        const uint32_t* vm = &sh.vmask[(X < NC ? X : 0) * NW];
        if (face) {
#pragma unroll
            for (int w = 0; w < NW; ++w) cnt += __popc(vm[w]);
        }
        int t;
        const int off = tot_pts + warp_excl_scan(cnt + (cnt > 2 ? 1 : 0), lane, &t);
        tot_pts += t;
        if (tot_pts > Sh::pts) return Sh::over;
        int first_arc = -1, seed = -1;
        if (X < NC) {
            sh.foff[X] = (uint16_t)off;
            sh.fnp[X] = (uint8_t)min(cnt, 255);
            if (face) {
                int k = off;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    uint32_t m = vm[w];
                    if (first_arc < 0 && (m & arcm[w])) first_arc = 32 * w + __ffs(m & arcm[w]) - 1;
                    if (seed < 0 && (m & regm[w])) seed = 32 * w + __ffs(m & regm[w]) - 1;
                    #pragma unroll 1
                    for (; m; m &= m - 1) sh.u.f.pt[k++] = (uint8_t)(32 * w + __ffs(m) - 1);
                }
            }
            sh.fseed[X] = (uint8_t)seed;   // (-1: kNone)
        }
        const bool cand = face && cnt > 2 && first_arc >= 0;
        const unsigned m = __ballot_sync(kFull, cand);
        if (3 * (nf + __popc(m)) > Sh::items / 2) return Sh::over;
        if (lane == 0) sh.cmask[x0 >> 5] = m;
        if (cand) {
            const int fi = nf + __popc(m & lanemask_lt());
            sh.flist[fi] = (uint8_t)X;
            const real4 cp = centre_of(sh.pl[X]);
            const real4 pv = sh.vx[first_arc];
            put_test_point(sh, fi, 2.0 * cp.x - pv.x, 2.0 * cp.y - pv.y, 2.0 * cp.z - pv.z);
        }
        nf += __popc(m);
    }
    __syncwarp();
    faces_inside(sh, NC, nf, lane);
    int n_extra = 0, fi0 = 0;
    #pragma unroll 1
    for (int x0 = 0; x0 < NC; x0 += 32) {
        const int X = x0 + lane;
        const uint32_t cm = sh.cmask[x0 >> 5], em = cm & ~sh.bad[x0 >> 5];
        const int t = __popc(em);
        if (NV + n_extra + t > Sh::verts - 1) return Sh::over;
        if ((em >> lane) & 1u) {
            const int w = NV + n_extra + __popc(em & lanemask_lt());
            if (hist) {
                hist_vx(hist)[w - NV] = sh.vx[w];
                hist_vp(hist)[w - NV] = sh.vp[w];
            }
            const double* ex = &sh.u.f.val[3 * (fi0 + __popc(cm & lanemask_lt()))];
            sh.vx[w] = make_real4(ex[0], ex[1], ex[2], rado);
            sh.vp[w] = make_uchar4((uint8_t)X, kNone, kNone, 0);
            sh.u.f.pt[sh.foff[X] + sh.fnp[X]] = (uint8_t)w;
            sh.fnp[X] += 1;
        }
        n_extra += t;
        fi0 += __popc(cm);
    }
    __syncwarp();
    // ordering around each face (pt[0], a neighbour of it, then decreasing cosine): the second
    // point per face (one face per lane), the cosines of all faces' points spread over the lanes,
    // then each face's sort and its history (one face per lane)
    int np_miss = 0, np_lost = 0, t_run = 0;
    #pragma unroll 1
    for (int x0 = 0; x0 < NC; x0 += 32) {
        const int X = x0 + lane;
        const bool face = X < NC && sh.flag[X] != 0;
        const int np = face ? sh.fnp[X] : 0;
        int tt;
        const int to = t_run + warp_excl_scan(np > 2 ? np - 2 : 0, lane, &tt);
        t_run += tt;
        if (t_run > Sh::items) return Sh::over;
        if (X < NC) sh.toff[X] = (uint16_t)to;
        if (!face) continue;
        uint8_t* pt = &sh.u.f.pt[sh.foff[X]];
        int stale_prev = kNone;   // point 1 of the face before a replayed read of the slot past its end
        if (np > 3) {
            const uchar4 P0 = sh.vp[pt[0]];
            const int pY = (P0.x == X) ? P0.y : P0.x;
            // the first later point of the face on plane pY (the face's vertices are its mask's bits in order)
            const uint32_t* vm = &sh.vmask[X * NW];
            const int v = first_vertex<Sh>(vm, &sh.vmask[pY * NW], pt[0] + 1);
            int vi = 1;
            bool replayed = false;
            if (v >= 0) {
                vi = __popc(vm[v >> 5] & ((1u << (v & 31)) - 1u));
                #pragma unroll 1
                for (int w = 0; w < v >> 5; ++w) vi += __popc(vm[w]);
            } else {
                ++np_miss;
                const int s = (hist && np < kHistPts) ? (int)hist[X * kHistPts + np] : -1;
                if (s >= 0 && s < Sh::verts - 1) {
                    // the reference swaps pt[1] with the stale slot: the slot's vertex becomes
                    // point 1, the old point 1 stays behind in the slot
                    replayed = true;
                    stale_prev = pt[1];
                    pt[1] = (uint8_t)s;
                } else {
                    if (hist) ++np_lost;
                    const int pZ = (P0.x == X || P0.y == X) ? P0.z : P0.y;
                    if (pZ != kNone) {
                        int w = 1;
                        #pragma unroll 1
                        for (; w < np; ++w) {
                            const uchar4 q = sh.vp[pt[w]];
                            if (q.x == pZ || q.y == pZ || q.z == pZ) break;
                        }
                        if (w < np) vi = w;
                    }
                }
            }
            if (!replayed) {
                const uint8_t tmp = pt[vi];
                pt[vi] = pt[1];
                pt[1] = tmp;
            }
            #pragma unroll 1
            for (int j = 2; j < np; ++j) sh.u.f.item[to + j - 2] = (uint32_t)X | ((uint32_t)pt[j] << 8);
        } else if (np == 3) {
            sh.u.f.item[to] = kNone;   // (no cosine)
        }
        sh.sprev[X] = (uint8_t)stale_prev;
    }
    miss += np_miss;
    lost += np_lost;
    __syncwarp();
    long long* const key = reinterpret_cast<long long*>(sh.u.f.val);
    #pragma unroll 1
    for (int k = lane; k < t_run; k += 32) {
        const uint32_t it = sh.u.f.item[k];
        const int X = it & 0xffu;
        if (X == kNone) continue;
        const uint8_t* pt = &sh.u.f.pt[sh.foff[X]];
        // point 1 is read as it stood when the reference ordered this face: a replayed
        // slot that a later face's antipodal point takes still held its old vertex
        const int s1 = pt[1];
        const real4 v1 = (hist && s1 >= NV && s1 < NV + n_extra && sh.vp[s1].x > X) ? hist_vx(hist)[s1 - NV] : sh.vx[s1];
        key[k] = cos_key(cos_pqr(v1, sh.vx[pt[0]], sh.vx[it >> 8]));
    }
    __syncwarp();
    #pragma unroll 1
    for (int X = lane; X < NC; X += 32) {
        if (sh.flag[X] == 0) continue;
        const int np = sh.fnp[X];
        uint8_t* pt = &sh.u.f.pt[sh.foff[X]];
        if (np > 3) {
            long long* cs = key + sh.toff[X] - 2;
            #pragma unroll 1
            for (int a = 2; a < np - 1; ++a) {
                long long ca = cs[a];
                int pa = pt[a];
                #pragma unroll 1
                for (int b = a + 1; b < np; ++b) {
                    const long long cb = cs[b];
                    if (key_less(ca, cb)) {
                        cs[b] = ca;
                        ca = cb;
                        const int pb = pt[b];
                        pt[b] = (uint8_t)pa;
                        pa = pb;
                    }
                }
                cs[a] = ca;
                pt[a] = (uint8_t)pa;
            }
        }
        if (hist) {
            uint8_t* h = hist + X * kHistPts;
            const int nw = np < kHistPts ? np : kHistPts;
            #pragma unroll 1
            for (int k = 0; k < nw; ++k) h[k] = pt[k];
            if (sh.sprev[X] != kNone) h[np] = sh.sprev[X];
        }
    }
    __syncwarp();
    sh.nt = t_run;
    return kAtomOk;
}

// Whether consecutive points of planes qa and qb of a face bound an arc segment: both arc points,
// of different edges (LIB/Vcontacts.cpp:943-954).
__device__ __forceinline__ int arc_segment(const uchar4& qa, const uchar4& qb) {
    if (qa.z != kNone || qb.z != kNone) return 0;
    const int sa = (qa.y == kNone ? -1 : qa.y) + qa.x;
    const int sb = (qb.y == kNone ? -1 : qb.y) + qb.x;
    return sa != sb;
}

// The items of calc_areas (LIB/Vcontacts.cpp:838-1044): fan triangles of every face (v0, va, vb),
// the arcs between its consecutive arc points and a lens's one arc (face, point, point), then the
// arcs of the engulfed faces credited to their neighbours (:963-1041), in the reference's order; and
// the caps' and lenses' inside tests. With three engulfing planes the reference overwrites every
// area, so there is nothing to evaluate.
template <class Sh>
__device__ __forceinline__ int area_items(Vor<Sh>& sh, int NC, int NV, double rado, double rr, int lane) {
    // the first three engulfing planes in plane order
    int epi = 0;
    #pragma unroll 1
    for (int x0 = 0; x0 < NC && epi < 3; x0 += 32) {
        const int X = x0 + lane;
        unsigned mm = __ballot_sync(kFull, X < NC && (sh.flag[X] & kEngulf));
        while (mm && epi < 3) {
            const int b = __ffs(mm) - 1;
            mm &= mm - 1;
            if (lane == 0) sh.eng[epi] = x0 + b;
            ++epi;
        }
    }
    __syncwarp();
    sh.epi = epi;
    bool lens2 = false;
    if (epi > 0) {
        // project_points (LIB/Vcontacts.cpp:1278-1344)
        double pp[3];
        if (epi == 1) {
            const real4 c = centre_of(sh.pl[sh.eng[0]]);
            pp[0] = c.x; pp[1] = c.y; pp[2] = c.z;
        } else if (epi == 2) {
            double q0[3], q1[3];
            lens2 = solve2s(sh.pl[sh.eng[0]], sh.pl[sh.eng[1]], rr, q0, q1);
            if (!lens2) {
                const float4 c = sh.centre;
                pp[0] = c.x; pp[1] = c.y; pp[2] = c.z;
            } else {
                pp[0] = (q0[0] + q1[0]) * 0.5;   // the same value as / 2
                pp[1] = (q0[1] + q1[1]) * 0.5;
                pp[2] = (q0[2] + q1[2]) * 0.5;
                if (lane == 0) {
                    sh.vx[Sh::verts] = make_real4(q0[0], q0[1], q0[2], rado);
                    sh.vx[Sh::verts + 1] = make_real4(q1[0], q1[1], q1[2], rado);
                }
            }
        } else {
            solve3(sh.pl[sh.eng[0]], sh.pl[sh.eng[1]], sh.pl[sh.eng[2]], pp);
        }
        #pragma unroll 1
        for (int vi = lane; vi < NV; vi += 32) {
            if (sh.vp[vi].z == kNone) continue;
            real4 P = sh.vx[vi];
            const double Vx = P.x - pp[0], Vy = P.y - pp[1], Vz = P.z - pp[2];
            const double a = Vx * Vx + Vy * Vy + Vz * Vz;
            const double b = 2 * (P.x * Vx + P.y * Vy + P.z * Vz);
            const double c = P.x * P.x + P.y * P.y + P.z * P.z - rr;
            const double k = ddiv(dsqrt(b * b - 4.0 * a * c) - b, 2 * a);
            P.x += k * Vx; P.y += k * Vy; P.z += k * Vz;
            P.w = rado;
            sh.vx[vi] = P;
        }
        __syncwarp();
        if (epi == 3) {
            sh.nt = sh.na = sh.ne = 0;
            return kAtomOk;
        }
    }
    const int T = sh.nt;
    int a_run = 0, nf = 0;
    #pragma unroll 1
    for (int x0 = 0; x0 < NC; x0 += 32) {
        const int X = x0 + lane;
        const bool face = X < NC && sh.flag[X] != 0;
        const int np = face ? sh.fnp[X] : 1;
        const uint8_t* pt = &sh.u.f.pt[face ? sh.foff[X] : 0];
        const bool ring = np == 0 || np == 2;
        int na = np == 2 ? 1 : 0;
        if (np > 2) {
            uchar4 qa = sh.vp[pt[np - 1]];
            #pragma unroll 1
            for (int vi = 0; vi < np; ++vi) {
                const uchar4 qb = sh.vp[pt[vi]];
                na += arc_segment(qa, qb);
                qa = qb;
            }
        }
        int ta;
        int ao = a_run + warp_excl_scan(na, lane, &ta);
        a_run += ta;
        const unsigned m = __ballot_sync(kFull, ring);
        if (T + a_run > Sh::items || 3 * (nf + __popc(m)) > Sh::items / 2) return Sh::over;
        if (X < NC) sh.aoff[X] = (uint16_t)ao;
        if (ring) {
            const int fi = nf + __popc(m & lanemask_lt());
            sh.flist[fi] = (uint8_t)X;
            const real4 cp = centre_of(sh.pl[X]);
            put_test_point(sh, fi, cp.x, cp.y, cp.z);
        }
        nf += __popc(m);
        const uint32_t self = (uint32_t)X | ((uint32_t)X << 24);
        if (np == 2) {
            sh.u.f.item[T + ao] = self | ((uint32_t)pt[0] << 8) | ((uint32_t)pt[1] << 16);
        } else if (np > 2) {
            const uint32_t p0 = pt[0];
            uint32_t pa = p0;
            uchar4 qa = sh.vp[pa];
            uint32_t* tri = &sh.u.f.item[sh.toff[X]];
            #pragma unroll 1
            for (int vi = 1; vi <= np; ++vi) {
                const uint32_t pb = vi < np ? pt[vi] : p0;
                const uchar4 qb = sh.vp[pb];
                if (vi > 1 && vi < np) tri[vi - 2] = p0 | (pa << 8) | (pb << 16);
                if (arc_segment(qa, qb)) sh.u.f.item[T + ao++] = self | (pa << 8) | (pb << 16);
                pa = pb;
                qa = qb;
            }
        }
    }
    if (lane == 0) {
        sh.toff[NC] = (uint16_t)T;
        sh.aoff[NC] = (uint16_t)a_run;
        sh.na = a_run;
    }
    __syncwarp();
    faces_inside(sh, NC, nf, lane);
    int ne = 0;
    #pragma unroll 1
    for (int i = 0; i < epi; ++i) {
        const int X = sh.eng[i], np = sh.fnp[X];
        const uint8_t* pt = &sh.u.f.pt[sh.foff[X]];
        #pragma unroll 1
        for (int v0 = 0; v0 < np; v0 += 32) {
            const int vi = v0 + lane;
            int comm = -1, cur = 0, nxt = 0;
            // a face of two points stops after its first credited (or sphere-bound) arc
            if (vi < np && !(np == 2 && vi == 1 && engulf_comm(sh, NC, X, pt[0], pt[1]) >= 0)) {
                cur = pt[vi];
                nxt = pt[vi + 1 < np ? vi + 1 : 0];
                const int c = engulf_comm(sh, NC, X, cur, nxt);
                if (c >= 0 && c < NC) comm = c;
            }
            const unsigned m = __ballot_sync(kFull, comm >= 0);
            if (T + a_run + ne + __popc(m) + 2 > Sh::items) return Sh::over;
            if (comm >= 0)
                sh.u.f.item[T + a_run + ne + __popc(m & lanemask_lt())] =
                    (uint32_t)X | ((uint32_t)cur << 8) | ((uint32_t)nxt << 16) | ((uint32_t)comm << 24);
            ne += __popc(m);
        }
    }
    if (lens2) {
        // the lens their circles cut: its two arcs, the last two items
        if (T + a_run + ne + 2 > Sh::items) return Sh::over;
        if (lane < 2)
            sh.u.f.item[T + a_run + ne + lane] = (uint32_t)sh.eng[lane] | ((uint32_t)Sh::verts << 8) |
                                                 ((uint32_t)(Sh::verts + 1) << 16) | ((uint32_t)kNone << 24);
        ne += 2;
    }
    sh.ne = ne;
    __syncwarp();
    return kAtomOk;
}

// The warps of a block that step together: kSize of them, of which this warp is `slot`.
template <int kSize>
struct Group {
    static constexpr int size = kSize;
    int slot, barrier;
    int4* step;              // per pose: triangle items, arc items, whether the pose goes on, and an atom
    int2* saved;             // saved in the step before whose terms are to be summed (-1: none); its pose, job
    int* n_retry;            // poses to score again in the large shape
    int* retry;              // [2 * size]
};

// The group's barrier (a named one: 1 ..; 0 is the block's own).
template <int kSize>
__device__ __forceinline__ void group_sync(const Group<kSize>& g) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(g.barrier), "n"(kSize * 32) : "memory");
}

// The area of face X from its items' values, the sum in the reference's order (triangles, then
// arcs, then credited arcs).
template <class Sh>
__device__ __forceinline__ double face_area(const Vor<Sh>& sh, int X) {
    const int epi = sh.epi, T = sh.nt, nA = sh.na, ne = sh.ne;
    const double rado = sh.rado;
    const double two_pi_r = 2.0 * kPi * rado;
    double a = 0.0;
    const int flag = sh.flag[X];
    if (epi == 3) {
        if (flag & kEngulf) a = ddiv(4.0 * kPi * rado * rado, 3.0);
    } else if (flag != 0) {
        const int np = sh.fnp[X];
        if (np == 0 || np == 2) {
            const bool inside = !((sh.bad[X >> 5] >> (X & 31)) & 1u);
            if (inside) a = two_pi_r * (rado - fabs(sh.pl[X].w));
            if (np == 2) {
                const double v = sh.u.f.val[T + sh.aoff[X]];
                a = inside ? a - v : v;
            }
        } else {
            #pragma unroll 1
            for (int i = sh.toff[X]; i < sh.toff[X + 1]; ++i) a += sh.u.f.val[i];
            #pragma unroll 1
            for (int i = T + sh.aoff[X]; i < T + sh.aoff[X + 1]; ++i) a += sh.u.f.val[i];
        }
        #pragma unroll 1
        for (int i = T + nA; i < T + nA + ne; ++i)
            if ((int)(sh.u.f.item[i] >> 24) == X) a += sh.u.f.val[i];
        if (epi == 1 && X == sh.eng[0]) {
            a = two_pi_r * (rado + fabs(sh.pl[X].w));
        } else if (epi == 2 && (X == sh.eng[0] || X == sh.eng[1])) {
            a = two_pi_r * rado;
            // the lens's arcs, when there is one, are the last two items
            if (ne >= 2 && (sh.u.f.item[T + nA + ne - 1] >> 24) == kNone)
                a -= 0.5 * (sh.u.f.val[T + nA + ne - 2] + sh.u.f.val[T + nA + ne - 1]);
        }
    }
    return a;
}

// Planes of the contacts of one scored atom (LIB/Vcontacts.cpp:186-221): the candidates whose
// bit in sh.excl is clear (the list get_contlist4 gives; an excluded candidate is a saved atom that
// kept no contact with this one, or one at distance zero), packed in candidate order, so that
// each plane's index, and every tie-break on it, is the reference's contact index. Returns NC.
template <class Sh>
__device__ __forceinline__ int load_planes(Vor<Sh>& sh, const DevSystem& S, const DevWork& W, int p, int a,
                                           int n_cand, float4 me, int lane) {
    const int nm = n_mobile(S);
    const size_t cb = ((size_t)p * nm + a) * kMaxCand;
    const float rado = me.w + kRw, rr = rado * rado;   // single-precision products, as in the reference
    const double rrd = f2d(rr);
    int NC = 0;
    #pragma unroll 1
    for (int c0 = 0; c0 < n_cand; c0 += 32) {
        const int c = c0 + lane;
        const bool keep = c < n_cand && !((sh.excl[c0 >> 5] >> lane) & 1u);
        const unsigned m = __ballot_sync(kFull, keep);
        if (keep) {
            const int r = NC + __popc(m & lanemask_lt());
            const int j = W.cand_idx[cb + c];
            const float d2 = W.cand_d2[cb + c];
            sh.cidx[r] = j;
            sh.cslot[r] = (uint8_t)c;
            const int mj = mobile_of(S, j);
            const float4 pj = mj < 0 ? S.rec_pos[j] : W.mob_pos[(size_t)p * nm + mj];
            const double d = dsqrt(f2d(d2));
            const float q = kRw + pj.w;
            const float qq = q * q;
            const double num = (d * d + rrd) - f2d(qq);
            const real4 P = make_real4(ddiv(f2d(pj.x - me.x), d), ddiv(f2d(pj.y - me.y), d), ddiv(f2d(pj.z - me.z), d),
                                       -ddiv(num, 2.0 * d));
            sh.pl[r] = P;
            sh.plf[r] = make_float4(d2f_trunc(P.x), d2f_trunc(P.y), d2f_trunc(P.z), d2f_trunc(P.w));
            sh.flag[r] = lt0(num) ? kEngulf : 0;
        }
        NC += __popc(m);
    }
    if (lane < 4) {   // the bounding planes
        const double bx = lane < 2 ? 0.707 : -0.707;
        const double by = lane == 0 ? 1.0 : lane == 1 ? -1.0 : 0.0, bz = lane == 2 ? 1.0 : lane == 3 ? -1.0 : 0.0;
        sh.pl[NC + lane] = make_real4(bx, by, bz, -10.0);
        sh.plf[NC + lane] = make_float4(lane < 2 ? 0.707f : -0.707f, d2f_trunc(by), d2f_trunc(bz), -10.0f);
        sh.flag[NC + lane] = 0;
    }
    if (lane == 0) {
        // project_points' fallback centre for two engulfing planes: the atom's own coordinates + rado
        sh.centre = make_float4(me.x + rado, me.y, me.z, 0.0f);
        sh.rado = f2d(rado);
        sh.rr = rr;
    }
    __syncwarp();
    return NC;
}

__device__ __forceinline__ double pose_clash_sum(const DevSystem& S, const DevWork& W, int p, int lane) {
    const int nm = n_mobile(S);
    double s = 0.0;
    #pragma unroll 1
    for (int m = lane; m < nm; m += 32) s += W.clash_part[(size_t)p * nm + m];
    return warp_sum(s);
}

__device__ __forceinline__ bool bit(const uint32_t* m, int l) { return (m[l >> 5] >> (l & 31)) & 1u; }

__device__ __forceinline__ void finish_failed(const DevWork& W, int p, int lane, int status, double wal) {
    fxe_cf cf;
    memset(&cf, 0, sizeof(cf));
    cf.status = status;
    if (status != FXE_POSE_CAPACITY) {
        // the reference's positional initialiser puts 1 into metal_coord (LIB/ic2cf.cpp:127-131)
        cf.wal = wal;
        cf.metal_coord = 1.0;
        cf.evalue = cf.wal + cf.metal_coord;
    }
    if (lane == 0) W.out[p] = cf;
}

// The entry of the energy matrix at curve position rel (taken lazily: a single-valued entry does
// not need it): the curve's value, times `area` when it is a weight.
__device__ __forceinline__ double matrix_term(const DevSystem& S, int idx, double area, double surf) {
    const int o = S.em_off[idx], e = S.em_off[idx + 1];
    if (S.em_weight[idx]) return f2d(S.em_y[o]) * area;
    const double rel = area / surf;
    int k = o;
    while (k + 1 < e && rel > (double)S.em_x[k + 1]) ++k;
    if ((double)S.em_x[k] > rel) return 0.0;
    if (k + 1 >= e) return (double)S.em_y[k];
    return (double)S.em_y[k] + (rel - (double)S.em_x[k]) / (double)(S.em_x[k + 1] - S.em_x[k]) *
                                   (double)(S.em_y[k + 1] - S.em_y[k]);
}

// vcfunction (LIB/vcfunction.cpp:84-513) for scored atom i of a pose (mobile atoms lb ..): the terms of
// its kept contacts and its solvent term into W.atom_terms (complementarity, wall, solvent, and the
// accessible surface). Called as each atom is saved, so that no pose's scoring holds its group.
__device__ __noinline__ void score_atom(const DevSystem& S, const DevWork& W, size_t lb, int i, int lane) {
    const int T = S.ntypes, nsc = S.n_sc;
    const int NC = W.cand_n[lb + i];
    const size_t cb = (lb + i) * kMaxCand;
    const bool side = i < nsc;
    const float radf = W.mob_pos[lb + i].w;
    const double radA = f2d(radf);
    const double radoA = radA + (double)kRw;
    const double surfA = 4.0 * kPi * radoA * radoA;
    const int ti = side ? S.rec_type[S.sc_slot[i]] : S.lig_type[i - nsc];
    double c_com = 0.0, c_wal = 0.0, c_area = 0.0;
    #pragma unroll 1
    for (int c = lane; c < NC; c += 32) {
        if (!(W.cand_flag[cb + c] & kRecorded)) continue;
        const int j = W.cand_idx[cb + c];
        const double area = W.cand_area[cb + c];
        c_area += area;
        const int rel = residue_pair(S, i, j);
        if (rel == 1) continue;                      // bonded within the residue
        const int mj = mobile_of(S, j);
        if (mj >= 0 && mj < i) continue;             // FA->contacts: scored from that atom
        const bool lig_j = j >= S.n_rec;
        const float rj = lig_j ? S.lig_radius[j - S.n_rec] : (mj >= 0 ? W.mob_pos[lb + mj].w : S.rec_pos[j].w);
        const int tj = lig_j ? S.lig_type[j - S.n_rec] : S.rec_type[j];
        // intramolecular: one residue, or two protein residues (LIB/vcfunction.cpp:283-291)
        const bool intra = rel != 0 || (side && !lig_j);
        if (S.intramolecular || !intra) c_com += matrix_term(S, (ti - 1) * T + (tj - 1), area, surfA);
        const float d2 = W.cand_d2[cb + c];
        const float cdf = S.permeability * (radf + rj);   // the clash distance, to single precision
        if (d2 < cdf * cdf * 1.0002f) {
            const double permea = (double)S.permeability;
            const double rAB = radA + (double)rj;
            const float clash_distance = (float)(permea * rAB);
            if (d2 < clash_distance * clash_distance * 1.0001f) {
                const double dd = sqrt((double)d2);
                if (dd < (double)clash_distance) {
                    const double q2 = dd * dd, q4 = q2 * q2, q6 = q4 * q2;
                    const double cr = permea * rAB;
                    const double r2 = cr * cr, r4 = r2 * r2, r6 = r4 * r2;
                    c_wal += (double)kKwall * (1.0 / (q6 * q6) - 1.0 / (r6 * r6));
                }
            }
        }
    }
    // both sums in one reduction: after the first exchange the lower half holds c_com's
    // partial sums, the upper half c_area's (the additions are warp_sum's)
    {
        const bool up = lane >= 16;
        double x = (up ? c_area : c_com) + __shfl_xor_sync(kFull, up ? c_com : c_area, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
        c_com = __shfl_sync(kFull, x, 0);
        c_area = __shfl_sync(kFull, x, 16);
    }
    if (__any_sync(kFull, !is0(c_wal))) c_wal = warp_sum(c_wal);
    double SAS = surfA - c_area;
    if (lt0(SAS)) SAS = 0.0;
    const double sas = S.solventterm != 0.0f ? (double)S.solventterm * SAS : matrix_term(S, (ti - 1) * T + (T - 1), SAS, surfA);
    if (lane == 0) {
        double* t = W.atom_terms + (lb + i) * 4;
        t[0] = c_com;
        t[1] = c_wal;
        t[2] = sas;
        t[3] = SAS;
    }
}

// The pose's record from its atoms' terms, in Calc order (side-chain atoms, then the ligand): each
// residue's are summed on their own and the records added up ligand first, then the side chains in
// order (LIB/ic2cf.cpp:133-245). One term per lane.
__device__ __noinline__ void finish_scored(const DevSystem& S, const DevWork& W, int p, int lane) {
    const int nl = n_mobile(S), nsc = S.n_sc;
    const double* t = W.atom_terms + (size_t)p * nl * 4 + (lane & 3);
    double sum = 0.0;
    for (int i = nsc; i < nl; ++i) sum += t[4 * i];
    if ((lane & 3) < 3) {
        double res = 0.0;
        for (int i = 0; i < nsc; ++i) {
            res += t[4 * i];
            if (i + 1 == nsc || S.sc_res[i + 1] != S.sc_res[i]) {
                sum += res;
                res = 0.0;
            }
        }
    }
    fxe_cf cf;
    memset(&cf, 0, sizeof(cf));
    cf.com = __shfl_sync(kFull, sum, 0);
    cf.wal = __shfl_sync(kFull, sum, 1);
    cf.sas = __shfl_sync(kFull, sum, 2);
    cf.totsas = __shfl_sync(kFull, sum, 3);
    cf.evalue = cf.com + cf.wal + cf.sas + cf.con + cf.elec + cf.hbond + cf.gist_desolv + cf.metal_coord;
    cf.status = FXE_POSE_SCORED;
    if (lane == 0) W.out[p] = cf;
}

// The start of scored atom a of pose p: its contact list, planes and first vertex. kAtomNone when it
// has no contacts.
template <class Sh>
__device__ __forceinline__ int start_atom(const DevSystem& S, const DevWork& W, int p, int a, int lane, PoseShared<Sh>& ps, size_t cb,
                                          int n_cand, const uint32_t* kept, const int* seed, int* NC_out, Walk& walk) {
    Vor<Sh>& sh = ps.v;
    // get_contlist4's list: saved atoms drop out unless they kept a contact with this one, and so
    // does an atom at distance zero
    const uint4 kp = *reinterpret_cast<const uint4*>(kept);
    int kept_n = 0;
    #pragma unroll 1
    for (int c0 = 0; c0 < n_cand; c0 += 32) {
        const int c = c0 + lane;
        bool ex = c >= n_cand;
        if (!ex) {
            const int l = mobile_of(S, W.cand_idx[cb + c]);
            if (l >= 0) {
                const uint32_t kw = l < 64 ? (l < 32 ? kp.x : kp.y) : (l < 96 ? kp.z : kp.w);
                ex = bit(ps.done, l) && !((kw >> (l & 31)) & 1u);
            }
            if (W.cand_d2[cb + c] < 1e-20f) ex = true;
        }
        const uint32_t em = __ballot_sync(kFull, ex);
        if (lane == 0) sh.excl[c0 >> 5] = em;
        kept_n += __popc(~em);
    }
    __syncwarp();
    if (kept_n == 0) {
        #pragma unroll 1
        for (int c = lane; c < n_cand; c += 32) {
            W.cand_area[cb + c] = 0.0;
            W.cand_flag[cb + c] = 0;
        }
        __syncwarp();
        score_atom(S, W, (size_t)p * n_mobile(S), a, lane);
        return kAtomNone;
    }
    const float4 me = W.mob_pos[(size_t)p * n_mobile(S) + a];
    const int NC = load_planes(sh, S, W, p, a, n_cand, me, lane);
    *NC_out = NC;
    // the first vertex: the seed left by an earlier atom, if all three of its planes are in the
    // list, else the search from the closest plane
    int sA = -1, sB = -1, sC = -1;
    const int s0 = seed[0], s1 = seed[1], s2 = seed[2];
    if (s0 != -1) {
        #pragma unroll 1
        for (int c0 = 0; c0 < NC; c0 += 32) {
            const int c = c0 + lane;
            const int j = c < NC ? sh.cidx[c] : -2;
            const unsigned m0 = __ballot_sync(kFull, j == s0);
            const unsigned m1 = __ballot_sync(kFull, j == s1 && j != s0);
            const unsigned m2 = __ballot_sync(kFull, j == s2 && j != s0 && j != s1);
            if (m0) sA = c0 + 31 - __clz(m0);
            if (m1) sB = c0 + 31 - __clz(m1);
            if (m2) sC = c0 + 31 - __clz(m2);
        }
    }
    if (sA < 0 || sB < 0 || sC < 0)
        if (!first_planes_fast(sh, NC, lane, &sA, &sB, &sC) && !first_planes_exact(sh, NC, lane, &sA, &sB, &sC)) return kAtomCapacity;
    walk_start(sh, lane, sA, sB, sC, walk);
    return kAtomOk;
}

// A warp's pose: its place and its current atom's state.
struct Pose {
    int p, entry, job;       // index in the workspace, queue entry, job
    int r, a, n_cand, NC;    // the atom's place in Calclist order, the atom, its candidates and contacts
    int miss, lost;          // per lane: faces without a neighbour, and those not replayed
    bool alive, walking;     // walking: the atom's hull walk goes on
    Walk walk;
};

// Where a launch's poses lie: one system's, or several jobs' (their descriptors are read from the job
// table and stay in L1, keeping shared memory for the polyhedron workspace).
struct OneJob {
    const DevSystem& s;
    const DevWork& w;
    __device__ __forceinline__ const DevSystem& S(const Pose&) const { return s; }
    __device__ __forceinline__ const DevWork& W(const Pose&) const { return w; }
    __device__ __forceinline__ void place(Pose& q) const { q.p = q.entry; }
};
struct ManyJobs {
    const Job* jobs;
    int n;
    __device__ __forceinline__ const DevSystem& S(const Pose& q) const { return jobs[q.job].S; }
    __device__ __forceinline__ const DevWork& W(const Pose& q) const { return jobs[q.job].W; }
    __device__ __forceinline__ void place(Pose& q) const {
        q.job = find_job(jobs, n, q.entry, false);
        q.p = q.entry - jobs[q.job].pose0;
    }
};

// Takes pose q.p up: false when it is done already (clash pre-filter, or it left the grid).
template <class Sh, class Jobs>
__device__ __forceinline__ bool begin_pose(const Jobs& jobs, Pose& q, int lane, PoseShared<Sh>& ps, uint8_t* hist) {
    const DevSystem& S = jobs.S(q);
    const DevWork& W = jobs.W(q);
    const int p = q.p, nl = n_mobile(S);
    if (W.pose_grid[p].z) {
        finish_failed(W, p, lane, FXE_POSE_CAPACITY, 0.0);
        return false;
    }
    // clash pre-filter (LIB/Vcontacts.cpp:36-51)
    const double clash = pose_clash_sum(S, W, p, lane);
    if (clash >= kClashThreshold) {
        finish_failed(W, p, lane, FXE_POSE_CLASHED, clash);
        return false;
    }
    const size_t lb = (size_t)p * nl;
    #pragma unroll 1
    for (int l = lane; l < nl; l += 32) {
        ps.order[W.mob_rank[lb + l]] = (uint8_t)l;
        int* seed = W.pose_seed + ((size_t)p * kMaxLig + l) * 3;
        seed[0] = seed[1] = seed[2] = -1;
        *reinterpret_cast<uint4*>(W.pose_rec + ((size_t)p * kMaxLig + l) * kMaskWords) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (lane < kMaskWords) ps.done[lane] = 0;
    // the face history starts the pose at zero, as the reference's ptorder does on a workspace
    // cleared before the pose
    if (hist) {
        uint4* h4 = reinterpret_cast<uint4*>(hist);
        #pragma unroll 1
        for (int k = lane; k < kHistBytes / 16; k += 32) h4[k] = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncwarp();
    q.r = q.miss = q.lost = 0;
    q.walking = false;
    return true;
}

// The pose's share of a group step up to the area items: its next atom (or more of its walk).
// kAtomOk: the atom has items and areas to sum; kAtomWalking; kAtomNone: an atom without contacts;
// else the pose ends here.
template <class Sh, class Jobs>
__device__ __forceinline__ int step_pose(const Jobs& jobs, Pose& q, int lane, PoseShared<Sh>& ps, uint8_t* hist) {
    static_assert(kMaskWords == 4, "an atom's mask is read as one uint4");
    const DevSystem& S = jobs.S(q);
    const DevWork& W = jobs.W(q);
    Vor<Sh>& sh = ps.v;
    const size_t lb = (size_t)q.p * n_mobile(S);
    if (!q.walking) {
        q.a = ps.order[q.r];
        q.n_cand = W.cand_n[lb + q.a];
        if (q.n_cand < 0) return kAtomCapacity;
        const int st = start_atom(S, W, q.p, q.a, lane, ps, (lb + q.a) * kMaxCand, q.n_cand,
                                  W.pose_rec + ((size_t)q.p * kMaxLig + q.a) * kMaskWords,
                                  W.pose_seed + ((size_t)q.p * kMaxLig + q.a) * 3, &q.NC, q.walk);
        if (st != kAtomOk) return st;
    }
    const double rr = f2d(sh.rr), rado = sh.rado;
    int st = hull_walk(sh, q.NC, rr, lane, q.walk), NV = 0;
    q.walking = st == kAtomWalking;
    if (st == kAtomOk) st = arc_points(sh, rado, rr, lane, q.walk.vn, q.walk.edges, &NV);
    if (st == kAtomOk) st = order_faces(sh, q.NC, NV, rado, lane, hist, q.miss, q.lost);
    if (st == kAtomOk) st = area_items(sh, q.NC, NV, rado, rr, lane);
    return st;
}

// Saves the atom whose areas are in: save_areas (LIB/Vcontacts.cpp:1149-1220: contacts with area > 0 on
// a contact plane; candidates outside the contact list record nothing), save_seeds (:601-629: the first
// vertex naming a later atom's plane).
template <class Sh, class Jobs>
__device__ __forceinline__ void save_atom(const Jobs& jobs, const Pose& q, int lane, PoseShared<Sh>& ps) {
    const DevSystem& S = jobs.S(q);
    const DevWork& W = jobs.W(q);
    Vor<Sh>& sh = ps.v;
    const size_t lb = (size_t)q.p * n_mobile(S), cb = (lb + q.a) * kMaxCand;
    const int az = slot_of(S, q.a);
    #pragma unroll 1
    for (int c = lane; c < q.n_cand; c += 32) {
        if (bit(sh.excl, c)) {
            W.cand_area[cb + c] = 0.0;
            W.cand_flag[cb + c] = 0;
        }
    }
    #pragma unroll 1
    for (int k = lane; k < q.NC; k += 32) {
        const double ar = face_area(sh, k);
        const uint8_t f = sh.flag[k];
        const bool keep = gt0(ar) && (f & (kOnHull | kEngulf));
        const int c = sh.cslot[k];
        W.cand_area[cb + c] = ar;
        W.cand_flag[cb + c] = (uint8_t)(f | (keep ? kRecorded : 0));
        const int m = mobile_of(S, sh.cidx[k]);
        if (m >= 0) {
            if (keep) W.pose_rec[((size_t)q.p * kMaxLig + m) * kMaskWords + (q.a >> 5)] |= 1u << (q.a & 31);
            int* seed = W.pose_seed + ((size_t)q.p * kMaxLig + m) * 3;
            const int vi = sh.fseed[k];
            if (vi != kNone && seed[0] == -1) {
                const uchar4 v = sh.vp[vi];
                const int p1 = v.x == k ? v.y : v.x, p2 = v.z == k ? v.y : v.z;
                seed[0] = az;
                seed[1] = sh.cidx[p1];
                seed[2] = sh.cidx[p2];
            }
        }
    }
    if (lane == 0) ps.done[q.a >> 5] |= 1u << (q.a & 31);
    __syncwarp();
}

// The launch's counters of a finished pose.
__device__ __forceinline__ void count_faces(const DevWork& W, const Pose& q, int lane) {
    const int miss = warp_sum(q.miss), lost = warp_sum(q.lost);
    if (lane == 0 && miss) atomicAdd(&W.counters[3], miss);
    if (lane == 0 && lost) atomicAdd(&W.counters[0], lost);
}

// Whether a saved atom's terms are summed by any of the group's warps in the next step, beside the areas,
// or by its own warp at once. In the groups of few poses most warps have nothing else to do: one pose of
// 24 atoms takes 1,283 us so and 1,355 otherwise, 500 poses 1,683 and 1,744. A full group's warps are busy
// with the areas (2,000 poses: 7.53 ms and 7.37).
template <int kSize>
constexpr bool kScoreLater = kSize < kWarps;

// What the group's warps share out in a step: every pose's triangles as one list, 32 at a time, then
// every pose's arcs, then the atoms saved in the step before whose terms are still to be summed. Group
// barriers around it keep the items' owners out.
template <class Sh, int kSize, class Jobs>
__device__ __forceinline__ void pooled_work(const Jobs& jobs, PoseShared<Sh>* all, const Group<kSize>& g, int lane) {
    static_assert(kWarps <= 32, "one lane per pose in the prefix sums");
    const int4 n = lane < g.size ? g.step[lane] : make_int4(0, 0, 0, -1);
    const unsigned scores = kScoreLater<kSize> ? __ballot_sync(kFull, n.w >= 0) : 0u;
    int T, A;
    const int tpre = warp_excl_scan(n.x, lane, &T), apre = warp_excl_scan(n.y, lane, &A);
    const int tch = (T + 31) >> 5, ach = (A + 31) >> 5;
    #pragma unroll 1
    for (int ch = g.slot; ch < tch + ach + __popc(scores); ch += g.size) {
        if (kScoreLater<kSize> && ch >= tch + ach) {
            unsigned m = scores;
            for (int k = ch - tch - ach; k > 0; --k) m &= m - 1;
            const int slot = __ffs(m) - 1;
            Pose q;
            q.p = g.saved[slot].x;
            q.job = g.saved[slot].y;
            score_atom(jobs.S(q), jobs.W(q), (size_t)q.p * n_mobile(jobs.S(q)), g.step[slot].w, lane);
            continue;
        }
        const bool tri = ch < tch;
        const int k = (tri ? ch : ch - tch) * 32 + lane, pre = tri ? tpre : apre;
        // the pose of item k: the last one whose first item is at or before it (a pose without
        // items shares its successor's first item)
        int w = 0;
        #pragma unroll 1
        for (int q = 1; q < Sh::poses; ++q)
            if (__shfl_sync(kFull, pre, q) <= k) w = q;
        const int first = __shfl_sync(kFull, pre, w);
        if (k < (tri ? T : A)) {
            Vor<Sh>& q = all[w].v;
            const int i = k - first + (tri ? 0 : q.nt);
            const uint32_t it = q.u.f.item[i];
            double v;
            if (tri) v = fan_triangle(q.vx[it & 0xffu], q.vx[(it >> 8) & 0xffu], q.vx[it >> 16], q.rado);
            else v = sph_arc(centre_of(q.pl[it & 0xffu]), q.vx[(it >> 8) & 0xffu], q.vx[(it >> 16) & 0xffu], q.rado);
            q.u.f.val[i] = v;
        }
    }
}

// Scores poses group step by group step: in each step every pose of the group takes its next atom (or
// goes on with its walk), the group evaluates the areas' items, and each pose saves its atom. A warp
// whose pose is through takes another (next_pose(&q): false when it gets none; warps without a pose
// help with the others' areas). Returns when no warp has one. all: the group's workspaces, for its
// first `poses` warps.
template <class Sh, int kSize, class Jobs, typename NextPose>
__device__ __forceinline__ void score_poses(const Jobs& jobs, int lane, PoseShared<Sh>* all, int poses, const Group<kSize>& g,
                                            uint8_t* hist, NextPose next_pose) {
    PoseShared<Sh>& ps = all[g.slot < poses ? g.slot : 0];
    Pose q;
    q.alive = false;
    bool more = g.slot < poses;          // poses may be left for this warp
    int to_score = -1;                   // the atom saved in the step before
    #pragma unroll 1
    for (;;) {
        while (!q.alive && more) {
            more = next_pose(q);
            if (more) q.alive = begin_pose(jobs, q, lane, ps, hist);
            to_score = -1;
        }
        int st = kAtomNone;
        if (q.alive) {
            st = step_pose(jobs, q, lane, ps, hist);
            if (st == kAtomNone) {
                __syncwarp();
                ++q.r;
            } else if (st == kAtomRetry) {
                q.alive = false;
                if (lane == 0) g.retry[atomicAdd(g.n_retry, 1)] = q.entry;
            } else if (st != kAtomOk && st != kAtomWalking) {
                const DevWork& W = jobs.W(q);
                q.alive = false;
                if (lane == 0) atomicAdd(&W.counters[st == kAtomHullFail ? 1 : 2], 1);
                if (st == kAtomHullFail) finish_failed(W, q.p, lane, FXE_POSE_POLYHEDRON_FAILED, (double)kPolyPenalty);
                else finish_failed(W, q.p, lane, FXE_POSE_CAPACITY, 0.0);
                count_faces(W, q, lane);
            }
        }
        const bool pending = q.alive && st == kAtomOk;
        if (lane == 0) {
            g.step[g.slot] = make_int4(pending ? ps.v.nt : 0, pending ? ps.v.na + ps.v.ne : 0, q.alive || more,
                                       q.alive ? to_score : -1);
            if (kScoreLater<kSize>) g.saved[g.slot] = make_int2(q.p, q.job);
        }
        to_score = -1;
        group_sync(g);
        if (!__any_sync(kFull, lane < g.size && g.step[lane].z != 0)) break;
        pooled_work(jobs, all, g, lane);
        group_sync(g);
        if (pending) {
            save_atom(jobs, q, lane, ps);
            ++q.r;
            if (kScoreLater<kSize> && q.r < n_mobile(jobs.S(q)))
                to_score = q.a;
            else
                score_atom(jobs.S(q), jobs.W(q), (size_t)q.p * n_mobile(jobs.S(q)), q.a, lane);
        }
        if (q.alive && !q.walking && q.r == n_mobile(jobs.S(q))) {
            __syncwarp();
            finish_scored(jobs.S(q), jobs.W(q), q.p, lane);
            count_faces(jobs.W(q), q, lane);
            q.alive = false;
        }
    }
    group_sync(g);
}

constexpr size_t kPoseSmem = sizeof(PoseShared<Compact>) * kWarps;
static_assert(kPoseSmem + 768 <= 227 * 1024, "sixteen poses per SM");
static_assert(sizeof(PoseShared<Large>) * Large::poses <= kPoseSmem && sizeof(PoseShared<Large>) <= kPoseSmem / 4,
              "the large shape's poses fit a block, and one fits the smallest group's share");

// Poses are handed out from a queue (order: n entries): the launch keeps only as many blocks as the
// SMs hold at once. The first `active` warps of each group score poses: their first ones are dealt,
// costliest first, over the launch's groups and back, so that each group gets costly and cheap ones;
// then each takes the next (`next`, zeroed before the launch) when it is through with one, at the
// group's next step. (When a block took sixteen poses at a time and waited for the last of them, 30,011
// poses of a screen took 19.4 ms; 13.8 so.)
template <int kSize, class Jobs>
__device__ __forceinline__ void score_queue(const Jobs& jobs, int n, int* next, const int* __restrict__ order, uint8_t* hist_all,
                                            int active) {
    extern __shared__ __align__(32) unsigned char smem[];
    __shared__ int4 step[kWarps];
    __shared__ int2 saved[kWarps];
    __shared__ int n_retry_of[kWarps], retry[2 * kWarps];
    const int lane = threadIdx.x & 31, warp = (int)(threadIdx.x >> 5);
    constexpr int groups = kWarps / kSize;
    const int group = warp / kSize;
    Group<kSize> g;
    g.slot = (warp + group * (4 / groups)) % kSize;   // (a group's first slots: each in another quarter of the SM)
    g.barrier = group + 1;
    g.step = step + group * kSize;
    g.saved = saved + group * kSize;
    g.n_retry = n_retry_of + group;
    g.retry = retry + 2 * group * kSize;
    unsigned char* const mem = smem + sizeof(PoseShared<Compact>) * kSize * group;
    constexpr int large = kSize * Large::poses / kWarps;
    // the warp's face history (hist_all: kHistStride bytes per warp of the launch), or null
    uint8_t* hist = hist_all ? hist_all + (size_t)(blockIdx.x * kWarps + warp) * kHistStride : nullptr;
    const int all_groups = groups * gridDim.x, at = group * gridDim.x + blockIdx.x;
    int dealt = g.slot * all_groups + (g.slot & 1 ? all_groups - 1 - at : at);
    bool empty = g.slot >= active;       // no more poses for this warp
    #pragma unroll 1
    for (;;) {
        if (g.slot == 0 && lane == 0) *g.n_retry = 0;
        group_sync(g);
        score_poses(jobs, lane, reinterpret_cast<PoseShared<Compact>*>(mem), kSize, g, hist, [&](Pose& q) {
            if (empty) return false;
            int e = dealt;
            dealt = -1;
            if (e < 0) {
                // (the list of poses to score again has room for those under way)
                if (lane == 0 && *(volatile int*)g.n_retry <= g.size) e = active * all_groups + atomicAdd(next, 1);
                e = __shfl_sync(kFull, e, 0);
                if (e < 0) return false;
                empty = e >= n;
                if (empty) return false;
            } else if (e >= n) {
                empty = true;
                return false;
            }
            q.entry = order[e];
            jobs.place(q);
            return true;
        });
        const int n_retry = *g.n_retry;
        if (n_retry == 0) break;
        int i = g.slot;
        score_poses(jobs, lane, reinterpret_cast<PoseShared<Large>*>(mem), large, g, hist, [&](Pose& q) {
            if (i >= n_retry) return false;
            q.entry = g.retry[i];
            i += large;
            jobs.place(q);
            return true;
        });
    }
}

template <int kSize>
__global__ void __launch_bounds__(kWarps * 32)
pose_kernel(const __grid_constant__ DevSystem S, const __grid_constant__ DevWork W, int n, int* next, uint8_t* hist_all, int active) {
    score_queue<kSize>(OneJob{S, W}, n, next, W.pose_order, hist_all, active);
}

template <int kSize>
__global__ void __launch_bounds__(kWarps * 32)
pose_kernel_jobs(const Job* __restrict__ jobs, int n_jobs, int n, int* next, const int* __restrict__ order, uint8_t* hist_all,
                 int active) {
    score_queue<kSize>(ManyJobs{jobs, n_jobs}, n, next, order, hist_all, active);
}

static int g_sms = 0, g_per_sm = 0;   // SMs, and blocks of pose_kernel one SM holds

size_t pose_hist_bytes() { return (size_t)g_sms * g_per_sm * kWarps * kHistStride; }

// Blocks a launch may run at once: as many as the device holds, no more than blocks_per_sm per
// SM when that is set (> 0; the autotuner's occupancy cap), no more than the face history holds
// (hist_bytes; 0, or less than a block's: no history).
static int max_blocks(size_t hist_bytes, int blocks_per_sm) {
    int b = g_sms * (blocks_per_sm > 0 && blocks_per_sm < g_per_sm ? blocks_per_sm : g_per_sm);
    if (hist_bytes >= kWarps * kHistStride) {
        const size_t cap = hist_bytes / (kWarps * kHistStride);
        if ((size_t)b > cap) b = (int)cap;
    }
    return b > 0 ? b : 1;
}

// A launch's blocks, its groups' size, and the warps of each group that take poses: all of them, or
// fewer when the launch's poses would not reach every block the device runs at once, so that they
// spread over more SMs (a pose's time is its chain of atoms, shorter with fewer warps sharing the
// SM's double-precision unit). Up to kSplitPoses poses per block two groups of eight warps share it: a
// pose waits for fewer others (500 poses of 24 atoms: 1,725 us, one group of sixteen 1,924); with the
// block full their code no longer meets in the instruction cache (2,000 poses of 63 atoms: 8.21 ms, one
// group 7.43).
constexpr int kSplitPoses = 4;
static void launch_shape(int n, size_t hist_bytes, int blocks_per_sm, int* blocks, int* group, int* active) {
    const int r = max_blocks(hist_bytes, blocks_per_sm);
    const int t = std::max(1, std::min((n + r - 1) / r, kWarps));
    *group = t <= kSplitPoses ? kWarps / 2 : kWarps;
    const int groups = kWarps / *group;
    *active = (t + groups - 1) / groups;
    const int per = *active * groups;
    *blocks = std::max(1, std::min((n + per - 1) / per, r));
}

int pose_max_blocks_per_sm() { return g_per_sm; }

// hist / hist_bytes: the launch's face history (reference face order), or null / 0;
// blocks_per_sm: occupancy cap (0: as many as fit).
void launch_poses(const DevSystem& S, const DevWork& W, int n, int* next, uint8_t* hist, size_t hist_bytes,
                  int blocks_per_sm, cudaStream_t st) {
    if (hist_bytes < kWarps * kHistStride) hist = nullptr;
    int blocks, group, active;
    launch_shape(n, hist ? hist_bytes : 0, blocks_per_sm, &blocks, &group, &active);
    cudaMemsetAsync(next, 0, sizeof(int), st);
    auto* kernel = group == kWarps ? pose_kernel<kWarps> : pose_kernel<kWarps / 2>;
    kernel<<<blocks, kWarps * 32, kPoseSmem, st>>>(S, W, n, next, hist, active);
}

void launch_poses_jobs(const Job* jobs, int n_jobs, int total, int* next, const int* order, uint8_t* hist,
                       size_t hist_bytes, int blocks_per_sm, cudaStream_t st) {
    if (hist_bytes < kWarps * kHistStride) hist = nullptr;
    int blocks, group, active;
    launch_shape(total, hist ? hist_bytes : 0, blocks_per_sm, &blocks, &group, &active);
    cudaMemsetAsync(next, 0, sizeof(int), st);
    auto* kernel = group == kWarps ? pose_kernel_jobs<kWarps> : pose_kernel_jobs<kWarps / 2>;
    kernel<<<blocks, kWarps * 32, kPoseSmem, st>>>(jobs, n_jobs, total, next, order, hist, active);
}

cudaError_t configure_voronoi() {
    for (const void* k : {(const void*)pose_kernel<kWarps>, (const void*)pose_kernel<kWarps / 2>,
                          (const void*)pose_kernel_jobs<kWarps>, (const void*)pose_kernel_jobs<kWarps / 2>}) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPoseSmem);
        if (e != cudaSuccess) return e;
    }
    cudaError_t e;
    int dev = 0, sms = 0, per_sm = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pose_kernel<kWarps>, kWarps * 32, kPoseSmem)) != cudaSuccess) return e;
    g_sms = sms;
    g_per_sm = per_sm > 0 ? per_sm : 1;
    return cudaSuccess;
}

}  // namespace f64
}  // namespace fxe
