// Narrowphase: MPR with a search per lane (NarrowPhase.cs:98-347), EPA with the polytope in shared
// memory and a warp per deep pair (NarrowPhase.cs:39-95, ConvexPolytope.cs), the triangle-edge
// filter (TriangleEdgeCollisionFilter.cs:243-420) and the one-shot manifold
// (CollisionManifold.cs:393-566) with a thread, or in small steps a warp, per record; colliding
// pairs append one record (key, normal, up to four point pairs) to the compacted contact stream.
//
// In the warp-per-pair stages the lanes hold identical copies of the MPR state; point-cloud
// support maps, the EPA face scans (closest face, visibility, horizon), the FP64 face geometry
// (four lanes per face) and the manifold's segment intersections are split across lanes.  EPA
// keeps the reference's FP64 face data and polytope capacity (128 vertices, 256 faces); side
// tests run an FP32 filter, the reference's FP64 filter, then exact expansions.  Running out
// of capacity ends EPA with the MPR result, the reference's behaviour on any EPA failure.
//
// The MPR follows code the reference adapted from XenoCollide (zlib license, (c) 2007-2014
// Gary Snethen, http://xenocollide.com): provided 'as-is', without any express or implied
// warranty; altered source versions must be plainly marked as such; this notice may not
// be removed or altered from any source distribution.
#include "jg_shapes.cuh"

namespace {

constexpr unsigned FULL = 0xffffffffu;

struct MV { v3 V, A, B; };

// MinkowskiDifference.Support (MinkowskiDifference.cs:57-69), by one thread.
__device__ __forceinline__ void mk_support_lane(const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb, v3 d, MV& v) {
    v.A = support_lane(sa, d);
    v.B = support_lane(sb, rotate_inv(-d, qb));
    v.B = rotate(v.B, qb);
    v.B = v.B + pb;
    v.V = v.A - v.B;
}
// The same by the 32 lanes of a warp together (point clouds split across lanes).
// (One copy of the support maps for both shapes, and a call: EPA, MPR and the manifold of a warp
// kernel share an instruction cache that they fill.)
__device__ __noinline__ void mk_support(const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb, v3 d, MV& v) {
    const v3 db = rotate_inv(-d, qb);
    v3 p[2];
#pragma unroll 1
    for (int k = 0; k < 2; k++) p[k] = support(k ? sb : sa, k ? db : d);
    v.A = p[0];
    v.B = rotate(p[1], qb);
    v.B = v.B + pb;
    v.V = v.A - v.B;
}
__device__ __forceinline__ void mk_center(const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb, MV& c) {
    c.A = shape_center(sa);
    c.B = rotate(shape_center(sb), qb);
    c.B = pb + c.B;
    c.V = c.A - c.B;
}

// ---- exact arithmetic (double expansions), used only on unresolved EPA predicates -------
struct Exp {
    __device__ __noinline__ static int diff(double a, double b, double* o) {
        double v = a - b, vb = a - v;
        double res = (a - (v + vb)) + (vb - b);
        int n = 0;
        if (res != 0) o[n++] = res;
        if (v != 0) o[n++] = v;
        return n;
    }
    __device__ __noinline__ static int grow(double* e, int len, double value) {
        int cnt = 0;
#pragma unroll 1
        for (int i = 0; i < len; i++) {
            double part = e[i];
            double sum = value + part;
            double vp = sum - value;
            double res = (value - (sum - vp)) + (part - vp);
            if (res != 0) e[cnt++] = res;
            value = sum;
        }
        if (value != 0) e[cnt++] = value;
        return cnt;
    }
    __device__ __noinline__ static int addp(double* r, int len, const double* a, int na, const double* b, int nb, bool neg, int cap) {
#pragma unroll 1
        for (int i = 0; i < na; i++)
#pragma unroll 1
            for (int j = 0; j < nb; j++) {
                double x = a[i], y = b[j];
                double p = __dmul_rn(x, y);
                double res = fma(x, y, -p);
                if (neg) { p = -p; res = -res; }
                if (res != 0 && len < cap) len = grow(r, len, res);
                if (p != 0 && len < cap) len = grow(r, len, p);
            }
        return len;
    }
    __device__ __noinline__ static int crossterm(const double* a, int na, const double* b, int nb, const double* c, int nc,
                                    const double* d, int nd, double* o) {
        int len = addp(o, 0, a, na, b, nb, false, 16);
        return addp(o, len, c, nc, d, nd, true, 16);
    }
    // ExpansionArithmetic.Side (ExactArithmetic/ExpansionArithmetic.cs:20-41)
    __device__ __noinline__ static int side(v3 a, v3 b, v3 c, v3 p) {
        double ux[2], uy[2], uz[2], vx[2], vy[2], vz[2], dx[2], dy[2], dz[2];
        int nx = diff(a.x, b.x, ux), ny = diff(a.y, b.y, uy), nz = diff(a.z, b.z, uz);
        int mx = diff(a.x, c.x, vx), my = diff(a.y, c.y, vy), mz = diff(a.z, c.z, vz);
        int px = diff(p.x, a.x, dx), py = diff(p.y, a.y, dy), pz = diff(p.z, a.z, dz);
        double cr[16], det[192];
        int len = crossterm(uy, ny, vz, mz, uz, nz, vy, my, cr);
        int cnt = addp(det, 0, cr, len, dx, px, false, 192);
        len = crossterm(uz, nz, vx, mx, ux, nx, vz, mz, cr);
        cnt = addp(det, cnt, cr, len, dy, py, false, 192);
        len = crossterm(ux, nx, vy, my, uy, ny, vx, mx, cr);
        cnt = addp(det, cnt, cr, len, dz, pz, false, 192);
        if (cnt == 0) return 0;
        double t = det[cnt - 1];
        return t > 0 ? 1 : (t < 0 ? -1 : 0);
    }
    // ExpansionArithmetic.Normal (ExpansionArithmetic.cs:43-55): each component of
    // (a-b) x (a-c) as an exact expansion, summed from the least significant part up
    __device__ __noinline__ static void normal(v3 a, v3 b, v3 c, double& x, double& y, double& z) {
        double ux[2], uy[2], uz[2], vx[2], vy[2], vz[2], cr[16];
        int nx = diff(a.x, b.x, ux), ny = diff(a.y, b.y, uy), nz = diff(a.z, b.z, uz);
        int mx = diff(a.x, c.x, vx), my = diff(a.y, c.y, vy), mz = diff(a.z, c.z, vz);
        double r[3];
        int len = crossterm(uy, ny, vz, mz, uz, nz, vy, my, cr);
        double s = 0; for (int i = 0; i < len; i++) s += cr[i]; r[0] = s;
        len = crossterm(uz, nz, vx, mx, ux, nx, vz, mz, cr);
        s = 0; for (int i = 0; i < len; i++) s += cr[i]; r[1] = s;
        len = crossterm(ux, nx, vy, my, uy, ny, vx, mx, cr);
        s = 0; for (int i = 0; i < len; i++) s += cr[i]; r[2] = s;
        x = r[0]; y = r[1]; z = r[2];
    }
};

// PlaneFilter in double (ExactArithmetic/PlaneFilter.cs:29-70); the FP32 filter below
// tries first.
__device__ __noinline__ bool dfilter_side(v3 a, v3 b, v3 c, v3 p, int& sign) {
    const double EF = 16 * 1.1102230246251565e-16;
    double ux = (double)a.x - b.x, uy = (double)a.y - b.y, uz = (double)a.z - b.z;
    double vx = (double)a.x - c.x, vy = (double)a.y - c.y, vz = (double)a.z - c.z;
    double yz = uy * vz, zy = uz * vy, zx = uz * vx, xz = ux * vz, xy = ux * vy, yx = uy * vx;
    double nx = yz - zy, ny = zx - xz, nz = xy - yx;
    double ex = EF * (fabs(yz) + fabs(zy)), ey = EF * (fabs(zx) + fabs(xz)), ez = EF * (fabs(xy) + fabs(yx));
    double dx = (double)p.x - a.x, dy = (double)p.y - a.y, dz = (double)p.z - a.z;
    double x = nx * dx, y = ny * dy, z = nz * dz;
    double value = (x + y) + z;
    double round = EF * ((fabs(x) + fabs(y)) + fabs(z));
    double coef = (ex * fabs(dx) + ey * fabs(dy)) + ez * fabs(dz);
    if (fabs(value) <= round + 2 * coef) return false;
    sign = value > 0 ? 1 : -1;
    return true;
}

// FP32 version of the same filter: identical bound structure with u = 2^-24.
__device__ __forceinline__ bool ffilter_side(v3 a, v3 b, v3 c, v3 p, int& sign) {
    const float EF = 16.0f * 5.9604645e-08f;
    float ux = a.x - b.x, uy = a.y - b.y, uz = a.z - b.z;
    float vx = a.x - c.x, vy = a.y - c.y, vz = a.z - c.z;
    float yz = uy * vz, zy = uz * vy, zx = uz * vx, xz = ux * vz, xy = ux * vy, yx = uy * vx;
    float nx = yz - zy, ny = zx - xz, nz = xy - yx;
    float ex = EF * (fabsf(yz) + fabsf(zy)), ey = EF * (fabsf(zx) + fabsf(xz)), ez = EF * (fabsf(xy) + fabsf(yx));
    float dx = p.x - a.x, dy = p.y - a.y, dz = p.z - a.z;
    float x = nx * dx, y = ny * dy, z = nz * dz;
    float value = (x + y) + z;
    float round = EF * ((fabsf(x) + fabsf(y)) + fabsf(z));
    float coef = (ex * fabsf(dx) + ey * fabsf(dy)) + ez * fabsf(dz);
    // the difference of two float coordinates is inexact in float: widen the bound for
    // the extra rounding of the displacement (covered by the factor 4)
    if (fabsf(value) <= 4.0f * (round + 2.0f * coef) || !isfinite(value)) return false;
    sign = value > 0 ? 1 : -1;
    return true;
}

// Per-warp EPA polytope, in dynamic shared memory.  Vertices and faces at the reference's
// capacity (ConvexPolytope.cs:53-54).  Each face keeps what the reference's Triangle and
// FaceData keep for the search: the squared distance of its closest point in FP64 (the
// closest-face choice compares these), and the closest point and its squared distance
// rounded to FP32 (the support direction and the convergence test).  Everything else a
// face has in FP64 (plane normal, barycentric coordinates) is a deterministic function of
// its corners and is recomputed, bit for bit, where it is needed: for the rare search
// along a face normal and for the witness points of the final face.
struct EpaSmem {
    float4 vV[JG_EPA_MAXV], vA[JG_EPA_MAXV], vB[JG_EPA_MAXV];
    double fd[JG_EPA_MAXT];     // squared distance of the closest point (FP64)
    float4 fc[JG_EPA_MAXT];     // closest point xyz, squared distance (both rounded to FP32)
    uchar4 fi[JG_EPA_MAXT];     // a, b, c, flags (1: facing the origin, 2: corners swapped)
    unsigned char ea[3 * JG_EPA_MAXT], eb[3 * JG_EPA_MAXT];
    unsigned lit[JG_EPA_MAXT / 32];
    int nv, nt, ne, enclosed;
    // manifold scratch
    float4 mA[12], mB[12];
    float4 left[6], right[6];
};
#define EPA_FACING 1
#define EPA_SWAPPED 2

enum { ADDED = 0, NO_HORIZON = 1, DEGENERATE = 2, CAPACITY = 3, NUMERICAL = 4 };

struct NpStats { int exact; };

// ConvexPolytope.Side (ConvexPolytope.cs:321-327): orientation of point p relative to face
// (a,b,c).  Every filter that answers is certified, so the sign is the exact one whichever
// answers: the FP32 filter first, then the reference's FP64 filter, then exact expansions.
__device__ __forceinline__ int side_pt(v3 a, v3 b, v3 c, v3 p, NpStats& st) {
    if (p == a || p == b || p == c) return 0;
    int s;
    if (ffilter_side(a, b, c, p, s)) return s;
    st.exact++;
    if (dfilter_side(a, b, c, p, s)) return s;
    return Exp::side(a, b, c, p);
}

// PlaneFilter.IsSafe (ExactArithmetic/PlaneFilter.cs:73-77) for float coordinates.
__device__ __forceinline__ bool safe_coord(float v) {
    float a = fabsf(v);
    return v == 0.f || (a >= 1e-30f && a <= 1e30f);
}
__device__ __forceinline__ bool is_safe(v3 p) { return safe_coord(p.x) && safe_coord(p.y) && safe_coord(p.z); }

// ---- FP64 face geometry, four lanes per face ----------------------------------------------
// An FP64 instruction holds its warp scheduler for 64 cycles on this part, whatever the number
// of active lanes (measured, add, multiply and FMA alike; a division takes nine of them), and a
// face needs about 250 when one lane evaluates it.  Here lane c of a group of four holds
// component c of the vectors (the fourth repeats the first), so that an operation on three
// components is one instruction, and the sums and quotients of a face that do not depend on
// each other take one lane each: about 60 instructions for up to eight faces, with what only
// signs or orders are needed of decided without a division.  Every value that is used comes
// from the reference's operations in their order, so it is that of the one-lane form bit for bit.
// EPA of a settled 100k-body pile (7.2k deep pairs) 1374 -> 597 us, of a few hundred pairs that leave
// only the latency of the longest one 545 -> 249 (as a launch of its own; k_deep has more to do).
// Signs and maxima of finite doubles are decided on their bit patterns (integer pipe).
__device__ __forceinline__ double grp(double x, int src) { return __shfl_sync(FULL, x, src, 4); }
__device__ __forceinline__ bool x_nonzero(double x) { return (__double_as_longlong(x) << 1) != 0; }
__device__ __forceinline__ bool d_lt0(double x) { return __double_as_longlong(x) < 0 && x_nonzero(x); }
__device__ __forceinline__ bool d_ge0(double x) { return !d_lt0(x); }
__device__ __forceinline__ bool d_finite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ long long d_absbits(double x) { return __double_as_longlong(x) & 0x7fffffffffffffffll; }

__device__ __forceinline__ int d_exp(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// A float that is zero or normal, widened on the integer pipe.
__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f), m = u & 0x7fffffffu;
    return __hiloint2double((int)((u & 0x80000000u) | (m ? (m >> 3) + (896u << 20) : 0u)), (int)(u << 29));
}

// (x0 + x1) + x2 of up to four vectors at once: lane k of the group returns the sum of the
// components of the k-th argument, in the order of the reference's dot products.
__device__ __forceinline__ double grp_sums(int c, double p, double q, double r, double s) {
    const double p0 = grp(p, 0), p1 = grp(p, 1), p2 = grp(p, 2);
    const double q0 = grp(q, 0), q1 = grp(q, 1), q2 = grp(q, 2);
    const double r0 = grp(r, 0), r1 = grp(r, 1), r2 = grp(r, 2);
    const double s0 = grp(s, 0), s1 = grp(s, 1), s2 = grp(s, 2);
    const double x0 = c == 0 ? p0 : (c == 1 ? q0 : (c == 2 ? r0 : s0));
    const double x1 = c == 0 ? p1 : (c == 1 ? q1 : (c == 2 ? r1 : s1));
    const double x2 = c == 0 ? p2 : (c == 1 ? q2 : (c == 2 ? r2 : s2));
    return (x0 + x1) + x2;
}

// The FP64 geometry of a face (ConvexPolytope.CreateTriangle, ConvexPolytope.cs:267-318, and
// CalcBarycentric, :328-395) from its corners in creation order i0, i1, i2; `swapped` when the
// orientation test exchanged the first two.  The raw normal is the FP64 plane filter's cross
// product of the creation order (PlaneFilter.cs:29-45), negated on a swap, and replaced by the
// exact expansion normal of the final order when the filter calls it unreliable
// (PlaneFilter.cs:24-27).  sn, cl: this lane's component; bc: all three weights; ok is false on
// a numerical failure.  Called by the whole warp; the coordinates are safe_coord's, so that no
// value up to the quotients overflows.
struct FaceGeo { double sn, cl, d2; double bx, by, bz; bool ok; };
__device__ __noinline__ FaceGeo face_geo(const EpaSmem& E, int i0, int i1, int i2, bool swapped, bool weights, bool count, NpStats& st) {
    const double EF = 16 * 1.1102230246251565e-16;
    const int c = threadIdx.x & 3, k = c == 3 ? 0 : c, k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
    const double p0 = widen((&E.vV[i0].x)[k]), p1 = widen((&E.vV[i1].x)[k]), p2 = widen((&E.vV[i2].x)[k]);
    FaceGeo g;
    const double u = p0 - p1, v = p0 - p2;
    const double a = swapped ? p1 : p0, b = swapped ? p0 : p1;
    double raw;
    long long rmax;
    bool exact;
    {
        const double s = grp(u, k1) * grp(v, k2), t = grp(u, k2) * grp(v, k1);
        raw = s - t;
        if (swapped) raw = -raw;
        const long long m = d_absbits(raw), e = max(d_absbits(s), d_absbits(t));
        rmax = max(max(__shfl_sync(FULL, m, 0, 4), __shfl_sync(FULL, m, 1, 4)), __shfl_sync(FULL, m, 2, 4));
        const long long big = max(max(__shfl_sync(FULL, e, 0, 4), __shfl_sync(FULL, e, 1, 4)), __shfl_sync(FULL, e, 2, 4));
        // unreliable unless the largest component exceeds 2^20 times the largest error bound, which
        // is 2^-49 (|s| + |t|): decided by 2^-28 max(|s|, |t|) where that is enough
        exact = !(rmax > max(big - (28ll << 52), 0ll));
        if (__any_sync(FULL, exact)) {
            const long long r = d_absbits(EF * (fabs(s) + fabs(t)));
            const long long emax = max(max(__shfl_sync(FULL, r, 0, 4), __shfl_sync(FULL, r, 1, 4)), __shfl_sync(FULL, r, 2, 4));
            exact = !(rmax > (emax ? emax + (20ll << 52) : 0));
        }
    }
    if (__any_sync(FULL, exact)) {
        double x = 0, y = 0, z = 0;
        if (exact) {
            if (count) st.exact++;
            if (c == 0) {
                const int ia = swapped ? i1 : i0, ib = swapped ? i0 : i1;
                Exp::normal(mk3(E.vV[ia]), mk3(E.vV[ib]), mk3(E.vV[i2]), x, y, z);
            }
        }
        __syncwarp();
        x = grp(x, 0); y = grp(y, 0); z = grp(z, 0);
        if (exact) {
            raw = k == 0 ? x : (k == 1 ? y : z);
            rmax = max(max(d_absbits(x), d_absbits(y)), d_absbits(z));
        }
    }
    const double ns = __longlong_as_double(rmax);
    g.ok = rmax > 0 && d_finite(ns);
    const double sn = raw / ns;
    g.sn = sn;
    const double nn = sn * sn;
    const double nsq = (grp(nn, 0) + grp(nn, 1)) + grp(nn, 2);
    const double uf = swapped && x_nonzero(u) ? -u : u, vf = a - p2;  // a - b and a - c of the final order
    const double a1 = grp(a, k1), a2 = grp(a, k2), uf1 = grp(uf, k1), uf2 = grp(uf, k2), vf1 = grp(vf, k1), vf2 = grp(vf, k2);
    // lanes 0 to 2: gamma times nsq ns, beta times nsq ns, the plane's distance times nsq
    const double num = grp_sums(c, (uf1 * a2 - uf2 * a1) * sn, (a1 * vf2 - a2 * vf1) * sn, sn * a, 0.0);
    const double n0 = grp(num, 0), n1 = grp(num, 1);
    // The weights' signs decide what is closest.  Those of gamma and beta are the numerators'
    // (coordinates and ns in this range leave no underflow); alpha = 1 - gamma - beta has that of
    // ns nsq - (n0 + n1) if that is not within 2^-40 of the terms, where the roundings could decide.
    // So the two divisions that give the weights themselves are left to the calls that ask for
    // them, and to those cases.
    const double den = ns * nsq, rest = den - (n0 + n1);
    const int e = d_exp(ns);
    const bool sure = e > 1023 - 200 && e < 1023 + 200 && d_exp(rest) + 40 > max(d_exp(den), max(d_exp(n0), d_exp(n1)));
    double gamma = n0, beta = n1, alpha = rest;  // (or positive multiples of them)
    if (__any_sync(FULL, weights || !sure)) {
        const double q2 = (num / nsq) / ns;
        gamma = grp(q2, 0);
        beta = grp(q2, 1);
        alpha = 1.0 - gamma - beta;
    }
    const bool c1 = d_ge0(alpha) && d_lt0(beta), c2 = !c1 && d_ge0(beta) && d_lt0(gamma),
               c3 = !c1 && !c2 && d_ge0(gamma) && d_lt0(alpha);
    const bool clamped = c1 || c2 || c3, some = __any_sync(FULL, clamped);
    double top = grp(num, 2), bottom = nsq;
    bool first = false;
    if (some) {
        // the three cases differ in the corner P, the edge Q tried first and the edge R taken
        // otherwise: (a, u, v), (b, w, u), (c, v, w)
        const double w = b - p2;
        const double P = c1 ? a : (c2 ? b : p2), Q = c1 ? uf : (c2 ? w : vf), R = c1 ? vf : (c2 ? uf : w);
        const double s = grp_sums(c, P * Q, P * R, Q * Q, R * R);
        double t = grp(s, 0), o = grp(s, 1);
        if (c3) t = -t;
        if (!c1) o = -o;
        first = d_lt0(c1 ? gamma : (c2 ? alpha : beta)) && !d_lt0(t) && x_nonzero(t);
        const double qq = grp(s, 2), rr = grp(s, 3);
        if (clamped) { top = first ? t : o; bottom = first ? qq : rr; }
    }
    double r = top / bottom;  // the plane's distance, or the point's place on its edge
    g.cl = sn * r;
    if (some) {
        const long long one = 0x3ff0000000000000ll, rb = __double_as_longlong(r);
        // to [0, 1]; 0/0 of the second edge goes through as it is unless it counts as negative
        if (first ? rb > one : rb > one && rb <= 0x7ff0000000000000ll) r = 1.0;
        else if (!first && d_lt0(r)) r = 0.0;
        const double q = 1.0 - r;
        if (clamped) {
            if (c1) { alpha = q; beta = first ? r : 0.0; gamma = first ? 0.0 : r; }
            else if (c2) { beta = q; gamma = first ? r : 0.0; alpha = first ? 0.0 : r; }
            else { gamma = q; alpha = first ? r : 0.0; beta = first ? 0.0 : r; }
            g.cl = (a * alpha + b * beta) + p2 * gamma;
        }
        __syncwarp();
    }
    const double cc = g.cl * g.cl;
    g.d2 = (grp(cc, 0) + grp(cc, 1)) + grp(cc, 2);
    g.bx = alpha; g.by = beta; g.bz = gamma;
    g.ok = g.ok && d_finite(g.cl) && d_finite(alpha) && d_finite(beta) && d_finite(gamma) && d_finite(g.d2);
    const unsigned bad = __ballot_sync(FULL, !g.ok);
    g.ok = ((bad >> (threadIdx.x & 28)) & 15u) == 0;
    return g;
}

// The geometry of a stored face, by every group of the warp alike.
__device__ __forceinline__ FaceGeo face_geo_of(const EpaSmem& E, int f, NpStats& st) {
    uchar4 t = E.fi[f];
    bool sw = (t.w & EPA_SWAPPED) != 0;
    return face_geo(E, sw ? t.y : t.x, sw ? t.x : t.y, t.z, sw, true, true, st);
}

// The FP32 normal of a face and its squared length (Triangle.Normal / NormalSq).
__device__ __forceinline__ float4 face_normal32(const FaceGeo& g) {
    const float s = (float)g.sn;
    v3 n = mk3(__shfl_sync(FULL, s, 0), __shfl_sync(FULL, s, 1), __shfl_sync(FULL, s, 2));
    return f4(n, len2(n));
}

// ConvexPolytope.CreateTriangle (ConvexPolytope.cs:267-318), four lanes per face, eight faces
// per call; `live` is false for the groups beyond the last face (they repeat another face's
// arithmetic and store nothing).  Called by the whole warp.
__device__ __noinline__ int create_tris(EpaSmem& E, int a, int b, int c, int slot, bool live, NpStats& st) {
    const int comp = threadIdx.x & 3;
    NpStats mine;
    mine.exact = 0;
    v3 va = mk3(E.vV[a]), vb = mk3(E.vV[b]), vc = mk3(E.vV[c]);
    const int i0 = a, i1 = b;
    int orient = 0;
#pragma unroll 1
    for (int i = 0; i < 4 && orient == 0; i++) {
        if (i == a || i == b || i == c) continue;
        orient = -side_pt(va, vb, vc, mk3(E.vV[i]), mine);
    }
    const bool swapped = orient < 0;
    if (swapped) { int t = a; a = b; b = t; v3 tv = va; va = vb; vb = tv; }
    bool facing = orient != 0 && side_pt(va, vb, vc, mk3(0.f), mine) <= 0;
    __syncwarp();
    const bool counts = live && comp == 0;  // one lane counts for its face
    if (counts) st.exact += mine.exact;
    const FaceGeo g = face_geo(E, i0, i1, c, swapped, false, counts && orient != 0, st);
    const float out = (float)(comp == 3 ? g.d2 : g.cl);
    const unsigned bad = __ballot_sync(FULL, !isfinite(out));
    int r = ADDED;
    if (orient == 0) r = DEGENERATE;
    else if (!g.ok || ((bad >> (threadIdx.x & 28)) & 15u)) r = NUMERICAL;
    if (live && r == ADDED) {
        (&E.fc[slot].x)[comp] = out;
        if (comp == 0) {
            E.fi[slot] = make_uchar4((unsigned char)a, (unsigned char)b, (unsigned char)c,
                                     (unsigned char)((facing ? EPA_FACING : 0) | (swapped ? EPA_SWAPPED : 0)));
            E.fd[slot] = g.d2;
        }
    }
    return live ? r : ADDED;
}

// ConvexPolytope.InitTetrahedron (ConvexPolytope.cs:113-132)
__device__ bool epa_init(EpaSmem& E, NpStats& st) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) { E.nv = 4; E.nt = 0; E.enclosed = 0; }
    __syncwarp();
    bool safe = true;
    for (int i = 0; i < 4; i++) safe = safe && is_safe(mk3(E.vV[i]));
    if (!safe) return false;
    const int idx[12] = {0, 2, 1, 0, 1, 3, 0, 3, 2, 1, 2, 3};
    const int f = min(lane >> 2, 3);
    int r = create_tris(E, idx[3 * f], idx[3 * f + 1], idx[3 * f + 2], f, lane < 16, st);
    bool ok = __all_sync(FULL, r == ADDED);
    __syncwarp();
    if (ok && lane == 0) E.nt = 4;
    __syncwarp();
    return ok;
}

// ConvexPolytope.GetClosestTriangle (ConvexPolytope.cs:147-166): the smallest FP64 squared
// distance, the first such face on a tie.
__device__ int epa_closest(EpaSmem& E) {
    const int lane = threadIdx.x & 31;
    // squared distances are finite and not negative: they order as their bit patterns
    unsigned long long best = ~0ull;
    int bi = 0x7fffffff;
    bool notfacing = false;
    int nt = E.nt;
    for (int i = lane; i < nt; i += 32) {
        const unsigned long long d = (unsigned long long)__double_as_longlong(E.fd[i]);
        if (d < best) { best = d; bi = i; }
        if (!(E.fi[i].w & EPA_FACING)) notfacing = true;
    }
    const unsigned hi = __reduce_min_sync(FULL, (unsigned)(best >> 32));
    const unsigned lo = __reduce_min_sync(FULL, (unsigned)(best >> 32) == hi ? (unsigned)best : 0xffffffffu);
    bi = (int)__reduce_min_sync(FULL, best == (((unsigned long long)hi << 32) | lo) ? (unsigned)bi : 0x7fffffffu);
    bool any_nf = __any_sync(FULL, notfacing);
    bool skip = E.enclosed != 0;
    __syncwarp();
    if (lane == 0) E.enclosed = any_nf ? (skip ? 1 : 0) : 1;
    __syncwarp();
    if (bi == 0x7fffffff) bi = 0;
    return bi;
}

// ConvexPolytope.AddVertexDetailed (ConvexPolytope.cs:199-265)
__device__ __noinline__ int epa_add(EpaSmem& E, const MV& v, NpStats& st) {
    const int lane = threadIdx.x & 31;
    if (E.nt == 0 || !is_safe(v.V)) return NUMERICAL;
    int nv = E.nv;
    if (nv == JG_EPA_MAXV) return CAPACITY;
    if (lane == 0) { E.vV[nv] = f4(v.V, 0.f); E.vA[nv] = f4(v.A, 0.f); E.vB[nv] = f4(v.B, 0.f); }
    __syncwarp();
    int nt = E.nt;
    // visibility of every face, lanes in parallel
#pragma unroll 1
    for (int base = 0; base < nt; base += 32) {
        int i = base + lane;
        bool lit = false;
        if (i < nt) {
            uchar4 f = E.fi[i];
            lit = side_pt(mk3(E.vV[f.x]), mk3(E.vV[f.y]), mk3(E.vV[f.z]), v.V, st) > 0;
        }
        unsigned m = __ballot_sync(FULL, lit);
        if (lane == 0) E.lit[base >> 5] = m;
    }
    __syncwarp();
    // Horizon edges in the reference's order (faces from last to first; an edge met twice
    // leaves the list, the last edge taking its place).  The list lives in registers, edge e in
    // lane e, so that a search is one vote; a list that outgrows the warp is rebuilt by one lane
    // in shared memory.
    int ne = 0, edge = 0;
    bool wide = false;
#pragma unroll 1
    for (int word = (nt - 1) >> 5; word >= 0 && !wide; word--) {
#pragma unroll 1
        for (unsigned m = E.lit[word]; m && !wide;) {
            const int bit = 31 - __clz(m);
            m ^= 1u << bit;
            const uchar4 f = E.fi[word * 32 + bit];
            const int cs[4] = {f.x, f.y, f.z, f.x};
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const int key = cs[k] | (cs[k + 1] << 8), rev = cs[k + 1] | (cs[k] << 8);
                const unsigned hit = __ballot_sync(FULL, lane < ne && (edge == key || edge == rev));
                if (hit) {
                    --ne;
                    const int last = __shfl_sync(FULL, edge, ne);
                    if (lane == 31 - __clz(hit)) edge = last;
                } else {
                    if (ne == 32) { wide = true; break; }
                    if (lane == ne) edge = key;
                    ne++;
                }
            }
        }
    }
    if (wide) {
        if (lane == 0) {
            int n = 0;
#pragma unroll 1
            for (int index = nt; index-- > 0;) {
                if (!((E.lit[index >> 5] >> (index & 31)) & 1u)) continue;
                uchar4 f = E.fi[index];
                unsigned char cs[3] = {f.x, f.y, f.z};
#pragma unroll 1
                for (int k = 0; k < 3; k++) {
                    unsigned char A = cs[k], B = cs[(k + 1) % 3];
                    bool added = true;
#pragma unroll 1
                    for (int e = n; e-- > 0;) {
                        bool match = (E.ea[e] == A && E.eb[e] == B) || (E.ea[e] == B && E.eb[e] == A);
                        if (!match) continue;
                        --n;
                        E.ea[e] = E.ea[n]; E.eb[e] = E.eb[n];
                        added = false;
                        break;
                    }
                    if (added && n < 3 * JG_EPA_MAXT) { E.ea[n] = A; E.eb[n] = B; n++; }
                }
            }
            E.ne = n;
        }
        __syncwarp();
        ne = E.ne;
    }
    if (ne == 0) return NO_HORIZON;
    int nlit = 0;
#pragma unroll 1
    for (int k = 0; k < (nt + 31) / 32; k++) nlit += __popc(E.lit[k] & (k * 32 + 32 <= nt ? 0xffffffffu : ((1u << (nt & 31)) - 1u)));
    if (nt - nlit + ne > JG_EPA_MAXT) return CAPACITY;
    // order-preserving compaction of the surviving faces
    int surv = 0;
#pragma unroll 1
    for (int base = 0; base < nt; base += 32) {
        int i = base + lane;
        bool keep = i < nt && !((E.lit[i >> 5] >> (i & 31)) & 1u);
        uchar4 fi; float4 fc; double fd;
        if (keep) { fi = E.fi[i]; fc = E.fc[i]; fd = E.fd[i]; }
        unsigned m = __ballot_sync(FULL, keep);
        int dst = surv + __popc(m & ((1u << lane) - 1u));
        __syncwarp();
        if (keep) { E.fi[dst] = fi; E.fc[dst] = fc; E.fd[dst] = fd; }
        surv += __popc(m);
        __syncwarp();
    }
    // the new fan, eight faces at a time
    int res = ADDED;
#pragma unroll 1
    for (int base = 0; base < ne; base += 8) {
        const int e = min(base + (lane >> 2), ne - 1);
        int ea, eb;
        if (wide) { ea = E.ea[e]; eb = E.eb[e]; }
        else { const int k = __shfl_sync(FULL, edge, e); ea = k & 255; eb = k >> 8; }
        const int r = create_tris(E, ea, eb, nv, surv + e, base + (lane >> 2) < ne, st);
        const unsigned worst = __reduce_min_sync(FULL, r == ADDED ? 0x7fffffffu : (unsigned)r);
        if (worst != 0x7fffffffu && res == ADDED) res = (int)worst;
    }
    __syncwarp();
    if (res != ADDED) {
        if (lane == 0) { E.nt = 0; E.enclosed = 0; }
        __syncwarp();
        return res;
    }
    if (lane == 0) { E.nt = surv + ne; E.nv = nv + 1; }
    __syncwarp();
    return ADDED;
}

// MprEpaSolver.SolveMprEpa (NarrowPhase.cs:39-95).  Seed vertices are in E.v*[0..3].
__device__ __noinline__ bool solve_epa(EpaSmem& E, const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb,
                          v3& p1, v3& p2, v3& n, float& pen, NpStats& st) {
    const float eps = 1e-5f;
    const int maxIter = 85;
    if (!epa_init(E, st)) return false;
    int iter = 0;
    int ci = 0;
    while (++iter < maxIter) {
        ci = epa_closest(E);
        float4 fc = E.fc[ci];
        v3 sd = mk3(fc), cl = mk3(fc);
        float sdsq = fc.w;
        if (!E.enclosed) sd = -sd;
        if (fc.w < 1e-16f) {
            // search along the face normal (Triangle.Normal / NormalSq)
            const float4 fn = face_normal32(face_geo_of(E, ci, st));
            sd = mk3(fn); sdsq = fn.w;
        }
        MV v;
        mk_support(sa, sb, qb, pb, sd, v);
        float delta = dot(cl - v.V, sd);
        if (delta * delta <= eps * eps * sdsq) goto converged;
        {
            int r = epa_add(E, v, st);
            if (r == NO_HORIZON) goto converged;
            if (r != ADDED) return false;
        }
    }
    return false;
converged:
    if (!E.enclosed) return false;
    {
        // ConvexPolytope.CalculatePoints (ConvexPolytope.cs:169-185): the FP64 barycentric
        // combination of the corners' support points, rounded to FP32
        uchar4 f = E.fi[ci];
        const FaceGeo g = face_geo_of(E, ci, st);
        // lanes 0-2: the components of A's point, lanes 4-6: of B's
        const int lane = threadIdx.x & 31, k = (lane & 3) == 3 ? 0 : lane & 3;
        const float4* P = (lane & 4) ? E.vB : E.vA;
        const float pt = (float)(((double)(&P[f.x].x)[k] * g.bx + (double)(&P[f.y].x)[k] * g.by) + (double)(&P[f.z].x)[k] * g.bz);
        p1 = mk3(__shfl_sync(FULL, pt, 0), __shfl_sync(FULL, pt, 1), __shfl_sync(FULL, pt, 2));
        p2 = mk3(__shfl_sync(FULL, pt, 4), __shfl_sync(FULL, pt, 5), __shfl_sync(FULL, pt, 6));
        float4 fn = face_normal32(g);
        n = mk3(fn) * (1.0f / sqrtf(fn.w));
        pen = sqrtf(E.fc[ci].w);
    }
    return true;
}

// MprEpaSolver.SolveMpr (NarrowPhase.cs:98-347) up to the EPA hand-off.  Returns 0 (no
// overlap), 1 (overlap, result final) or 2 (overlap deeper than epa_threshold: the MPR
// result is in pA/pB/normal/pen as the fallback, and `portal` holds the tetrahedron EPA
// starts from).
// The search is a sequence of support evaluations, each followed by a few vector operations that
// choose the next direction; here it is a machine that is handed one support point at a time,
// so that the support maps stand in the code once and the lanes of a warp meet at them wherever
// their searches are.  KEEP_MISS: pA and pB of a miss are wanted (the first support point).
struct Mpr {
    static constexpr int MAX_ITER = 34;
    static constexpr float EPS = 1e-5f, TINY = 1e-16f;
    v3 v0, normal, pA, pB;  // v0: the origin ray's start; normal: the direction to evaluate next
    MV v1, v2, v3v;
    float pen;
    int stage, phase;       // stage 0, 1: first two points; 2: portal discovery; 3: refinement
    bool hit;

    __device__ __forceinline__ void begin(const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb) {
        MV c;
        mk_center(sa, sb, qb, pb, c);
        if (fabsf(c.V.x) < TINY && fabsf(c.V.y) < TINY && fabsf(c.V.z) < TINY) c.V.x = 1e-05f;
        v0 = c.V;
        normal = -v0;
        pen = 0.0f;
        stage = phase = 0;
        hit = false;
    }
    // The portal's plane; 0 when it is degenerate, else -1.
    __device__ __forceinline__ int face() {
        phase++;
        normal = cross(v2.V - v1.V, v3v.V - v1.V);
        if (len2(normal) < TINY) return 0;
        if (!hit) hit = dot(normal, v1.V) >= 0;
        return -1;
    }
    // Takes the support point along `normal`: -1 to go on, else the result code.
    template <bool KEEP_MISS>
    __device__ __forceinline__ int step(const MV& v, float epa_threshold) {
        if (stage < 3) {
            if (KEEP_MISS && stage == 0) { pA = v.A; pB = v.B; }
            if (dot(v.V, normal) <= 0.0f) return 0;
            if (stage == 0) {
                v1 = v;
                normal = cross(v1.V, v0);
                if (len2(normal) < 1e-12f) {
                    normal = v1.V - v0;
                    normal = normalize(normal);
                    pen = dot(v1.A - v1.B, normal);
                    pA = v1.A; pB = v1.B;
                    return 1;
                }
                stage = 1;
                return -1;
            }
            if (stage == 1) {
                v2 = v;
                normal = cross(v1.V - v0, v2.V - v0);
                if (dot(normal, v0) > 0.0f) {
                    const MV t = v1;
                    v1 = v2; v2 = t;
                    normal = -normal;
                }
                stage = 2;
                phase = 1;
                return -1;
            }
            v3v = v;
            const bool first = dot(cross(v1.V, v3v.V), v0) < 0.0f;
            if (first || dot(cross(v3v.V, v2.V), v0) < 0.0f) {
                if (first) v2 = v3v; else v1 = v3v;
                normal = cross(v1.V - v0, v2.V - v0);
                if (phase > MAX_ITER) return 0;
                phase++;
                return -1;
            }
            stage = 3;
            phase = 0;
            return face();
        }
        const float nsq = len2(normal);
        const float delta = dot(v.V - v3v.V, normal);
        pen = dot(v.V, normal);
        if (delta * delta <= EPS * EPS * nsq || pen <= 0.0f || phase > MAX_ITER) {
            if (!hit) return 0;
            const float invn = 1.0f / sqrtf(nsq);
            pen *= invn;
            normal = normal * invn;
            const float gamma = dot(cross(v1.V, v2.V - v1.V), normal) * invn;
            const float beta = dot(cross(v3v.V - v1.V, v1.V), normal) * invn;
            const float alpha = 1.0f - gamma - beta;
            pA = alpha * v1.A + beta * v2.A + gamma * v3v.A;
            pB = alpha * v1.B + beta * v2.B + gamma * v3v.B;
            return pen > epa_threshold ? 2 : 1;
        }
        const v3 t = cross(v.V, v0);
        if (dot(t, v1.V) >= 0.0f) {
            if (dot(t, v2.V) >= 0.0f) v1 = v; else v3v = v;
        } else {
            if (dot(t, v3v.V) >= 0.0f) v2 = v; else v1 = v;
        }
        return face();
    }
    // The tetrahedron EPA starts from.
    __device__ __forceinline__ MV corner(int k, const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb) const {
        MV c;
        mk_center(sa, sb, qb, pb, c);
        c.V = v0;
        return k == 0 ? c : (k == 1 ? v1 : (k == 2 ? v2 : v3v));
    }
};

// One search by a whole warp.
__device__ int mpr_warp(const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb, float epa_threshold,
                        v3& pA, v3& pB, v3& normal, float& pen, MV* portal) {
    Mpr M;
    M.begin(sa, sb, qb, pb);
    int code;
    do {
        MV v;
        mk_support(sa, sb, qb, pb, M.normal, v);
        code = M.step<true>(v, epa_threshold);
    } while (code < 0);
    pA = M.pA; pB = M.pB; normal = M.normal; pen = M.pen;
    if (code == 2)
        for (int k = 0; k < 4; k++) portal[k] = M.corner(k, sa, sb, qb, pb);
    return code;
}

// n searches, one per lane.  Most pairs separate after one or two support points and few
// take ten, so that a warp that waits for its last lane runs with a sixth of its lanes (5.0 of
// 32 measured): here a lane that is done waits only until half of its warp is, which then
// hands in its results and takes the next pairs.  A warp takes its pairs in rounds of `share`
// neighbours, fewer than 32 where there are fewer pairs than lanes: lanes of one warp that take
// different branches wait for each other.  load(q, sa, sb, qb, pb) returns a tag, negative for
// a pair to skip; flush(done, code, q, tag, M, sa, sb, qb, pb) is called by whole warps.
template <bool KEEP_MISS, class Load, class Flush>
__device__ __forceinline__ void mpr_lanes(int n, float epa_threshold, Load load, Flush flush) {
    const int lane = threadIdx.x & 31, per = blockDim.x >> 5;
    const int warps = gridDim.x * per, W = blockIdx.x * per + (threadIdx.x >> 5);
    const int rounds = (n - 1) / (32 * warps) + 1, share = (n - 1) / (warps * rounds) + 1, total = rounds * share;
    const int refill = (share + 1) / 2;
    Mpr M;
    ShapeRef sa, sb;
    q4 qb;
    v3 pb;
    int taken = 0, q = -1, code = 0, tag = 0;  // q: this lane's pair; code -1: in progress
    for (;;) {
        const unsigned running = __ballot_sync(FULL, code < 0);
        if (!running || (taken < total && share - __popc(running) >= refill)) {
            flush(q >= 0 && code >= 0, code, q, tag, M, sa, sb, qb, pb);
            const bool idle = code >= 0 && lane < share;
            const unsigned m = __ballot_sync(FULL, idle);
            if (idle) {
                q = -1;
                code = 0;
                const int k = taken + __popc(m & ((1u << lane) - 1u)), r = k / share;
                const int i = (r * warps + W) * share + k - r * share;
                if (k < total && i < n && (tag = load(i, sa, sb, qb, pb)) >= 0) {
                    q = i;
                    code = -1;
                    M.begin(sa, sb, qb, pb);
                }
            }
            taken += __popc(m);
            if (taken >= total && !__any_sync(FULL, code < 0)) break;
            continue;
        }
        if (code < 0) {
            MV v;
            mk_support_lane(sa, sb, qb, pb, M.normal, v);
            code = M.step<KEEP_MISS>(v, epa_threshold);
        }
    }
}
__device__ __forceinline__ void save_portal(const WorldDev& w, int e, const Mpr& M, const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb) {
    for (int k = 0; k < 4; k++) {
        const MV c = M.corner(k, sa, sb, qb, pb);
        w.col_portal[12 * e + 3 * k + 0] = f4(c.V, 0.f);
        w.col_portal[12 * e + 3 * k + 1] = f4(c.A, 0.f);
        w.col_portal[12 * e + 3 * k + 2] = f4(c.B, 0.f);
    }
}

// EPA from a saved MPR portal, by the whole warp; on failure the MPR result stands
// (NarrowPhase.cs:287-298).
__device__ void run_epa(EpaSmem& E, const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb, const MV* portal,
                        v3& pA, v3& pB, v3& normal, float& pen, NpStats& st, int& epa_calls, int& epa_fail) {
    const int lane = threadIdx.x & 31;
    if (lane < 4) {
        E.vV[lane] = f4(portal[lane].V, 0.f);
        E.vA[lane] = f4(portal[lane].A, 0.f);
        E.vB[lane] = f4(portal[lane].B, 0.f);
    }
    __syncwarp();
    epa_calls++;
    v3 a, b, n;
    float p;
    if (solve_epa(E, sa, sb, qb, pb, a, b, n, p, st)) { pA = a; pB = b; normal = n; pen = p; }
    else epa_fail++;
}

// MprEpaSolver.SolveMpr with its EPA refinement, whole warp (the edge filter's rerun).
__device__ __noinline__ bool solve_mpr(EpaSmem& E, const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb, float epa_threshold,
                          v3& pA, v3& pB, v3& normal, float& pen, NpStats& st, int& epa_calls, int& epa_fail) {
    MV portal[4];
    int code = mpr_warp(sa, sb, qb, pb, epa_threshold, pA, pB, normal, pen, portal);
    if (code == 2) run_epa(E, sa, sb, qb, pb, portal, pA, pB, normal, pen, st, epa_calls, epa_fail);
    return code != 0;
}

// NarrowPhase.MprEpa world-space wrapper (NarrowPhase.cs:902-927)
__device__ bool mpr_epa_world(EpaSmem& E, const ShapeRef& sa, const ShapeRef& sb, q4 qa, q4 qb, v3 pa, v3 pb,
                              v3& pA, v3& pB, v3& n, float& pen, float threshold, NpStats& st, int& ec, int& ef) {
    q4 q = qmul(qconj(qa), qb);
    v3 p = rotate_inv(pb - pa, qa);
    bool res = solve_mpr(E, sa, sb, q, p, threshold, pA, pB, n, pen, st, ec, ef);
    pA = rotate(pA, qa); pA = pA + pa;
    pB = rotate(pB, qa); pB = pB + pa;
    n = rotate(n, qa);
    return res;
}

// ---- TriangleEdgeCollisionFilter (TriangleEdgeCollisionFilter.cs:183-420) ---------------
enum { KEEP = 0, DISCARD = 1, EDGE = 2 };
__device__ __noinline__ int edge_evaluate(const WorldDev& w, int tri, q4 tq, v3 tp, bool tri_is_b, v3 cp, v3 n, v3& tn, v3& nn) {
    const TriDev& T = w.tris[tri];
    const float cosAngle = 0.999f, edgeThreshold = 0.01f;
    tn = rotate(mk3(T.n), tq);
    nn = mk3(0.f);
    if (tri_is_b) tn = -tn;
    if (dot(n, tn) < -cosAngle) return DISCARD;
    v3 a = rotate(mk3(T.a), tq) + tp, b = rotate(mk3(T.b), tq) + tp, c = rotate(mk3(T.c), tq) + tp;
    v3 pc = cp;
    {
        v3 ab = b - a, ac = c - a;
        v3 pn = normalize(cross(ab, ac));
        v3 ap = pc - a;
        float d = dot(ap, pn);
        pc = pc - d * pn;
    }
    v3 e = b - a, pma = pc - a;
    float d0 = len2(pma - dot(pma, e) * e * (1.0f / len2(e)));
    e = c - a; pma = pc - a;
    float d1 = len2(pma - dot(pma, e) * e * (1.0f / len2(e)));
    e = c - b; pma = pc - b;
    float d2 = len2(pma - dot(pma, e) * e * (1.0f / len2(e)));
    if (fminf(fminf(d0, d1), d2) > edgeThreshold * edgeThreshold) return KEEP;
    int which;
    if (d0 < d1 && d0 < d2) which = 2;
    else if (d1 < d2) which = 1;
    else which = 0;
    float4 nb = T.nb[which];
    if (nb.w == 0.f) return KEEP;
    nn = rotate(mk3(nb), tq);
    if (tri_is_b) nn = -nn;
    return EDGE;
}

// ---- one-shot manifold (CollisionManifold.cs) --------------------------------------------
__device__ __noinline__ bool polygon_sign(const float4* poly, int cnt, v3 n, float& sign) {
    float area = 0.0f;
    v3 prev = mk3(poly[cnt - 1]);
#pragma unroll 1
    for (int i = 0; i < cnt; i++) { v3 cur = mk3(poly[i]); area += dot(cross(prev, cur), n); prev = cur; }
    if (fabsf(area) <= 1e-6f) { sign = 0.f; return false; }
    sign = area < 0.0f ? -1.0f : 1.0f;
    return true;
}
__device__ __forceinline__ bool contains_pt(const float4* poly, int cnt, v3 p, v3 n, float sign) {
    v3 prev = mk3(poly[cnt - 1]);
#pragma unroll 1
    for (int i = 0; i < cnt; i++) {
        v3 cur = mk3(poly[i]);
        float sd = sign * dot(cross(cur - prev, p - prev), n);
        if (sd < -1e-3f) return false;
        prev = cur;
    }
    return true;
}
__device__ __noinline__ int clip_segment(v3 s, v3 e, const float4* poly, int pc, v3 n, float sign, v3* out) {
    const float eps = 1e-3f;
    float enter = 0.0f, exit = 1.0f;
    v3 delta = e - s;
#pragma unroll 1
    for (int i = 0; i < pc; i++) {
        v3 es = mk3(poly[i]), ee = mk3(poly[(i + 1) % pc]);
        float ss = sign * dot(cross(ee - es, s - es), n);
        float se = sign * dot(cross(ee - es, e - es), n);
        bool si = ss >= -eps, ei = se >= -eps;
        if (!si && !ei) return 0;
        if (si && ei) continue;
        float den = ss - se;
        if (fabsf(den) <= eps) return 0;
        float t = fminf(fmaxf(ss / den, 0.0f), 1.0f);
        if (!si) enter = fmaxf(enter, t); else exit = fminf(exit, t);
        if (exit < enter) return 0;
    }
    out[0] = s + enter * delta;
    if (len2(s + exit * delta - out[0]) < eps) return 1;
    out[1] = s + exit * delta;
    return 2;
}
__device__ __forceinline__ float cross_along(v3 l, v3 r, v3 n) { return dot(cross(l, r), n); }
__device__ __forceinline__ int intersect_seg(v3 sA, v3 eA, v3 sB, v3 eB, v3 n, v3* cA, v3* cB) {
    const float eps = 1e-3f;
    v3 dA = eA - sA, dB = eB - sB, off = sB - sA;
    float cr = cross_along(dA, dB, n);
    if (fabsf(cr) <= eps) {
        if (fabsf(cross_along(off, dA, n)) > eps) return 0;
        float la = len2(dA), lb = len2(dB);
        if (la <= eps || lb <= eps) return 0;
        float b0 = dot(sB - sA, dA) / la, b1 = dot(eB - sA, dA) / la;
        float enter = fmaxf(0.0f, fminf(b0, b1));
        float exit = fminf(1.0f, fmaxf(b0, b1));
        if (exit < enter - eps) return 0;
        cA[0] = sA + enter * dA;
        float a0 = fminf(fmaxf(dot(cA[0] - sB, dB) / lb, 0.0f), 1.0f);
        cB[0] = sB + a0 * dB;
        cA[1] = sA + exit * dA;
        if (len2(cA[1] - cA[0]) <= eps) return 1;
        float a1 = fminf(fmaxf(dot(cA[1] - sB, dB) / lb, 0.0f), 1.0f);
        cB[1] = sB + a1 * dB;
        return 2;
    }
    float t = cross_along(off, dB, n) / cr;
    float u = cross_along(off, dA, n) / cr;
    if (t < -eps || t > 1.0f + eps || u < -eps || u > 1.0f + eps) return 0;
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    u = fminf(fmaxf(u, 0.0f), 1.0f);
    cA[0] = sA + t * dA;
    cB[0] = sB + u * dB;
    return 1;
}
__device__ bool is_dup(const float4* m, int cnt, v3 p) {
#pragma unroll 1
    for (int i = 0; i < cnt; i++) if (len2(mk3(m[i]) - p) < 0.001f) return true;
    return false;
}
struct MF {
    EpaSmem* E;
    int count;
    __device__ __forceinline__ bool seen(const float4* m, v3 p) const {
        const int lane = threadIdx.x & 31;
        return __any_sync(FULL, lane < count && len2(mk3(m[lane]) - p) < 0.001f);
    }
    __device__ void set(int i, v3 a, v3 b) {
        if ((threadIdx.x & 31) == 0) { E->mA[i] = f4(a, 0.f); E->mB[i] = f4(b, 0.f); }
        __syncwarp();
    }
    __device__ __noinline__ void on_a(v3 p, v3 pB, v3 n) {
        if (count == 12) return;
        float diff = dot(p - pB, n);
        if (diff < 0.0f) return;
        if (seen(E->mA, p)) return;
        set(count, p, p - diff * n);
        count++;
    }
    __device__ __noinline__ void on_b(v3 p, v3 pA, v3 n) {
        if (count == 12) return;
        float diff = dot(p - pA, n);
        if (diff > 0.0f) return;
        if (seen(E->mB, p)) return;
        set(count, p - diff * n, p);
        count++;
    }
    __device__ __noinline__ void pair(v3 a, v3 b, v3 n) {
        if (count == 12) return;
        if (dot(a - b, n) < 0.0f) return;
        if (seen(E->mA, a)) return;
        if (seen(E->mB, b)) return;
        set(count, a, b);
        count++;
    }
};

// The directions of the six samples around the normal.
__device__ __constant__ float c_hex[12] = {1.0f, 0.0f, 0.5f, 0.86602540378f, -0.5f, 0.86602540378f,
                                           -1.0f, 0.0f, -0.5f, -0.86602540378f, 0.5f, -0.86602540378f};
// A sampled polygon from the points of lanes `first` .. `first` + 5, without the points that
// repeat its first or last one.
__device__ __forceinline__ int sample_polygon(float4* arr, v3 pt, int first) {
    int cnt = 0;
    v3 head = mk3(0.f), tail = mk3(0.f);
#pragma unroll 1
    for (int e = first; e < first + 6; e++) {
        const v3 v = mk3(__shfl_sync(FULL, pt.x, e), __shfl_sync(FULL, pt.y, e), __shfl_sync(FULL, pt.z, e));
        if (cnt > 0 && len2(head - v) < 0.001f) continue;
        if (cnt > 1 && len2(tail - v) < 0.001f) continue;
        if (cnt == 0) head = v;
        tail = v;
        if ((threadIdx.x & 31) == 0) arr[cnt] = f4(v, 0.f);
        cnt++;
    }
    __syncwarp();
    return cnt;
}
// A point cloud's samples, by the whole warp; lane first + e keeps the e-th.
__device__ __noinline__ v3 sample_hull(const ShapeRef& s, q4 q, v3 dir, int first) {
    v3 mine = mk3(0.f);
#pragma unroll 1
    for (int e = first; e < first + 6; e++) {
        const v3 d = mk3(__shfl_sync(FULL, dir.x, e), __shfl_sync(FULL, dir.y, e), __shfl_sync(FULL, dir.z, e));
        const v3 p = hull_support_warp(s.hull, s.nhull, d) + s.d;
        if ((threadIdx.x & 31) == e) mine = p;
    }
    return mine;
}

// CollisionManifold.BuildManifold by a whole warp: a lane per sample, polygon corner, edge pair
// and angle; the points are inserted in the reference's order.  (With every lane at the same
// sample the twelve support maps stood in the code one after the other, and the warps of an SM,
// each at another place, waited for instructions half of the time.)
__device__ __noinline__ int build_manifold(EpaSmem& E, const ShapeRef& sa, const ShapeRef& sb, q4 qa, q4 qb, v3 pa, v3 pb,
                              v3 pA, v3 pB, v3 n, v3* outA, v3* outB) {
    const int lane = threadIdx.x & 31;
    const float P = 0.01f;
    v3 c1 = create_orthonormal(n);
    v3 c2 = cross(n, c1);
    v3 relB = pb - pa, pAl = pA - pa, pBl = pB - pa;
    // lanes 0 to 5: A's samples, 6 to 11: B's
    const bool onB = lane >= 6;
    const int e = onB ? lane - 6 : lane, h = e < 6 ? e : 0;
    v3 pn = n + c_hex[2 * h] * P * c1 + c_hex[2 * h + 1] * P * c2;
    if (onB) pn = -pn;
    const q4 q = onB ? qb : qa;
    const v3 dir = rotate_inv(pn, q);
    v3 pt = mk3(0.f);
    const bool hullA = sa.kind == JG_SHAPE_POINTCLOUD, hullB = sb.kind == JG_SHAPE_POINTCLOUD;
    if (lane < 12 && !(onB ? hullB : hullA)) pt = support_lane(onB ? sb : sa, dir);
    __syncwarp();
    if (hullA) { const v3 p = sample_hull(sa, qa, dir, 0); if (!onB) pt = p; }
    if (hullB) { const v3 p = sample_hull(sb, qb, dir, 6); if (onB) pt = p; }
    pt = rotate(pt, q);
    if (onB) pt = pt + relB;
    const int lc = sample_polygon(E.left, pt, 0), rc = sample_polygon(E.right, pt, 6);
    float ls = 0.f, rs = 0.f;
    bool lp = lc > 2 && polygon_sign(E.left, lc, n, ls);
    bool rp = rc > 2 && polygon_sign(E.right, rc, n, rs);
    MF m; m.E = &E; m.count = 0;
    if (lp) {
        for (unsigned in = __ballot_sync(FULL, lane < rc && contains_pt(E.left, lc, mk3(E.right[lane]), n, ls)); in; in &= in - 1) {
            m.on_b(mk3(E.right[__ffs(in) - 1]), pAl, n);
            if (m.count == 12) goto finalize;
        }
        if (rc == 2) {
            v3 cl[2];
            int k = clip_segment(mk3(E.right[0]), mk3(E.right[1]), E.left, lc, n, ls, cl);
            for (int i = 0; i < k; i++) { m.on_b(cl[i], pAl, n); if (m.count == 12) goto finalize; }
        }
    }
    if (rp) {
        for (unsigned in = __ballot_sync(FULL, lane < lc && contains_pt(E.right, rc, mk3(E.left[lane]), n, rs)); in; in &= in - 1) {
            m.on_a(mk3(E.left[__ffs(in) - 1]), pBl, n);
            if (m.count == 12) goto finalize;
        }
        if (lc == 2) {
            v3 cl[2];
            int k = clip_segment(mk3(E.left[0]), mk3(E.left[1]), E.right, rc, n, rs, cl);
            for (int i = 0; i < k; i++) { m.on_a(cl[i], pBl, n); if (m.count == 12) goto finalize; }
        }
    }
    if (lc == 2 && rc == 2) {
        v3 cA[2], cB[2];
        int k = intersect_seg(mk3(E.left[0]), mk3(E.left[1]), mk3(E.right[0]), mk3(E.right[1]), n, cA, cB);
        for (int i = 0; i < k; i++) { m.pair(cA[i], cB[i], n); if (m.count == 12) goto finalize; }
    }
    if (lp && rp) {
        // every (left edge, right edge) intersection, one lane per edge pair, inserted in
        // the reference's (i, j) order
        int total = lc * rc;
        for (int base = 0; base < total; base += 32) {
            int idx = base + lane;
            v3 cA[2], cB[2];
            int k = 0;
            if (idx < total) {
                int i = idx / rc, j = idx % rc;
                k = intersect_seg(mk3(E.left[i]), mk3(E.left[(i + 1) % lc]), mk3(E.right[j]), mk3(E.right[(j + 1) % rc]), n, cA, cB);
            }
            unsigned any = __ballot_sync(FULL, k > 0);
            while (any) {
                int src = __ffs(any) - 1;
                any &= any - 1;
                int kk = __shfl_sync(FULL, k, src);
                for (int q = 0; q < kk; q++) {
                    v3 a, b;
                    a.x = __shfl_sync(FULL, cA[q].x, src); a.y = __shfl_sync(FULL, cA[q].y, src); a.z = __shfl_sync(FULL, cA[q].z, src);
                    b.x = __shfl_sync(FULL, cB[q].x, src); b.y = __shfl_sync(FULL, cB[q].y, src); b.z = __shfl_sync(FULL, cB[q].z, src);
                    m.pair(a, b, n);
                    if (m.count == 12) goto finalize;
                }
            }
        }
    }
    if (m.count <= 1) { m.set(0, pAl, pBl); m.count = 1; }
    else if (m.count < 4) { m.set(m.count, pAl, pBl); m.count++; }
finalize:
    int count = m.count;
    if (count > 4) {
        // ReduceManifold (CollisionManifold.cs:321-375)
        v3 c = mk3(0.f);
#pragma unroll 1
        for (int i = 0; i < count; i++) c = c + mk3(E.mA[i]);
        c = c * (float)(1.0 / count);
        v3 t1 = create_orthonormal(n);
        v3 t2 = cross(n, t1);
        // the points' places in the order of their angles (equal ones as they come)
        const v3 d = mk3(E.mA[lane < count ? lane : 0]) - c;
        const float ang = StableMathF::atan2(dot(d, t2), dot(d, t1));
        int place = 0;
#pragma unroll 1
        for (int i = 0; i < count; i++) {
            const float o = __shfl_sync(FULL, ang, i);
            place += o < ang || (o == ang && i < lane);
        }
        if (lane >= count) place = -1;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int sel = max(__ffs(__ballot_sync(FULL, place == ((2 * i + 1) * count) / 8)) - 1, 0);
            outA[i] = mk3(E.mA[sel]) + pa;
            outB[i] = mk3(E.mB[sel]) + pa;
        }
        __syncwarp();
        return 4;
    }
    for (int i = 0; i < count; i++) { outA[i] = mk3(E.mA[i]) + pa; outB[i] = mk3(E.mB[i]) + pa; }
    __syncwarp();
    return count;
}

// ---- one-shot manifold, one thread per pair ----------------------------------------------
// The same steps as build_manifold (CollisionManifold.cs:393-566) with the candidate lists
// in thread-local storage, for analytic shapes and point clouds alike.
struct MFT {
    float4 A[12], B[12];
    int count;
    __device__ void on_a(v3 p, v3 pB, v3 n) {
        if (count == 12) return;
        float diff = dot(p - pB, n);
        if (diff < 0.0f) return;
        if (is_dup(A, count, p)) return;
        A[count] = f4(p, 0.f); B[count] = f4(p - diff * n, 0.f); count++;
    }
    __device__ void on_b(v3 p, v3 pA, v3 n) {
        if (count == 12) return;
        float diff = dot(p - pA, n);
        if (diff > 0.0f) return;
        if (is_dup(B, count, p)) return;
        A[count] = f4(p - diff * n, 0.f); B[count] = f4(p, 0.f); count++;
    }
    __device__ void pair(v3 a, v3 b, v3 n) {
        if (count == 12) return;
        if (dot(a - b, n) < 0.0f) return;
        if (is_dup(A, count, a)) return;
        if (is_dup(B, count, b)) return;
        A[count] = f4(a, 0.f); B[count] = f4(b, 0.f); count++;
    }
};
__device__ __forceinline__ void push_local(float4* arr, int& cnt, v3 v) {
    if (cnt > 0 && len2(mk3(arr[0]) - v) < 0.001f) return;
    if (cnt > 1 && len2(mk3(arr[cnt - 1]) - v) < 0.001f) return;
    arr[cnt++] = f4(v, 0.f);
}

__device__ __noinline__ int manifold_thread(const ShapeRef& sa, const ShapeRef& sb, q4 qa, q4 qb, v3 pa, v3 pb,
                                            v3 pA, v3 pB, v3 n, float4* outA, float4* outB) {
    const float P = 0.01f;
    const float* hx = c_hex;
    v3 c1 = create_orthonormal(n);
    v3 c2 = cross(n, c1);
    v3 relB = pb - pa, pAl = pA - pa, pBl = pB - pa;
    float4 left[6], right[6];
    int lc = 0, rc = 0;
#pragma unroll 1
    for (int e = 0; e < 6; e++) {
        v3 pn = n + hx[2 * e + 0] * P * c1 + hx[2 * e + 1] * P * c2;
        push_local(left, lc, rotate(support_lane(sa, rotate_inv(pn, qa)), qa));
        pn = -pn;
        push_local(right, rc, rotate(support_lane(sb, rotate_inv(pn, qb)), qb) + relB);
    }
    float ls = 0.f, rs = 0.f;
    bool lp = lc > 2 && polygon_sign(left, lc, n, ls);
    bool rp = rc > 2 && polygon_sign(right, rc, n, rs);
    MFT m;
    m.count = 0;
    if (lp) {
        for (int e = 0; e < rc; e++) {
            v3 p = mk3(right[e]);
            if (!contains_pt(left, lc, p, n, ls)) continue;
            m.on_b(p, pAl, n);
            if (m.count == 12) goto finalize;
        }
        if (rc == 2) {
            v3 cl[2];
            int k = clip_segment(mk3(right[0]), mk3(right[1]), left, lc, n, ls, cl);
            for (int i = 0; i < k; i++) { m.on_b(cl[i], pAl, n); if (m.count == 12) goto finalize; }
        }
    }
    if (rp) {
        for (int e = 0; e < lc; e++) {
            v3 p = mk3(left[e]);
            if (!contains_pt(right, rc, p, n, rs)) continue;
            m.on_a(p, pBl, n);
            if (m.count == 12) goto finalize;
        }
        if (lc == 2) {
            v3 cl[2];
            int k = clip_segment(mk3(left[0]), mk3(left[1]), right, rc, n, rs, cl);
            for (int i = 0; i < k; i++) { m.on_a(cl[i], pBl, n); if (m.count == 12) goto finalize; }
        }
    }
    if (lc == 2 && rc == 2) {
        v3 cA[2], cB[2];
        int k = intersect_seg(mk3(left[0]), mk3(left[1]), mk3(right[0]), mk3(right[1]), n, cA, cB);
        for (int i = 0; i < k; i++) { m.pair(cA[i], cB[i], n); if (m.count == 12) goto finalize; }
    }
    if (lp && rp) {
        for (int i = 0; i < lc; i++) {
            v3 sA = mk3(left[i]), eA = mk3(left[(i + 1) % lc]);
            for (int j = 0; j < rc; j++) {
                v3 cA[2], cB[2];
                int k = intersect_seg(sA, eA, mk3(right[j]), mk3(right[(j + 1) % rc]), n, cA, cB);
                for (int q = 0; q < k; q++) { m.pair(cA[q], cB[q], n); if (m.count == 12) goto finalize; }
            }
        }
    }
    if (m.count <= 1) { m.A[0] = f4(pAl, 0.f); m.B[0] = f4(pBl, 0.f); m.count = 1; }
    else if (m.count < 4) { m.A[m.count] = f4(pAl, 0.f); m.B[m.count] = f4(pBl, 0.f); m.count++; }
finalize:
    int count = m.count;
    if (count > 4) {
        // ReduceManifold (CollisionManifold.cs:321-375)
        v3 c = mk3(0.f);
        for (int i = 0; i < count; i++) c = c + mk3(m.A[i]);
        c = c * (float)(1.0 / count);
        v3 t1 = create_orthonormal(n);
        v3 t2 = cross(n, t1);
        float ang[12];
        int order[12];
        for (int i = 0; i < count; i++) {
            v3 d = mk3(m.A[i]) - c;
            ang[i] = StableMathF::atan2(dot(d, t2), dot(d, t1));
            order[i] = i;
        }
        for (int i = 1; i < count; i++) {
            int cur = order[i];
            float ca = ang[cur];
            int j = i - 1;
            while (j >= 0 && ang[order[j]] > ca) { order[j + 1] = order[j]; j--; }
            order[j + 1] = cur;
        }
        for (int i = 0; i < 4; i++) {
            int sel = order[((2 * i + 1) * count) / 8];
            outA[i] = f4(mk3(m.A[sel]) + pa, 0.f);
            outB[i] = f4(mk3(m.B[sel]) + pa, 0.f);
        }
        return 4;
    }
    for (int i = 0; i < count; i++) { outA[i] = f4(mk3(m.A[i]) + pa, 0.f); outB[i] = f4(mk3(m.B[i]) + pa, 0.f); }
    return count;
}

constexpr int NP_WARPS = 4;
// Up to this many records per warp of stage 3, its warps take them all: a manifold is a long chain
// of one thread (23 us for the 18 records of 27 boxes, 60 us for mixed shapes), which few records
// leave alone on the GPU, and a warp shortens.  Narrowphase in us, by warps and by threads: 18 records
// 47 and 53, 1149 (a pile of 700) 271 and 320, 6578 (48 worlds) 355 and 390, 13,700 (100 worlds) 416
// and 406.
constexpr int WARP_RECORDS = 4;
constexpr int COL_WORLD = 4;  // kind of a colliding record that stage 3 has put into world space
constexpr int COL_EDGE = 8;   // in a colliding record's kind: it waits in the edge list

__device__ __forceinline__ int warp_append(int* counter, bool pred) {
    const int lane = threadIdx.x & 31;
    unsigned m = __ballot_sync(FULL, pred);
    if (!m) return -1;
    int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(FULL, base, leader);
    return pred ? base + __popc(m & ((1u << lane) - 1u)) : -1;
}

// Pairs grouped by the kinds of their two shapes (a counting sort over the 64 kind
// combinations), so that the threads of a warp run the same support maps in MPR.  The
// order inside a group does not matter: results do not depend on the pair order.  The pairs are
// the broadphase's (`pairs` null: the world's list and count) or a query's.
constexpr int PAIR_ITEMS = 4;  // pairs per thread and round of the scatter
struct PairList {
    const int2* pairs;
    int n;
};
__device__ __forceinline__ int pair_count(const WorldDev& w, const PairList& L) {
    return L.pairs ? L.n : min(w.ctr->npairs, w.cap_pairs);
}
__device__ __forceinline__ int pair_kind_key(const WorldDev& w, const int2* pairs, int p) {
    int2 pr = pairs[p];
    return ((w.sinfo[pr.x].x & 7) << 3) | (w.sinfo[pr.y].x & 7);
}
__global__ void k_pair_hist(WorldDev w, PairList L) {
    __shared__ int h[64];
    if (threadIdx.x < 64) h[threadIdx.x] = 0;
    __syncthreads();
    const int n = pair_count(w, L);
    const int2* pairs = L.pairs ? L.pairs : w.pairs;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        atomicAdd(&h[pair_kind_key(w, pairs, p)], 1);
    __syncthreads();
    if (threadIdx.x < 64 && h[threadIdx.x]) atomicAdd(&w.pair_kind[threadIdx.x], h[threadIdx.x]);
}
__global__ void k_pair_scatter(WorldDev w, PairList L) {
    __shared__ int s_first[64];  // first place of each kind combination
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        const int x = w.pair_kind[lane], y = w.pair_kind[32 + lane];
        int a = x, b = y;
        for (int o = 1; o < 32; o <<= 1) {
            const int pa = __shfl_up_sync(FULL, a, o), pb = __shfl_up_sync(FULL, b, o);
            if (lane >= o) { a += pa; b += pb; }
        }
        s_first[lane] = a - x;
        s_first[32 + lane] = __shfl_sync(FULL, a, 31) + b - y;
    }
    __syncthreads();
    // A block takes its pairs a round at a time: counts per combination, one claim of places per
    // combination, then the places.  (A claim per warp and combination met at 64 counters:
    // 156 us for the 2.0 M pairs of 4096 worlds, now 20.)
    __shared__ int s_cnt[64], s_at[64];
    const int n = pair_count(w, L);
    const int2* pairs = L.pairs ? L.pairs : w.pairs;
    for (int base = blockIdx.x * blockDim.x * PAIR_ITEMS; base < n; base += gridDim.x * blockDim.x * PAIR_ITEMS) {
        if (threadIdx.x < 64) s_cnt[threadIdx.x] = 0;
        __syncthreads();
        int key[PAIR_ITEMS], at[PAIR_ITEMS];
#pragma unroll
        for (int r = 0; r < PAIR_ITEMS; r++) {
            const int p = base + r * blockDim.x + threadIdx.x;
            key[r] = p < n ? pair_kind_key(w, pairs, p) : 64 + lane;
            const unsigned same = __match_any_sync(FULL, key[r]);
            const int leader = __ffs(same) - 1;
            int first = 0;
            if (lane == leader && key[r] < 64) first = atomicAdd(&s_cnt[key[r]], __popc(same));
            at[r] = __shfl_sync(FULL, first, leader) + __popc(same & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (threadIdx.x < 64 && s_cnt[threadIdx.x])
            s_at[threadIdx.x] = s_first[threadIdx.x] + atomicAdd(&w.pair_kind[64 + threadIdx.x], s_cnt[threadIdx.x]);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < PAIR_ITEMS; r++) {
            const int p = base + r * blockDim.x + threadIdx.x;
            if (p < n) w.pair_order[s_at[key[r]] + at[r]] = p;
        }
        __syncthreads();
    }
}

// Stage 1, one thread per broadphase pair: the MPR overlap test in A's frame
// (NarrowPhase.MprEpa, NarrowPhase.cs:902-927, up to the EPA hand-off).  Overlapping pairs
// are appended to the colliding list with their MPR result; deeper than the EPA threshold,
// also to the EPA list with the MPR portal EPA starts from.  Separated pairs with a
// speculative body go to the sweep list (World.Detect.cs:162-170).  Bound by instruction issue
// and, where a lane takes its next pair, by the loads of the two shapes; as many warps as the
// registers of a search allow (three or four CTAs an SM spill: 0.5 ms more on 4096 worlds).
// Against one thread per pair to the end: 4096 worlds 1.30 -> 0.66 ms, a settled 100k pile
// 0.62 -> 0.33, a 20k pile 0.13 -> 0.11, a 700-body pile 0.064 -> 0.044.
__global__ void __launch_bounds__(256, 2) k_mpr(WorldDev w) {
    const int npairs = min(w.ctr->npairs, w.cap_pairs);
    const int cap = w.cap_arb;
    if (npairs <= 0) return;
    mpr_lanes<false>(
        npairs, 0.02f,
        [&](int q, ShapeRef& sa, ShapeRef& sb, q4& rot, v3& rel) {
            const int2 pr = w.pairs[w.pair_order[q]];
            const int s1 = pr.x, s2 = pr.y;  // s1 < s2: ShapeId order (World.Detect.cs:141-144)
            const int b1 = w.sinfo[s1].y, b2 = w.sinfo[s2].y;
            const int4 i1 = w.binfo[b1], i2 = w.binfo[b2];
            if ((!(i1.y & JG_BODY_ACTIVE) && !(i2.y & JG_BODY_ACTIVE)) ||
                (i1.x != JG_MOTION_DYNAMIC && i2.x != JG_MOTION_DYNAMIC)) return -1;
            sa = load_shape(w, s1);
            sb = load_shape(w, s2);
            const q4 qa = mkq(w.q[b1]);
            rot = qmul(qconj(qa), mkq(w.q[b2]));
            rel = rotate_inv(mk3(w.pos[b2]) - mk3(w.pos[b1]), qa);
            return ((i1.y | i2.y) & JG_BODY_SPECULATIVE) != 0 ? 1 : 0;
        },
        [&](bool done, int code, int q, int spec_body, const Mpr& M, const ShapeRef& sa, const ShapeRef& sb, q4 rot, v3 rel) {
            const int p = done ? w.pair_order[q] : 0;
            const int si = warp_append(&w.ctr->nspec, done && code == 0 && spec_body);
            if (si >= 0) w.spec_list[si] = p;
            int c = warp_append(&w.ctr->ncol, done && code != 0);
            if (c >= cap) { atomicCAS(&w.ctr->status, 0, JG_ERR_CAPACITY); c = -1; }
            if (c >= 0) {
                w.col_pair[c] = make_int2(p, code);
                w.col_res[3 * c + 0] = f4(M.pA, 0.f);
                w.col_res[3 * c + 1] = f4(M.pB, 0.f);
                w.col_res[3 * c + 2] = f4(M.normal, M.pen);
            }
            const int e = warp_append(&w.ctr->nepa_list, code == 2 && c >= 0);
            if (e >= 0) {
                w.epa_list[e] = c;
                save_portal(w, e, M, sa, sb, rot, rel);
            }
        });
}

// ---- speculative contacts: time of impact by conservative advancement --------------------
// GJK simplex with witness points (SimplexSolverAB.cs:28-359), one thread: up to four
// Minkowski vertices with their support points on A and B, the barycentric weights of the
// point nearest the origin, and the mask of the vertices spanning it.
struct SimplexAB {
    MV v[4];
    float bc[4];
    unsigned mask;

    // ClosestSegment (SimplexSolverAB.cs:60-100)
    __device__ v3 segment(int i0, int i1, float* w, unsigned& m) const {
        v3 a = v[i0].V, b = v[i1].V;
        v3 d = b - a;
        float dd = len2(d);
        if (dd < 1e-8f) { m = 1u << i1; w[i0] = 0.f; w[i1] = 1.f; return b; }
        float t = -dot(a, d) / dd;
        if (t > 1.0f) { m = 1u << i1; w[i0] = 0.f; w[i1] = 1.f; return b; }
        if (t < 0.0f) { m = 1u << i0; w[i0] = 1.f; w[i1] = 0.f; return a; }
        w[i0] = 1.0f - t; w[i1] = t;
        m = (1u << i0) | (1u << i1);
        return cross(d, cross(a, d)) * (1.0f / dd);
    }
    // ClosestTriangle (SimplexSolverAB.cs:102-176): the interior when every weight is
    // non-negative and the triangle is not degenerate, else the nearest edge among those
    // opposite a negative weight (all three edges when degenerate).
    __device__ v3 triangle(int i0, int i1, int i2, float* w, unsigned& m) const {
        m = 0;
        v3 a = v[i0].V, b = v[i1].V, c = v[i2].V;
        v3 u = a - b, e = a - c;
        v3 nrm = cross(u, e);
        float t = len2(nrm);
        float it = 1.0f / t;
        bool degenerate = t < 1e-8f;
        float l2 = dot(cross(u, a), nrm) * it;
        float l1 = dot(cross(a, e), nrm) * it;
        float l0 = 1.0f - l2 - l1;
        const int ea[3] = {i1, i0, i0}, eb[3] = {i2, i2, i1};
        const float lam[3] = {l0, l1, l2};
        float best = 3.402823466e+38f;
        v3 cp = mk3(0.f);
        float tmp[4];
        for (int k = 0; k < 3; k++) {
            if (!(lam[k] < 0.0f || degenerate)) continue;
            unsigned mk;
            v3 q = segment(ea[k], eb[k], tmp, mk);
            float dist = len2(q);
            if (dist < best) {
                for (int j = 0; j < 4; j++) w[j] = tmp[j];
                m = mk; cp = q; best = dist;
            }
        }
        if (m != 0) return cp;
        w[i0] = l0; w[i1] = l1; w[i2] = l2;
        m = (1u << i0) | (1u << i1) | (1u << i2);
        return nrm * (dot(nrm, a) * it);
    }
    __device__ static float det(v3 a, v3 b, v3 c, v3 d) { return dot(b - a, cross(c - a, d - a)); }
    // ClosestTetrahedron (SimplexSolverAB.cs:178-276)
    __device__ v3 tetra(float* w, unsigned& m) const {
        float dt = det(v[0].V, v[1].V, v[2].V, v[3].V);
        float idt = 1.0f / dt;
        bool degenerate = dt * dt < 1e-8f;
        v3 z = mk3(0.f);
        float l0 = det(z, v[1].V, v[2].V, v[3].V) * idt;
        float l1 = det(v[0].V, z, v[2].V, v[3].V) * idt;
        float l2 = det(v[0].V, v[1].V, z, v[3].V) * idt;
        float l3 = 1.0f - l0 - l1 - l2;
        const int fa[4] = {1, 0, 0, 0}, fb[4] = {2, 2, 1, 1}, fc[4] = {3, 3, 3, 2};
        const float lam[4] = {l0, l1, l2, l3};
        float best = 3.402823466e+38f;
        v3 cp = mk3(0.f);
        float tmp[4];
        m = 0;
        for (int k = 0; k < 4; k++) {
            if (!(lam[k] < 0.0f || degenerate)) continue;
            unsigned mk;
            v3 q = triangle(fa[k], fb[k], fc[k], tmp, mk);
            float dist = len2(q);
            if (dist < best) {
                for (int j = 0; j < 4; j++) w[j] = tmp[j];
                m = mk; cp = q; best = dist;
            }
        }
        if (m != 0) return cp;
        w[0] = l0; w[1] = l1; w[2] = l2; w[3] = l3;
        m = 15u;
        return mk3(0.f);
    }
    // AddVertex (SimplexSolverAB.cs:300-357): false when the tetrahedron encloses the origin.
    __device__ bool add(const MV& x, v3& closest) {
        int ix[4], used = 0, free_slot = 0;
        for (int i = 0; i < 4; i++) {
            if (mask & (1u << i)) ix[used++] = i;
            else free_slot = i;
        }
        ix[used++] = free_slot;
        v[free_slot] = x;
        if (used == 1) { closest = v[ix[0]].V; mask = 1u << ix[0]; bc[ix[0]] = 1.0f; return true; }
        if (used == 2) { closest = segment(ix[0], ix[1], bc, mask); return true; }
        if (used == 3) { closest = triangle(ix[0], ix[1], ix[2], bc, mask); return true; }
        closest = tetra(bc, mask);
        return mask != 15u;
    }
    // GetClosest (SimplexSolverAB.cs:278-293)
    __device__ void closest_points(v3& pA, v3& pB) const {
        pA = mk3(0.f); pB = mk3(0.f);
        for (int i = 0; i < 4; i++) {
            if (!(mask & (1u << i))) continue;
            pA = pA + bc[i] * v[i].A;
            pB = pB + bc[i] * v[i].B;
        }
    }
};

// NarrowPhase.Sweep with A at the origin (NarrowPhase.cs:1155-1222): B moves along `sweep`;
// a support point in front of the search direction advances the time of impact to the
// plane it spans.  False when B moves away from that plane (no hit); lambda = 0 when the
// shapes already overlap.  At most 34 support evaluations.
__device__ bool sweep_local(const ShapeRef& sa, const ShapeRef& sb, q4 qb, v3 pb, v3 sweep, v3& pA, v3& pB,
                            v3& normal, float& lambda) {
    SimplexAB sx;
    sx.mask = 0;
    MV c;
    mk_center(sa, sb, qb, pb, c);
    v3 pos = pb;
    lambda = 0.0f;
    v3 v = -c.V;
    normal = mk3(0.f);
    int iter = 34;
    float d2 = len2(v);
    while (d2 > 1e-4f * 1e-4f && iter-- != 0) {
        MV x;
        mk_support_lane(sa, sb, qb, pos, v, x);
        float vw = -dot(v, x.V);
        if (vw > 0.0f) {
            float vr = dot(v, sweep);
            if (vr >= -1e-12f) { lambda = __int_as_float(0x7f800000); return false; }
            lambda -= vw / vr;
            pos = pb + lambda * sweep;
            normal = v;
        }
        if (!sx.add(x, v)) break;
        v = -v;
        d2 = len2(v);
    }
    sx.closest_points(pA, pB);
    normal = normalize_safe(normal, 1e-16f);
    return true;
}

// Stage 1b, one thread per pair the MPR stage found separated with a speculative body
// (World.Detect.cs:168-196): pairs closing slower than the threshold speed are dropped; the
// rest run the sweep in A's frame (NarrowPhase.cs:1100-1136) and are kept when it hits
// within the step (0 < toi <= dt).  The record goes to the colliding list in world space
// with kind 3, penetration n . (pA - pB) * SpeculativeRelaxationFactor.
__global__ void __launch_bounds__(128) k_sweep(WorldDev w, StepParams sp) {
    const int ns = min(w.ctr->nspec, w.cap_pairs);
    const int cap = w.cap_arb;
    for (int base = blockIdx.x * blockDim.x; base < ns; base += gridDim.x * blockDim.x) {
        const int i = base + threadIdx.x;
        bool hit = false;
        int p = 0;
        v3 pA = mk3(0.f), pB = mk3(0.f), n = mk3(0.f);
        float pen = 0.f;
        if (i < ns) {
            p = w.spec_list[i];
            int2 pr = w.pairs[p];
            int b1 = w.sinfo[pr.x].y, b2 = w.sinfo[pr.y].y;
            ShapeRef sa = load_shape(w, pr.x), sb = load_shape(w, pr.y);
            q4 qa = mkq(w.q[b1]), qb = mkq(w.q[b2]);
            v3 pa = mk3(w.pos[b1]), pb = mk3(w.pos[b2]);
            v3 va = mk3(w.body[b1].v), vb = mk3(w.body[b2].v);
            v3 dv = vb - va;
            q4 q = qmul(qconj(qa), qb);
            v3 prl = rotate_inv(pb - pa, qa);
            v3 swl = rotate_inv(dv, qa);
            float toi;
            if (!(len2(dv) < sp.spec_threshold * sp.spec_threshold) &&
                sweep_local(sa, sb, q, prl, swl, pA, pB, n, toi)) {
                pA = rotate(pA, qa); pA = pA + pa;
                pB = rotate(pB, qa); pB = pB + pa;
                n = rotate(n, qa);
                pB = pB + toi * (va - vb);
                hit = !(toi > sp.dt) && toi != 0.0f;
                pen = dot(n, pA - pB) * sp.spec_relax;
            }
        }
        int c = warp_append(&w.ctr->ncol, hit);
        if (c >= cap) { atomicCAS(&w.ctr->status, 0, JG_ERR_CAPACITY); c = -1; }
        if (c >= 0) {
            w.col_pair[c] = make_int2(p, 3);
            w.col_res[3 * c + 0] = f4(pA, 0.f);
            w.col_res[3 * c + 1] = f4(pB, 0.f);
            w.col_res[3 * c + 2] = f4(n, pen);
        }
    }
}

// Contact stream record: shape pair, normal with the point count (low byte) and
// JG_STREAM_SPECULATIVE, and the points.
__device__ __forceinline__ void write_stream(WorldDev& w, int idx, int s1, int s2, v3 n, int cnt, bool spec,
                                             const float4* oA, const float4* oB) {
    if (idx >= w.cap_pairs) { atomicCAS(&w.ctr->status, 0, JG_ERR_CAPACITY); return; }
    w.cs_key[idx] = make_int2(s1, s2);
    w.cs_n[idx] = f4(n, __int_as_float(cnt | (spec ? JG_STREAM_SPECULATIVE : 0)));
    for (int k = 0; k < cnt; k++) { w.cs_pa[4 * idx + k] = oA[k]; w.cs_pb[4 * idx + k] = oB[k]; }
}

// A colliding record in world space; a speculative one (kind 3) is there already.
struct ColRec {
    int s1, s2, b1, b2;
    ShapeRef sa, sb;
    q4 qa, qb;
    v3 pa, pb, pA, pB, n;
    float pen;
};
__device__ __forceinline__ void load_record(const WorldDev& w, int c, int2 cp, ColRec& r) {
    const int2 pr = w.pairs[cp.x];
    r.s1 = pr.x; r.s2 = pr.y;
    r.sa = load_shape(w, r.s1); r.sb = load_shape(w, r.s2);
    r.b1 = w.sinfo[r.s1].y; r.b2 = w.sinfo[r.s2].y;
    r.qa = mkq(w.q[r.b1]); r.qb = mkq(w.q[r.b2]);
    r.pa = mk3(w.pos[r.b1]); r.pb = mk3(w.pos[r.b2]);
    r.pA = mk3(w.col_res[3 * c + 0]); r.pB = mk3(w.col_res[3 * c + 1]);
    const float4 nr = w.col_res[3 * c + 2];
    r.n = mk3(nr);
    r.pen = nr.w;
}
__device__ __forceinline__ void record_to_world(ColRec& r) {
    r.pA = rotate(r.pA, r.qa); r.pA = r.pA + r.pa;
    r.pB = rotate(r.pB, r.qa); r.pB = r.pB + r.pa;
    r.n = rotate(r.n, r.qa);
}
// A triangle of a body that is not dynamic against another kind of shape: the triangle-edge
// filter decides about the record.
__device__ __forceinline__ bool edge_filtered(const WorldDev& w, const StepParams& sp, const ColRec& r) {
    const bool c1 = r.sa.kind == JG_SHAPE_TRIANGLE, c2 = r.sb.kind == JG_SHAPE_TRIANGLE;
    return sp.edge_filter && c1 != c2 && w.binfo[c1 ? r.b1 : r.b2].x != JG_MOTION_DYNAMIC;
}
__device__ __forceinline__ int edge_test(const WorldDev& w, const ColRec& r, v3& tn, v3& nn) {
    const bool c1 = r.sa.kind == JG_SHAPE_TRIANGLE;
    return edge_evaluate(w, c1 ? r.sa.tri : r.sb.tri, c1 ? r.qa : r.qb, c1 ? r.pa : r.pb, !c1, c1 ? r.pA : r.pB, r.n, tn, nn);
}

// Stage 2, one thread per record that EPA does not change: the first test of the triangle-edge
// filter (TriangleEdgeCollisionFilter.cs:183-240).  Records near a mesh edge go to the warps of
// stage 3, discarded ones are struck out.  Not launched without triangles.
__global__ void __launch_bounds__(128) k_edge_list(WorldDev w, StepParams sp) {
    const int ncol = min(w.ctr->ncol, w.cap_arb);
    for (int base = blockIdx.x * blockDim.x; base < ncol; base += gridDim.x * blockDim.x) {
        const int c = base + threadIdx.x;
        bool to_edge = false;
        if (c < ncol) {
            const int2 cp = w.col_pair[c];
            const int2 pr = w.pairs[cp.x];
            if (cp.y != 2 && (w.sinfo[pr.x].x == JG_SHAPE_TRIANGLE || w.sinfo[pr.y].x == JG_SHAPE_TRIANGLE)) {
                ColRec r;
                load_record(w, c, cp, r);
                if (edge_filtered(w, sp, r)) {
                    if (cp.y != 3) record_to_world(r);
                    v3 tn, nn;
                    const int ev = edge_test(w, r, tn, nn);
                    to_edge = ev == EDGE;
                    if (ev != KEEP) w.col_pair[c].y = to_edge ? cp.y | COL_EDGE : 0;
                }
            }
        }
        const int e = warp_append(&w.ctr->nedge, to_edge);
        if (e >= 0) w.edge_list[e] = c;
    }
}

// The rest of the triangle-edge filter for a record near a mesh edge: normal snapping
// (TriangleEdgeCollisionFilter.cs:294-420); false when the record is discarded.
__device__ __noinline__ bool edge_snap(ColRec& r, bool spec, v3 tn, v3 nn) {
    v3 &pA = r.pA, &pB = r.pB, &n = r.n;
    v3 mid = 0.5f * (pA + pB);
    if (dot(tn, nn) > 0.999f) {
        float f5 = dot(n, nn), f6 = dot(n, tn);
        if (!spec) pA = pB = mid;
        n = f5 > f6 ? nn : tn;
        return true;
    }
    v3 cr = cross(nn, tn);
    float crl = len2(cr);
    v3 proj = n - (dot(cr, n) / crl) * cr;
    if (len2(proj) < 0.5f * 0.5f) return false;
    float f1 = dot(cross(proj, nn), cr);
    float f2 = dot(cross(proj, tn), cr);
    bool between = f1 <= 0.0f && f2 >= 0.0f;
    if (!between) {
        float f3 = dot(n, nn), f4v = dot(n, tn);
        if (!spec) pA = pB = mid;
        n = f3 > f4v ? nn : tn;
    }
    return true;
}
// The manifold of a record in world space and its contact stream record, by the whole warp.
__device__ __noinline__ void warp_contact(WorldDev& w, const StepParams& sp, EpaSmem& E, const ColRec& r, bool from_sweep, int& pts) {
    v3 oA[4], oB[4];
    int cnt;
    if (sp.aux_contacts && !from_sweep) cnt = build_manifold(E, r.sa, r.sb, r.qa, r.qb, r.pa, r.pb, r.pA, r.pB, r.n, oA, oB);
    else { cnt = 1; oA[0] = r.pA; oB[0] = r.pB; }
    if ((threadIdx.x & 31) == 0) {
        int idx = atomicAdd(&w.ctr->nstream, 1);
        float4 fa[4], fb[4];
        for (int k = 0; k < cnt; k++) { fa[k] = f4(oA[k], 0.f); fb[k] = f4(oB[k], 0.f); }
        write_stream(w, idx, r.s1, r.s2, r.n, cnt, from_sweep, fa, fb);
    }
    pts += cnt;
}

// Next work item of a warp: lane 0 takes it from the cursor, every lane gets it.
__device__ __forceinline__ int next_item(int* cursor, int lane) {
    int e = 0;
    if (lane == 0) e = atomicAdd(cursor, 1);
    return __shfl_sync(0xffffffffu, e, 0);
}

// Stage 3, one warp per deep pair and per record near a mesh edge.  A deep pair: EPA from the
// saved portal (NarrowPhase.cs:39-95); on success the record takes the EPA result, otherwise the
// MPR result stands; then the triangle-edge filter, as in stage 2.  A record near an edge: MPR
// and EPA again with threshold zero (for a deep pair that is what EPA has just returned, and is
// counted but not repeated), then edge_snap.  The manifolds are left to stage 4 (in here a warp's
// manifold, 60 KB of code, cost 84 us on the 100k pile and 30 on the 20k one), unless the colliding
// records are no more than `few`: then the warps take all of them.
// Both kinds of work are searches of very different lengths, and a launch for each ended in a few
// warps twice.  What bounds a full GPU is instruction fetch (half of the cycles between two
// instructions of a warp on the 100k pile) and the FP64 pipe, so rare and repeated code is kept in
// one copy, out of line; as many CTAs as shared memory holds.  Two launches -> one, in ms: a
// pile of 700 0.40 -> 0.24, of 20k 0.53 -> 0.33, of 100k 0.95 -> 0.82, 4096 worlds 1.93 -> 1.69;
// with the manifolds of many records in stage 4, 0.30 and 0.73 on the two larger piles.
__global__ void __launch_bounds__(NP_WARPS * 32) k_deep(WorldDev w, StepParams sp, int few) {
    extern __shared__ __align__(16) unsigned char np_smem_raw[];
    EpaSmem* smem = reinterpret_cast<EpaSmem*>(np_smem_raw);
    const int lane = threadIdx.x & 31;
    EpaSmem& E = smem[threadIdx.x >> 5];
    NpStats st; st.exact = 0;
    int epa_calls = 0, epa_fail = 0, pts = 0;
    const int ncol = min(w.ctr->ncol, w.cap_arb), ne = min(w.ctr->nepa_list, w.cap_arb), nk = ne + min(w.ctr->nedge, w.cap_arb);
    const bool all = ncol <= few;
    const int total = nk + (all ? ncol : 0);
    // handed out one at a time: the cost varies by an order of magnitude between pairs, so a fixed
    // share per warp would leave most warps idle behind a few
    for (int e = next_item(&w.ctr->epa_next, lane); e < total; e = next_item(&w.ctr->epa_next, lane)) {
        const bool deep = e < ne;
        const int c = deep ? w.epa_list[e] : (e < nk ? w.edge_list[e - ne] : e - nk);
        const int2 cp = w.col_pair[c];
        if (e >= nk && (cp.y == 0 || cp.y == 2 || cp.y >= COL_EDGE)) continue;  // in the lists, or struck out
        const bool from_sweep = (cp.y & ~COL_EDGE) == 3;
        ColRec r;
        load_record(w, c, cp, r);
        const bool spec = !deep && r.pen < 0.0f;
        v3 tn = mk3(0.f), nn = mk3(0.f);
        int ev = KEEP;
        if (deep) {
            MV portal[4];
            for (int k = 0; k < 4; k++) {
                portal[k].V = mk3(w.col_portal[12 * e + 3 * k + 0]);
                portal[k].A = mk3(w.col_portal[12 * e + 3 * k + 1]);
                portal[k].B = mk3(w.col_portal[12 * e + 3 * k + 2]);
            }
            const int exact = st.exact, fail = epa_fail;
            run_epa(E, r.sa, r.sb, qmul(qconj(r.qa), r.qb), rotate_inv(r.pb - r.pa, r.qa), portal, r.pA, r.pB, r.n, r.pen, st,
                    epa_calls, epa_fail);
            record_to_world(r);
            if (edge_filtered(w, sp, r)) ev = edge_test(w, r, tn, nn);
            if (ev == DISCARD) {
                if (lane == 0) w.col_pair[c].y = 0;
                continue;
            }
            if (ev == EDGE) {
                epa_calls++;
                epa_fail += epa_fail - fail;
                st.exact += st.exact - exact;
            }
        } else if (e >= nk) {
            if (!from_sweep) record_to_world(r);
        } else {
            if (!from_sweep) record_to_world(r);
            ev = edge_test(w, r, tn, nn);
            if (!spec) {
                if (!mpr_epa_world(E, r.sa, r.sb, r.qa, r.qb, r.pa, r.pb, r.pA, r.pB, r.n, r.pen, 0.0f, st, epa_calls, epa_fail)) continue;
                ev = edge_test(w, r, tn, nn);
                if (ev == DISCARD) continue;
            }
        }
        if (ev != KEEP && !edge_snap(r, spec, tn, nn)) {
            if (lane == 0) w.col_pair[c].y = 0;
            continue;
        }
        if (all) warp_contact(w, sp, E, r, from_sweep, pts);
        else if (lane == 0) {
            w.col_res[3 * c + 0] = f4(r.pA, 0.f);
            w.col_res[3 * c + 1] = f4(r.pB, 0.f);
            w.col_res[3 * c + 2] = f4(r.n, r.pen);
            w.col_pair[c].y = from_sweep ? 3 : COL_WORLD;
        }
    }
    if (lane == 0) {
        if (epa_calls) atomicAdd(&w.ctr->nepa, epa_calls);
        if (epa_fail) atomicAdd(&w.ctr->epa_fail, epa_fail);
        if (pts) atomicAdd(&w.ctr->points, pts);
    }
    int ex = st.exact;
    for (int off = 16; off > 0; off >>= 1) ex += __shfl_xor_sync(FULL, ex, off);
    if (lane == 0 && ex) atomicAdd(&w.ctr->exact, ex);
}

// Stage 4, one thread per record that is left: the one-shot manifold; appends the contact
// stream record.  A speculative record registers its one point (World.Detect.cs:185-196).
__global__ void __launch_bounds__(128) k_manifold(WorldDev w, StepParams sp, int few) {
    const int ncol = min(w.ctr->ncol, w.cap_arb);
    if (ncol <= few) return;  // stage 3 has done them
    int pts = 0;
    for (int base = blockIdx.x * blockDim.x; base < ncol; base += gridDim.x * blockDim.x) {
        const int c = base + threadIdx.x;
        const int2 cp = c < ncol ? w.col_pair[c] : make_int2(0, 0);
        const bool emit = cp.y > 0 && cp.y < COL_EDGE, spec = cp.y == 3;  // (3 and COL_WORLD are in world space)
        int cnt = 0;
        ColRec r;
        float4 oA[4], oB[4];
        if (emit) {
            load_record(w, c, cp, r);
            if (cp.y < 3) record_to_world(r);
            if (sp.aux_contacts && !spec) cnt = manifold_thread(r.sa, r.sb, r.qa, r.qb, r.pa, r.pb, r.pA, r.pB, r.n, oA, oB);
            else { cnt = 1; oA[0] = f4(r.pA, 0.f); oB[0] = f4(r.pB, 0.f); }
        }
        int idx = warp_append(&w.ctr->nstream, emit);
        if (idx >= 0) { write_stream(w, idx, r.s1, r.s2, r.n, cnt, spec, oA, oB); pts += cnt; }
    }
    for (int off = 16; off > 0; off >>= 1) pts += __shfl_xor_sync(FULL, pts, off);
    if ((threadIdx.x & 31) == 0 && pts) atomicAdd(&w.ctr->points, pts);
}

// Batched NarrowPhase.MprEpa query (NarrowPhase.cs:902-927) on the world's shapes and body poses.
// out holds 10 floats per pair (pointA, pointB, normal, penetration, world frame) and hit the
// method's return value; every slot is written, so neither buffer needs clearing.  Few pairs
// take one launch with a warp per pair; many the two stages of a step, MPR with one thread per pair
// (a warp per pair runs all its 32 lanes through the same arithmetic), then EPA with one warp per
// deep pair.  The deep pairs go through the world's EPA list and portals, free between steps.
// 30,001 pairs, mostly deep: 1773 us of kernels with a warp per pair, 780 in two stages.
__device__ __forceinline__ void write_query(float* o, v3 pA, v3 pB, v3 n, float pen, q4 qa, v3 pa) {
    pA = rotate(pA, qa); pA = pA + pa;
    pB = rotate(pB, qa); pB = pB + pa;
    n = rotate(n, qa);
    o[0] = pA.x; o[1] = pA.y; o[2] = pA.z;
    o[3] = pB.x; o[4] = pB.y; o[5] = pB.z;
    o[6] = n.x; o[7] = n.y; o[8] = n.z;
    o[9] = pen;
}
__global__ void __launch_bounds__(NP_WARPS * 32) k_collide_query(WorldDev w, const int2* pairs, int n, float threshold,
                                                                 float* out, int* hit) {
    extern __shared__ __align__(16) unsigned char np_smem_raw[];
    EpaSmem* smem = reinterpret_cast<EpaSmem*>(np_smem_raw);
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    EpaSmem& E = smem[wib];
    NpStats st; st.exact = 0;
    int ec = 0, ef = 0;
    for (int i = blockIdx.x * NP_WARPS + wib; i < n; i += gridDim.x * NP_WARPS) {
        int2 pr = pairs[i];
        ShapeRef sa = load_shape(w, pr.x), sb = load_shape(w, pr.y);
        int b1 = w.sinfo[pr.x].y, b2 = w.sinfo[pr.y].y;
        q4 qa = mkq(w.q[b1]), qb = mkq(w.q[b2]);
        v3 pa = mk3(w.pos[b1]), pb = mk3(w.pos[b2]);
        v3 pA = mk3(0.f), pB = mk3(0.f), nn = mk3(0.f);
        float pen = 0.f;
        const bool h = solve_mpr(E, sa, sb, qmul(qconj(qa), qb), rotate_inv(pb - pa, qa), threshold, pA, pB, nn, pen, st, ec, ef);
        if (lane == 0) {
            write_query(out + 10 * (size_t)i, pA, pB, nn, pen, qa, pa);
            hit[i] = h ? 1 : 0;
        }
    }
}

__global__ void __launch_bounds__(128, 4) k_query_mpr(WorldDev w, const int2* pairs, int n, bool grouped, float threshold,
                                                   float* out, int* hit) {
    if (n <= 0) return;
    mpr_lanes<true>(
        n, threshold,
        [&](int q, ShapeRef& sa, ShapeRef& sb, q4& rot, v3& rel) {
            const int2 pr = pairs[grouped ? w.pair_order[q] : q];
            sa = load_shape(w, pr.x);
            sb = load_shape(w, pr.y);
            const int b1 = w.sinfo[pr.x].y, b2 = w.sinfo[pr.y].y;
            const q4 qa = mkq(w.q[b1]);
            rot = qmul(qconj(qa), mkq(w.q[b2]));
            rel = rotate_inv(mk3(w.pos[b2]) - mk3(w.pos[b1]), qa);
            return b1;
        },
        [&](bool done, int code, int q, int b1, const Mpr& M, const ShapeRef& sa, const ShapeRef& sb, q4 rot, v3 rel) {
            const int i = done ? (grouped ? w.pair_order[q] : q) : 0;
            if (done) {
                hit[i] = code != 0;
                if (code != 2) write_query(out + 10 * (size_t)i, M.pA, M.pB, M.normal, M.pen, mkq(w.q[b1]), mk3(w.pos[b1]));
            }
            const int e = warp_append(&w.qctl[0], done && code == 2);
            if (e >= 0) {
                w.epa_list[e] = i;
                w.col_res[3 * e + 0] = f4(M.pA, 0.f);
                w.col_res[3 * e + 1] = f4(M.pB, 0.f);
                w.col_res[3 * e + 2] = f4(M.normal, M.pen);
                save_portal(w, e, M, sa, sb, rot, rel);
            }
        });
}
__global__ void __launch_bounds__(NP_WARPS * 32) k_query_epa(WorldDev w, const int2* pairs, float* out) {
    extern __shared__ __align__(16) unsigned char np_smem_raw[];
    EpaSmem* smem = reinterpret_cast<EpaSmem*>(np_smem_raw);
    const int lane = threadIdx.x & 31;
    EpaSmem& E = smem[threadIdx.x >> 5];
    NpStats st; st.exact = 0;
    int ec = 0, ef = 0;
    const int ne = w.qctl[0];
    for (int e = next_item(&w.qctl[1], lane); e < ne; e = next_item(&w.qctl[1], lane)) {
        const int i = w.epa_list[e];
        const int2 pr = pairs[i];
        ShapeRef sa = load_shape(w, pr.x), sb = load_shape(w, pr.y);
        const int b1 = w.sinfo[pr.x].y, b2 = w.sinfo[pr.y].y;
        const q4 qa = mkq(w.q[b1]), qb = mkq(w.q[b2]);
        const v3 pa = mk3(w.pos[b1]), pb = mk3(w.pos[b2]);
        MV portal[4];
        for (int k = 0; k < 4; k++) {
            portal[k].V = mk3(w.col_portal[12 * e + 3 * k + 0]);
            portal[k].A = mk3(w.col_portal[12 * e + 3 * k + 1]);
            portal[k].B = mk3(w.col_portal[12 * e + 3 * k + 2]);
        }
        v3 pA = mk3(w.col_res[3 * e + 0]), pB = mk3(w.col_res[3 * e + 1]);
        const float4 nr = w.col_res[3 * e + 2];
        v3 n = mk3(nr);
        float pen = nr.w;
        run_epa(E, sa, sb, qmul(qconj(qa), qb), rotate_inv(pb - pa, qa), portal, pA, pB, n, pen, st, ec, ef);
        if (lane == 0) write_query(out + 10 * (size_t)i, pA, pB, n, pen, qa, pa);
    }
}

// Batched CollisionManifold.BuildManifold (CollisionManifold.cs:393-566) for given witness
// points, one thread per pair, the same function the step's manifold stage runs.  in holds
// 9 floats per pair (pointA, pointB, normal, world frame); out receives 24 floats per pair
// (up to four point pairs A, B) and count the number of pairs.
__global__ void __launch_bounds__(128) k_manifold_query(WorldDev w, const int2* pairs, int n, const float* in, float* out,
                                                        int* count) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int2 pr = pairs[i];
        ShapeRef sa = load_shape(w, pr.x), sb = load_shape(w, pr.y);
        int b1 = w.sinfo[pr.x].y, b2 = w.sinfo[pr.y].y;
        q4 qa = mkq(w.q[b1]), qb = mkq(w.q[b2]);
        v3 pa = mk3(w.pos[b1]), pb = mk3(w.pos[b2]);
        const float* c = in + 9 * (size_t)i;
        float4 oA[4], oB[4];
        int cnt = manifold_thread(sa, sb, qa, qb, pa, pb, mk3(c[0], c[1], c[2]), mk3(c[3], c[4], c[5]), mk3(c[6], c[7], c[8]),
                                  oA, oB);
        float* o = out + 24 * (size_t)i;
        for (int k = 0; k < 4; k++) {
            float4 a = k < cnt ? oA[k] : make_float4(0.f, 0.f, 0.f, 0.f), b = k < cnt ? oB[k] : make_float4(0.f, 0.f, 0.f, 0.f);
            o[6 * k + 0] = a.x; o[6 * k + 1] = a.y; o[6 * k + 2] = a.z;
            o[6 * k + 3] = b.x; o[6 * k + 4] = b.y; o[6 * k + 5] = b.z;
        }
        count[i] = cnt;
    }
}

// Dynamic shared memory of the warp-per-pair kernels: one polytope per warp.
constexpr int kNpSmem = NP_WARPS * (int)sizeof(EpaSmem);

}  // namespace

// Lets the warp-per-pair kernels take their polytopes' shared memory (above the 48 KB
// default) on the current device; called when a world is created.
int jg_narrowphase_init() {
    cudaError_t e = cudaFuncSetAttribute(k_deep, cudaFuncAttributeMaxDynamicSharedMemorySize, kNpSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_collide_query, cudaFuncAttributeMaxDynamicSharedMemorySize, kNpSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_query_epa, cudaFuncAttributeMaxDynamicSharedMemorySize, kNpSmem);
    return e == cudaSuccess ? 0 : -1;
}

void jg_launch_manifold_query(WorldDev& w, const int2* pairs, int n, const float* in, float* out, int* count,
                              cudaStream_t s, int nsm) {
    if (n <= 0) return;
    int blocks = (n + 127) / 128;
    if (blocks > nsm * 8) blocks = nsm * 8;
    k_manifold_query<<<blocks, 128, 0, s>>>(w, pairs, n, in, out, count);
}

void jg_launch_collide_query(WorldDev& w, const int2* pairs, int n, float threshold, float* out, int* hit,
                             cudaStream_t s, int nsm) {
    if (n <= 0) return;
    // the stages take as many pairs at a time as the world's lists hold deep ones
    const int chunk = w.cap_arb < w.cap_pairs ? w.cap_arb : w.cap_pairs, few = nsm * 12 * NP_WARPS;
    // up to three pairs a warp: 1 pair 35 us a call (two stages 45), 1000 pairs 424 (472), 6000
    // 954 (976), 12000 1043 (866).  So where lists that hold no more would make several chunks, each of which
    // ends in its longest pair alone: 200,000 pairs with lists of 1,024 40.5 ms in chunks and 10.0 in one
    // launch, 30,000 with lists of 4,096 2.5 and 1.9; 12,000 (three chunks) 1.01 and 1.06.
    if (n <= few || (chunk <= few && n > 3 * chunk)) {
        const int blocks = (n + NP_WARPS - 1) / NP_WARPS;
        k_collide_query<<<blocks < nsm * 4 ? blocks : nsm * 4, NP_WARPS * 32, kNpSmem, s>>>(w, pairs, n, threshold, out, hit);
        return;
    }
    for (int first = 0; first < n; first += chunk) {
        const int m = n - first < chunk ? n - first : chunk;
        const int2* pr = pairs + first;
        const bool grouped = m >= 4096;  // (two launches: not for a last short chunk)
        cudaMemsetAsync(w.qctl, 0, sizeof(int) * 2, s);
        if (grouped) {
            cudaMemsetAsync(w.pair_kind, 0, sizeof(int) * 128, s);
            const int blocks = (m + 255) / 256 < nsm * 4 ? (m + 255) / 256 : nsm * 4;
            k_pair_hist<<<blocks, 256, 0, s>>>(w, PairList{pr, m});
            k_pair_scatter<<<blocks, 256, 0, s>>>(w, PairList{pr, m});
        }
        k_query_mpr<<<nsm * 4, 128, 0, s>>>(w, pr, m, grouped, threshold, out + 10 * (size_t)first, hit + first);
        const int blocks = (m + NP_WARPS - 1) / NP_WARPS;
        k_query_epa<<<blocks < nsm * 4 ? blocks : nsm * 4, NP_WARPS * 32, kNpSmem, s>>>(w, pr, out + 10 * (size_t)first);
    }
}

void jg_launch_narrowphase(WorldDev& w, const StepParams& p, cudaStream_t s, int nsm, int tile) {
    (void)tile;
    cudaMemsetAsync(w.pair_kind, 0, sizeof(int) * 128, s);
    k_pair_hist<<<nsm * 4, 256, 0, s>>>(w, PairList{nullptr, 0});
    k_pair_scatter<<<nsm * 4, 256, 0, s>>>(w, PairList{nullptr, 0});
    k_mpr<<<nsm * 2, 256, 0, s>>>(w);
    k_sweep<<<nsm * 2, 128, 0, s>>>(w, p);
    if (w.ntris > 0 && p.edge_filter) k_edge_list<<<nsm * 8, 128, 0, s>>>(w, p);
    const int few = WARP_RECORDS * nsm * 3 * NP_WARPS;
    k_deep<<<nsm * 3, NP_WARPS * 32, kNpSmem, s>>>(w, p, few);
    k_manifold<<<nsm * 16, 128, 0, s>>>(w, p, few);
}
