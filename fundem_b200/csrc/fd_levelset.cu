// fd_levelset.cu -- level-set templates on the GPU: the signed-distance grid of
// an analytic shape or of a closed triangle mesh, one thread per grid node.
//
// The reference builds these grids on the host, one virtual call per node
// (kernel/helper/LevelSetObjectGenerator.h:122-224, Base::buildGrid).  Each
// node stores f / |grad f| when |grad f| > 1e-12, else +-h/2 by the sign of f.
// The implicit functions follow the reference classes:
//   Superellipsoid  LevelSetObjectGenerator.h:1264-1354
//   Sphere          :1628-1661
//   BoxWall         :1781-1867
//   CylinderWall    :2050-2131 (its end-cap gradient is the unnormalised axis
//                   vector, so grid values there are divided by the axis length)
//   triangle mesh   :888-953 (closest point over all triangles, sign by the
//                   winding number |sum of solid angles / 4 pi| > 0.5)
// This file is compiled with -fmad=false: every add and multiply rounds on its
// own as in the reference's host code, so the grids differ from a host build
// only where CUDA's pow and atan2 round differently from the host library.
#include <cfloat>
#include <cmath>

#include "fundem_b200.h"

namespace {

struct Vec { double x, y, z; };

__device__ __forceinline__ Vec mk(double x, double y, double z) { return Vec{x, y, z}; }
__device__ __forceinline__ Vec operator+(Vec a, Vec b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ Vec operator-(Vec a, Vec b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ Vec operator-(Vec a) { return mk(-a.x, -a.y, -a.z); }
__device__ __forceinline__ Vec operator*(double s, Vec a) { return mk(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ Vec operator*(Vec a, double s) { return mk(a.x * s, a.y * s, a.z * s); }
// vector / scalar multiplies by the reciprocal, as the reference's double3 does (myVec.h:55-59)
__device__ __forceinline__ Vec operator/(Vec a, double s)
{
    const double inv = 1.0 / s;
    return mk(a.x * inv, a.y * inv, a.z * inv);
}
__device__ __forceinline__ double dot(Vec a, Vec b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ Vec cross(Vec a, Vec b)
{
    return mk(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double len(Vec a) { return sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }
// host-side normalisation of the reference (myVec.h:121-137): v * (1 / sqrt(|v|^2)), zero below 1e-20
__device__ __forceinline__ Vec unit(Vec v)
{
    const double l2 = v.x * v.x + v.y * v.y + v.z * v.z;
    if (fabs(l2) <= 1.0e-20) return mk(0.0, 0.0, 0.0);
    const double inv = 1.0 / sqrt(l2);
    return mk(v.x * inv, v.y * inv, v.z * inv);
}
__device__ __forceinline__ double sign_no_zero(double v) { return v >= 0.0 ? 1.0 : -1.0; }

struct Shape {
    int kind;
    int flip;  // positive inside: value and gradient negated
    double p[8];
};

// Superellipsoid |x/rx|^(2/ee) + |y/ry|^(2/ee))^(ee/en) + |z/rz|^(2/en) - 1 and its gradient
__device__ void eval_superellipsoid(const double* p, Vec x, double& f, Vec& g)
{
    const double rx = p[0], ry = p[1], rz = p[2], ee = p[3], en = p[4];
    const double ix = 1.0 / rx, iy = 1.0 / ry, iz = 1.0 / rz;
    const double ax = fabs(x.x * ix), ay = fabs(x.y * iy), az = fabs(x.z * iz);
    const double exy = 2.0 / ee, ez = 2.0 / en, eo = ee / en;
    const double sxy = pow(fabs(ax), exy) + pow(fabs(ay), exy);
    f = pow(fabs(sxy), eo) + pow(fabs(az), ez) - 1.0;
    const double tiny = 1e-30;
    const double outer = pow(fabs(fmax(sxy, tiny)), eo - 1.0);
    const double dsx = exy * pow(fabs(fmax(ax, tiny)), exy - 1.0) * sign_no_zero(x.x) * ix;
    const double dsy = exy * pow(fabs(fmax(ay, tiny)), exy - 1.0) * sign_no_zero(x.y) * iy;
    const double dz = ez * pow(fabs(fmax(az, tiny)), ez - 1.0) * sign_no_zero(x.z) * iz;
    g = mk(eo * outer * dsx, eo * outer * dsy, dz);
}

__device__ void eval_sphere(const double* p, Vec x, double& f, Vec& g)
{
    const double d = len(x);
    f = d - p[0];
    if (d > 1e-30) g = x / d;  // at the centre the gradient stays zero
}

__device__ void eval_box(const double* p, Vec x, double& f, Vec& g)
{
    const Vec hb = mk(0.5 * p[0], 0.5 * p[1], 0.5 * p[2]);
    const Vec q = mk(fabs(x.x) - hb.x, fabs(x.y) - hb.y, fabs(x.z) - hb.z);
    const Vec qo = mk(fmax(q.x, 0.0), fmax(q.y, 0.0), fmax(q.z, 0.0));
    const double out = len(qo);
    const double in = fmin(fmax(q.x, fmax(q.y, q.z)), 0.0);
    f = out + in;
    if (out > 1e-30) {
        g = qo / out;
        if (x.x < 0.0 && q.x > 0.0) g.x = -g.x;
        if (x.y < 0.0 && q.y > 0.0) g.y = -g.y;
        if (x.z < 0.0 && q.z > 0.0) g.z = -g.z;
    } else {
        // inside: the normal of the nearest face
        const double fx = hb.x - fabs(x.x), fy = hb.y - fabs(x.y), fz = hb.z - fabs(x.z);
        if (fx <= fy && fx <= fz) g = mk(x.x >= 0.0 ? 1.0 : -1.0, 0.0, 0.0);
        else if (fy <= fx && fy <= fz) g = mk(0.0, x.y >= 0.0 ? 1.0 : -1.0, 0.0);
        else g = mk(0.0, 0.0, x.z >= 0.0 ? 1.0 : -1.0);
    }
}

// capped cylinder between points A (p[0..2]) and B (p[3..5]) of radius p[6]
__device__ void eval_cylinder(const double* p, Vec x, double& f, Vec& g)
{
    const Vec A = mk(p[0], p[1], p[2]), B = mk(p[3], p[4], p[5]);
    const double r = p[6];
    const Vec axis = B - A;
    const double L = len(axis);
    const Vec dir = axis / L;
    const Vec rel = x - A;
    const double s = dot(rel, dir);
    const double sc = fmax(0.0, fmin(s, L));
    const Vec on_axis = A + sc * dir;
    const bool in_radius = len(cross(rel, dir)) <= r;
    const bool in_length = s >= 0.0 && s <= L;
    const bool near_a = s < 0.5 * L;
    if (in_radius && in_length) {
        const Vec radial = x - on_axis;
        const double rs = len(radial) - r;
        const double as = near_a ? -s : s - L;
        if (fabs(rs) <= fabs(as)) {
            f = rs;
            g = unit(radial);
        } else {
            f = as;
            g = near_a ? -axis : axis;
        }
    } else if (!in_radius && in_length) {
        const Vec radial = x - on_axis;
        f = len(radial) - r;
        g = unit(radial);
    } else if (!in_radius && !in_length) {
        const Vec rim = on_axis + unit(rel - s * dir) * r;
        f = len(x - rim);
        g = unit(x - rim);
    } else {
        f = s < 0.0 ? -s : s - L;
        g = s < 0.0 ? -axis : axis;
    }
}

__device__ __forceinline__ double grid_value(double f, Vec g, double h)
{
    const double gn = len(g);
    if (gn > 1e-12) return f / gn;
    return (f <= 0.0 ? -1.0 : 1.0) * 0.5 * h;
}

__device__ __forceinline__ Vec node_point(double3 o, double h, long long id, int3 n)
{
    const int i = (int)(id % n.x);
    const int j = (int)((id / n.x) % n.y);
    const int k = (int)(id / ((long long)n.x * n.y));
    return mk(o.x + double(i) * h, o.y + double(j) * h, o.z + double(k) * h);
}

__global__ void k_levelset_analytic(Shape s, double3 o, double h, int3 n, long long total, double* __restrict__ out)
{
    for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < total;
         id += (long long)gridDim.x * blockDim.x) {
        const Vec x = node_point(o, h, id, n);
        double f = 0.0;
        Vec g = mk(0.0, 0.0, 0.0);
        switch (s.kind) {
        case FUNDEM_SHAPE_SUPERELLIPSOID: eval_superellipsoid(s.p, x, f, g); break;
        case FUNDEM_SHAPE_SPHERE: eval_sphere(s.p, x, f, g); break;
        case FUNDEM_SHAPE_BOX: eval_box(s.p, x, f, g); break;
        default: eval_cylinder(s.p, x, f, g); break;
        }
        if (s.flip) { f = -f; g = -g; }
        out[id] = grid_value(f, g, h);
    }
}

// closest point of triangle abc to p: the Voronoi-region walk of Ericson,
// "Real-Time Collision Detection" (2005), section 5.1.5
__device__ __forceinline__ Vec closest_on_triangle(Vec p, Vec a, Vec b, Vec c)
{
    const Vec ab = b - a, ac = c - a, ap = p - a;
    const double d1 = dot(ab, ap), d2 = dot(ac, ap);
    if (d1 <= 0.0 && d2 <= 0.0) return a;
    const Vec bp = p - b;
    const double d3 = dot(ab, bp), d4 = dot(ac, bp);
    if (d3 >= 0.0 && d4 <= d3) return b;
    const double vc = d1 * d4 - d3 * d2;
    if (vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0) return a + (d1 / (d1 - d3)) * ab;
    const Vec cp = p - c;
    const double d5 = dot(ab, cp), d6 = dot(ac, cp);
    if (d6 >= 0.0 && d5 <= d6) return c;
    const double vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) return a + (d2 / (d2 - d6)) * ac;
    const double va = d3 * d6 - d5 * d4;
    if (va <= 0.0 && (d4 - d3) >= 0.0 && (d5 - d6) >= 0.0)
        return b + ((d4 - d3) / ((d4 - d3) + (d5 - d6))) * (c - b);
    const double inv = 1.0 / (va + vb + vc);
    return a + ab * (vb * inv) + ac * (vc * inv);
}

// signed solid angle of triangle abc seen from p (Van Oosterom and Strackee, 1983)
__device__ __forceinline__ double solid_angle(Vec p, Vec a, Vec b, Vec c)
{
    const Vec r0 = a - p, r1 = b - p, r2 = c - p;
    const double l0 = len(r0), l1 = len(r1), l2 = len(r2);
    if (l0 < 1e-30 || l1 < 1e-30 || l2 < 1e-30) return 0.0;
    const double num = dot(r0, cross(r1, r2));
    const double den = l0 * l1 * l2 + dot(r0, r1) * l2 + dot(r1, r2) * l0 + dot(r2, r0) * l1;
    return 2.0 * atan2(num, den);
}

// A triangle for the screening passes, in single precision about the grid's
// centre and in units of the whole extent (so that no length over- or
// underflows): corners, centroid, and the radius of its corners about the centroid
// (infinite for slivers, whose exact closest point may be badly rounded:
// those are always evaluated).
struct MeshTri {
    float4 sphere;
    float ax, ay, az, bx, by, bz, cx, cy, cz, pad[3];
};

__global__ void k_mesh_prepare(const double* __restrict__ tri, int ntri, double3 centre, double unit,
                               MeshTri* __restrict__ out)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    const double* T = tri + 9ll * t;
    const Vec o = mk(centre.x, centre.y, centre.z);
    const Vec a = unit * (mk(T[0], T[1], T[2]) - o), b = unit * (mk(T[3], T[4], T[5]) - o),
              c = unit * (mk(T[6], T[7], T[8]) - o);
    const Vec g = (1.0 / 3.0) * (a + b + c);
    const double edge2 = fmax(dot(b - a, b - a), fmax(dot(c - a, c - a), dot(c - b, c - b)));
    const Vec n = cross(b - a, c - a);
    const double r = sqrt(fmax(dot(a - g, a - g), fmax(dot(b - g, b - g), dot(c - g, c - g))));
    const bool sliver = !(dot(n, n) > 1e-10 * edge2 * edge2);
    MeshTri m;
    m.sphere = make_float4((float)g.x, (float)g.y, (float)g.z,
                           sliver ? __int_as_float(0x7f800000) : __double2float_ru(r));
    m.ax = (float)a.x; m.ay = (float)a.y; m.az = (float)a.z;
    m.bx = (float)b.x; m.by = (float)b.y; m.bz = (float)b.z;
    m.cx = (float)c.x; m.cy = (float)c.y; m.cz = (float)c.z;
    m.pad[0] = m.pad[1] = m.pad[2] = 0.f;
    out[t] = m;
}

// half the solid angle in single precision; exact (double precision) where
// the point lies near the triangle's plane inside it, or near its edges or
// corners, where the angle jumps or is ill-conditioned
__device__ __forceinline__ float half_angle32(float px, float py, float pz, const MeshTri& t, Vec x,
                                              const double* __restrict__ T)
{
    const float ax = t.ax - px, ay = t.ay - py, az = t.az - pz;
    const float bx = t.bx - px, by = t.by - py, bz = t.bz - pz;
    const float cx = t.cx - px, cy = t.cy - py, cz = t.cz - pz;
    const float la = sqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az)));
    const float lb = sqrtf(fmaf(bx, bx, fmaf(by, by, bz * bz)));
    const float lc = sqrtf(fmaf(cx, cx, fmaf(cy, cy, cz * cz)));
    const float num = fmaf(ax, fmaf(by, cz, -bz * cy), fmaf(ay, fmaf(bz, cx, -bx * cz), az * fmaf(bx, cy, -by * cx)));
    const float lll = la * lb * lc;
    const float den = lll + fmaf(fmaf(ax, bx, fmaf(ay, by, az * bz)), lc,
                                 fmaf(fmaf(bx, cx, fmaf(by, cy, bz * cz)), la,
                                      fmaf(cx, ax, fmaf(cy, ay, cz * az)) * lb));
    // lengths are in units of the extent, whose roundings are 6e-8: within 1e-4
    // of a corner the directions to it are too rough
    const float lim = 0.02f * lll;
    if (!(fminf(la, fminf(lb, lc)) > 1e-4f && (fabsf(num) > lim || den > lim)))
        return (float)(0.5 * solid_angle(x, mk(T[0], T[1], T[2]), mk(T[3], T[4], T[5]), mk(T[6], T[7], T[8])));
    return atan2f(num, den);
}

constexpr int MESH_SCREENED = 1 << 22;  // see k_levelset_mesh
constexpr int MESH_WARPS = 4;
constexpr int MESH_BLOCK = 32 * MESH_WARPS;  // also the triangles staged at a time

// 32 grid nodes (8 x 4 x 1) per block, its warps sharing out the triangles.
//
// The distance is the minimum over all triangles and the sign the winding
// number's (a sum of solid angles), in double precision that was three square
// roots, an arc tangent and a closest point for every node and triangle: 4.6
// ms for 48^3 nodes and 2,304 triangles, bound by the double-precision pipe (a
// call, with its copies, 5.1 ms; now 2.6).
// Here single precision screens both, and double precision decides:
//   * pass 1 sums the solid angles in single precision (half_angle32) and finds
//     the triangle of the nearest centroid; its exact distance bounds the
//     minimum;
//   * pass 2 takes the exact closest point of the triangles whose sphere comes
//     within that bound, ties to the first triangle as in a scan in order;
//   * a winding number within a quarter of the 0.5 it is compared with (no
//     closed mesh gives one) is summed again in double precision, in
//     triangle order.
// So every value is the one the double-precision scan gives.
//
// Why a quarter of a turn is enough.  Rounding the coordinates moves each
// vertex and the node by at most 6e-8 of the extent, the same way for all
// triangles: a closed mesh stays closed, and its winding number about the moved
// node differs only where the node changes sides, that is within 2e-7 of the
// surface.  There the triangle it would cross, and those next to an edge or a
// corner it is that close to, fail half_angle32's tests (their angle is near
// pi, or a corner is within 1e-4) and are evaluated exactly.  Of the other
// triangles each term is off by the products' roundings, some 4e-7 of lll,
// against a num or den of at least 0.02 lll: at most 2e-5 for the few that
// subtend a large angle, and some 1e-7 for a triangle whose corners lie close
// together seen from the node (den is about 4 lll there), as all but a few are
// in a mesh of many.  A quarter of a turn is 1.6 in half angles: sixteen
// million such triangles all off the same way.  A mesh of more than
// MESH_SCREENED triangles is summed in double precision.
__global__ void __launch_bounds__(MESH_BLOCK) k_levelset_mesh(const double* __restrict__ tri,
                                                              const MeshTri* __restrict__ mesh, int ntri, int flip,
                                                              double3 o, double h, int3 n, double3 centre, double unit,
                                                              double* __restrict__ out)
{
    __shared__ MeshTri s_tri[MESH_BLOCK];
    __shared__ double s_sum[MESH_WARPS][32], s_d2[MESH_WARPS][32];
    __shared__ float s_near[MESH_WARPS][32];
    __shared__ int s_at[MESH_WARPS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long bx = (n.x + 7) / 8, by = (n.y + 3) / 4;
    const long long blk = blockIdx.x;
    const int i = (int)(blk % bx) * 8 + (lane & 7), j = (int)((blk / bx) % by) * 4 + (lane >> 3);
    const int k = (int)(blk / (bx * by));
    const bool live = i < n.x && j < n.y;
    const Vec x = mk(o.x + double(i) * h, o.y + double(j) * h, o.z + double(k) * h);
    const float px = (float)(unit * (x.x - centre.x)), py = (float)(unit * (x.y - centre.y)),
                pz = (float)(unit * (x.z - centre.z));
    // what the screening's single precision can be off by in a length: a few
    // roundings of coordinates of at most one
    const float slack = 2e-6f;
    auto stage = [&](int t0) {
        __syncthreads();
        const int nt = min(MESH_BLOCK, ntri - t0);
        const float4* src = reinterpret_cast<const float4*>(mesh + t0);
        float4* dst = reinterpret_cast<float4*>(s_tri);
        for (int q = threadIdx.x; q < nt * (int)(sizeof(MeshTri) / sizeof(float4)); q += MESH_BLOCK) dst[q] = src[q];
        __syncthreads();
        return nt;
    };
    // pass 1
    double wsum = 0.0;
    float near2 = __int_as_float(0x7f800000);
    int at = 0;
    for (int t0 = 0; t0 < ntri; t0 += MESH_BLOCK) {
        const int nt = stage(t0);
        float part = 0.f;
        for (int t = 32 * w; t < min(32 * w + 32, nt); ++t) {
            const MeshTri& m = s_tri[t];
            const float dx = m.sphere.x - px, dy = m.sphere.y - py, dz = m.sphere.z - pz;
            const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (d2 < near2) {
                near2 = d2;
                at = t0 + t;
            }
            part += half_angle32(px, py, pz, m, x, tri + 9ll * (t0 + t));
        }
        wsum += (double)part;
    }
    s_sum[w][lane] = wsum;
    s_near[w][lane] = near2;
    s_at[w][lane] = at;
    __syncthreads();
    wsum = 0.0;
    for (int v = 0; v < MESH_WARPS; ++v) {
        wsum += s_sum[v][lane];
        if (s_near[v][lane] < near2 || (s_near[v][lane] == near2 && s_at[v][lane] < at)) {
            near2 = s_near[v][lane];
            at = s_at[v][lane];
        }
    }
    // pass 2
    double best = DBL_MAX;
    int best_at = 0x7fffffff;
    Vec near = x;
    float reach = __int_as_float(0x7f800000);
    auto exact = [&](int t) {
        const double* T = tri + 9ll * t;
        const Vec q = closest_on_triangle(x, mk(T[0], T[1], T[2]), mk(T[3], T[4], T[5]), mk(T[6], T[7], T[8]));
        const Vec dq = x - q;
        const double d2 = dot(dq, dq);
        if (d2 < best || (d2 == best && t < best_at)) {
            best = d2;
            best_at = t;
            near = q;
            reach = __double2float_ru(unit * sqrt(d2)) + slack;
        }
    };
    exact(at);
    for (int t0 = 0; t0 < ntri; t0 += MESH_BLOCK) {
        const int nt = stage(t0);
        for (int t = 32 * w; t < min(32 * w + 32, nt); ++t) {
            const float4 c = s_tri[t].sphere;
            const float dx = c.x - px, dy = c.y - py, dz = c.z - pz;
            const float far = (reach + c.w) * 1.00001f;
            if (!(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > far * far) && t0 + t != at) exact(t0 + t);
        }
    }
    s_d2[w][lane] = best;
    s_at[w][lane] = best_at;
    __syncthreads();
    int owner = 0;
    for (int v = 1; v < MESH_WARPS; ++v)
        if (s_d2[v][lane] < s_d2[owner][lane] ||
            (s_d2[v][lane] == s_d2[owner][lane] && s_at[v][lane] < s_at[owner][lane]))
            owner = v;
    // the warp that holds a node's nearest point finishes it
    if (!live || owner != w) return;
    wsum *= 2.0;
    const double turns = fabs(wsum / (4.0 * 3.14159265358979323846));
    bool inside = turns > 0.5;
    if (!(turns < 0.25 || turns > 0.75) || ntri > MESH_SCREENED) {
        wsum = 0.0;
        for (int t = 0; t < ntri; ++t) {
            const double* T = tri + 9ll * t;
            wsum += solid_angle(x, mk(T[0], T[1], T[2]), mk(T[3], T[4], T[5]), mk(T[6], T[7], T[8]));
        }
        inside = fabs(wsum / (4.0 * 3.14159265358979323846)) > 0.5;
    }
    const double d = len(x - near);
    double f = inside ? -d : d;
    Vec g = mk(0.0, 0.0, 0.0);
    if (d > 1e-30) {
        const Vec u = (x - near) / d;
        g = inside ? -u : u;
    }
    if (flip) { f = -f; g = -g; }
    out[((long long)k * n.y + j) * n.x + i] = grid_value(f, g, h);
}

}  // namespace

extern "C" int fundem_levelset_grid(int device, void* stream, const fundem_shape* shape, const double origin[3],
                                    double spacing, const int size[3], double* sdf)
{
    if (!shape || !origin || !size || !sdf || !(spacing > 0.0)) return FUNDEM_ERR_ARG;
    if (size[0] <= 0 || size[1] <= 0 || size[2] <= 0) return FUNDEM_ERR_ARG;
    const long long total = (long long)size[0] * size[1] * size[2];
    if (total > (1LL << 31)) return FUNDEM_ERR_ARG;
    const int kind = shape->kind;
    if (kind < FUNDEM_SHAPE_SUPERELLIPSOID || kind > FUNDEM_SHAPE_MESH) return FUNDEM_ERR_ARG;
    const double* p = shape->param;
    switch (kind) {
    case FUNDEM_SHAPE_SUPERELLIPSOID:
        if (!(p[0] > 0.0 && p[1] > 0.0 && p[2] > 0.0 && p[3] > 0.0 && p[4] > 0.0)) return FUNDEM_ERR_ARG;
        break;
    case FUNDEM_SHAPE_SPHERE:
        if (!(p[0] > 0.0)) return FUNDEM_ERR_ARG;
        break;
    case FUNDEM_SHAPE_BOX:
        if (!(p[0] > 0.0 && p[1] > 0.0 && p[2] > 0.0)) return FUNDEM_ERR_ARG;
        break;
    case FUNDEM_SHAPE_CYLINDER: {
        const double dx = p[3] - p[0], dy = p[4] - p[1], dz = p[5] - p[2];
        if (!(p[6] > 0.0) || !(std::sqrt(dx * dx + dy * dy + dz * dz) > 1e-30)) return FUNDEM_ERR_ARG;
        break;
    }
    default: {
        const int nv = shape->n_vertices, nt = shape->n_triangles;
        if (nv <= 0 || nt <= 0 || !shape->vertices || !shape->triangles) return FUNDEM_ERR_ARG;
        for (int t = 0; t < nt; ++t) {
            const int* T = shape->triangles + 3 * t;
            for (int k = 0; k < 3; ++k)
                if (T[k] < 0 || T[k] >= nv) return FUNDEM_ERR_ARG;
            if (T[0] == T[1] || T[1] == T[2] || T[2] == T[0]) return FUNDEM_ERR_ARG;
        }
    }
    }

    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess) return FUNDEM_ERR_CUDA;
    if (device >= 0 && device != prev && cudaSetDevice(device) != cudaSuccess) return FUNDEM_ERR_CUDA;
    cudaStream_t s = (cudaStream_t)stream;
    const double3 o = make_double3(origin[0], origin[1], origin[2]);
    const int3 n = make_int3(size[0], size[1], size[2]);
    double* d_out = nullptr;
    double* d_tri = nullptr;
    MeshTri* d_mesh = nullptr;
    double3 centre = make_double3(0.0, 0.0, 0.0);
    double unit = 1.0;
    int status = FUNDEM_OK;
    cudaError_t e = cudaMallocAsync((void**)&d_out, total * sizeof(double), s);
    if (e == cudaSuccess && kind == FUNDEM_SHAPE_MESH) {
        // triangle corners gathered on the host: 9 doubles per triangle
        const int nt = shape->n_triangles;
        double* h_tri = new double[(size_t)nt * 9];
        for (int t = 0; t < nt; ++t)
            for (int k = 0; k < 3; ++k)
                for (int c = 0; c < 3; ++c) h_tri[t * 9 + k * 3 + c] = shape->vertices[3 * shape->triangles[3 * t + k] + c];
        // the screening passes' frame
        centre = make_double3(o.x + 0.5 * (n.x - 1) * spacing, o.y + 0.5 * (n.y - 1) * spacing,
                              o.z + 0.5 * (n.z - 1) * spacing);
        double scale = 0.5 * spacing * (n.x + n.y + n.z);
        for (int v = 0; v < shape->n_vertices; ++v) {
            const double* q = shape->vertices + 3 * v;
            scale = std::fmax(scale, std::fabs(q[0] - centre.x) + std::fabs(q[1] - centre.y) + std::fabs(q[2] - centre.z));
        }
        unit = 1.0 / scale;
        e = cudaMallocAsync((void**)&d_tri, (size_t)nt * 9 * sizeof(double), s);
        if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_mesh, (size_t)nt * sizeof(MeshTri), s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(d_tri, h_tri, (size_t)nt * 9 * sizeof(double), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        delete[] h_tri;
    }
    if (e == cudaSuccess) {
        if (kind == FUNDEM_SHAPE_MESH) {
            const int nt = shape->n_triangles;
            k_mesh_prepare<<<(nt + 127) / 128, 128, 0, s>>>(d_tri, nt, centre, unit, d_mesh);
            const long long blocks = (long long)((n.x + 7) / 8) * ((n.y + 3) / 4) * n.z;
            k_levelset_mesh<<<(unsigned)blocks, MESH_BLOCK, 0, s>>>(d_tri, d_mesh, nt, shape->positive_inside != 0, o,
                                                                    spacing, n, centre, unit, d_out);
        } else {
            Shape sh;
            sh.kind = kind;
            sh.flip = shape->positive_inside != 0;
            for (int k = 0; k < 8; ++k) sh.p[k] = p[k];
            int sms = 148;
            int dev = 0;
            if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            const long long want = (total + 255) / 256;
            const long long cap = (long long)sms * 16;
            k_levelset_analytic<<<(unsigned)(want < cap ? want : cap), 256, 0, s>>>(sh, o, spacing, n, total, d_out);
        }
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(sdf, d_out, total * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (d_out) cudaFreeAsync(d_out, s);
    if (d_tri) cudaFreeAsync(d_tri, s);
    if (d_mesh) cudaFreeAsync(d_mesh, s);
    const cudaError_t e2 = cudaStreamSynchronize(s);
    if (e != cudaSuccess || e2 != cudaSuccess) status = FUNDEM_ERR_CUDA;
    if (device >= 0 && device != prev) cudaSetDevice(prev);
    return status;
}
