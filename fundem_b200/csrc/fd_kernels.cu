// fd_kernels.cu -- sm_100a kernels of the level-set DEM timestep.
//
// Per step (no host synchronisation; the bonds on a stream of their own):
//   kick, drift, hash (+ walls)            particleIntegrationKernel.cu:3-48, mySpatialGrid.cu:4-26
//   lists of the objects per cell          buildHashStartEnd.cu:47-137
//   broad phase: eight lanes per particle list candidate partners (bounding
//                spheres, or SDF-grid spheres for walls and ghosts), sorted
//                by partner id, into an A-major pair list
//   selection:   one warp per candidate pair culls A's clusters of surface
//                nodes, then the nodes, against B with exact-conservative
//                bounds; the rest become the pair's contact slots
//   predicate:   one thread per slot, the reference's node predicate bit for
//                bit (LSParticleContactDetectionKernel.cu:4-607)
//   contact law: one thread per contact, with the sliding spring of the
//                previous step (contactKernel.cuh:4-77)
//   pair sums, and the reverse index (pairs grouped by partner)
//   bonds (contactKernel.cu:293-371), one thread per bond
//   per-particle sums in a fixed order (no atomics on forces)
// Each stage is one launch for all contact lists; a small set's step is two
// launches in all.
#include "fd_kernels.cuh"
#include "../../include/fundem_b200.h"

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <stdexcept>
#include <type_traits>

namespace fd {

namespace {

// The two kernels of a small set's step take turns on one stream.  Each is
// launched while the other runs (launch_ahead): its blocks move in as the
// other's leave, and this wait, before anything else, holds them until that
// has finished and its writes are visible.  Every block waits first, so no
// kernel overtakes the one before.
__device__ __forceinline__ void step_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

constexpr int TPB = 256;
constexpr int MAX_CAND = 64;        // candidate partners per particle and kind
constexpr int MAX_CLUSTERS = 64;    // clusters per template (two warp-wide batches)
constexpr int MAX_NODE_QUEUE = 32 * MAX_CLUSTERS;  // per-warp queue of nodes for the exact test
constexpr int NARROW_WARPS = 8;     // warps per block in the narrow kernel
constexpr double PI_D = 3.14159265358979323846;

inline int nblocks(long long n, int tpb = TPB) { return (int)((n + tpb - 1) / tpb); }

__device__ __forceinline__ void set_flag(unsigned int* flags, unsigned int f)
{
    if (flags) atomicOr(flags, f);
}

// ---------------------------------------------------------------------------
// scan (exclusive, int), three-phase: tile scan, scan of tile sums, add
// ---------------------------------------------------------------------------
constexpr int SCAN_TPB = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_TPB * SCAN_ITEMS;

__device__ __forceinline__ int block_excl_scan(int v, int* total)
{
    __shared__ int warp_sum[SCAN_TPB / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int s = (lane < SCAN_TPB / 32) ? warp_sum[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < SCAN_TPB / 32) warp_sum[lane] = s;
    }
    __syncthreads();
    const int before = (wid > 0) ? warp_sum[wid - 1] : 0;
    if (total) *total = warp_sum[SCAN_TPB / 32 - 1];
    const int r = before + x - v;
    __syncthreads();
    return r;
}

template <bool INCLUSIVE>
__global__ void k_scan_tile(const int* in, int* out, long long n, int* tile_sums)
{
    const long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const long long i = base + k;
        v[k] = (i < n) ? in[i] : 0;
        s += v[k];
    }
    int total;
    int run = block_excl_scan(s, &total);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const long long i = base + k;
        if (INCLUSIVE) run += v[k];
        if (i < n) out[i] = run;
        if (!INCLUSIVE) run += v[k];
    }
    if (tile_sums && threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void k_scan_add(int* out, long long n, const int* tile_off)
{
    const long long i = (long long)blockIdx.x * SCAN_TILE + threadIdx.x;
    const int add = tile_off[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const long long j = i + (long long)k * SCAN_TPB;
        if (j < n && j < (long long)(blockIdx.x + 1) * SCAN_TILE) out[j] += add;
    }
}

// ---------------------------------------------------------------------------
// integration, particleIntegrationKernel.cu:3-48 and myQua.h:77-93
// ---------------------------------------------------------------------------
struct Body {
    double3 x, v, w;
    fd_quat q;
};

// The arithmetic below is written with explicit fused multiply-adds: one
// kernel runs a half kick alone, another two of them around the step boundary,
// and what the compiler contracts would differ between them.  The pattern is
// the compiler's for the expressions written out: in a sum of products the
// leftmost product is fused first.
__device__ __forceinline__ double3 fma3(double3 a, double s, double3 b)
{
    return mk3(__fma_rn(a.x, s, b.x), __fma_rn(a.y, s, b.y), __fma_rn(a.z, s, b.z));
}
__device__ __forceinline__ double dot3f(double ax, double ay, double az, double bx, double by, double bz)
{
    return __fma_rn(az, bz, __fma_rn(ax, bx, __dmul_rn(ay, by)));
}
__device__ __forceinline__ double3 smv_fma(fd_sym m, double3 v)
{
    return mk3(dot3f(m.xx, m.xy, m.xz, v.x, v.y, v.z), dot3f(m.xy, m.yy, m.yz, v.x, v.y, v.z),
               dot3f(m.xz, m.yz, m.zz, v.x, v.y, v.z));
}
__device__ __forceinline__ double3 cross_fma(double3 a, double3 b)
{
    return mk3(__fma_rn(a.y, b.z, -__dmul_rn(a.z, b.y)), __fma_rn(a.z, b.x, -__dmul_rn(a.x, b.z)),
               __fma_rn(a.x, b.y, -__dmul_rn(a.y, b.x)));
}
// R(q) I R(q)^T (rotateTensor, myMat.h:75-158)
__device__ __forceinline__ fd_sym rot_tensor_fma(fd_quat q, fd_sym I)
{
    const double x2 = 2.0 * q.q1, y2 = 2.0 * q.q2, z2 = 2.0 * q.q3;
    const double a = __fma_rn(-y2, q.q2, __fma_rn(-z2, q.q3, 1.0)), b = __fma_rn(x2, q.q2, -__dmul_rn(z2, q.q0)),
                 c = __fma_rn(x2, q.q3, __dmul_rn(y2, q.q0));
    const double d = __fma_rn(x2, q.q2, __dmul_rn(z2, q.q0)), e = __fma_rn(-x2, q.q1, __fma_rn(-z2, q.q3, 1.0)),
                 f = __fma_rn(y2, q.q3, -__dmul_rn(x2, q.q0));
    const double g = __fma_rn(x2, q.q3, -__dmul_rn(y2, q.q0)), h = __fma_rn(y2, q.q3, __dmul_rn(x2, q.q0)),
                 i = __fma_rn(-x2, q.q1, __fma_rn(-y2, q.q2, 1.0));
    const double3 r0 = smv_fma(I, mk3(a, b, c)), r1 = smv_fma(I, mk3(d, e, f)), r2 = smv_fma(I, mk3(g, h, i));
    fd_sym r;
    r.xx = dot3f(r0.x, r0.y, r0.z, a, b, c);
    r.yy = dot3f(r1.x, r1.y, r1.z, d, e, f);
    r.zz = dot3f(r2.x, r2.y, r2.z, g, h, i);
    r.xy = dot3f(r0.x, r0.y, r0.z, d, e, f);
    r.xz = dot3f(r0.x, r0.y, r0.z, g, h, i);
    r.yz = dot3f(r1.x, r1.y, r1.z, g, h, i);
    return r;
}

__device__ __forceinline__ void kick_body(Body& b, const FdGeo& geo, double3 F, double3 T, double3 g, double h)
{
    const double invM = geo.inv_mass;
    if (fd_is_zero(invM)) return;
    b.v = fma3(fma3(F, invM, g), h, b.v);
    const double3 wxL = cross_fma(b.w, smv_fma(rot_tensor_fma(b.q, geo.inertia), b.w));
    const double3 r = mk3(__dsub_rn(T.x, wxL.x), __dsub_rn(T.y, wxL.y), __dsub_rn(T.z, wxL.z));
    b.w = fma3(smv_fma(rot_tensor_fma(b.q, geo.inv_inertia), r), h, b.w);
}

__device__ __forceinline__ fd_quat quat_integrate(fd_quat q, double3 w, double dt)
{
    const double h = 0.5 * dt;
    const double3 v = mk3(__dmul_rn(w.x, h), __dmul_rn(w.y, h), __dmul_rn(w.z, h));
    fd_quat s;
    s.q0 = __dadd_rn(q.q0, -dot3f(q.q1, q.q2, q.q3, v.x, v.y, v.z));
    s.q1 = __dadd_rn(q.q1, dot3f(q.q0, q.q3, -q.q2, v.x, v.y, v.z));
    s.q2 = __dadd_rn(q.q2, dot3f(-q.q3, q.q0, q.q1, v.x, v.y, v.z));
    s.q3 = __dadd_rn(q.q3, dot3f(q.q2, -q.q1, q.q0, v.x, v.y, v.z));
    const double l2 = __fma_rn(s.q3, s.q3, dot3f(s.q0, s.q1, s.q2, s.q0, s.q1, s.q2));
    if (fd_is_zero(l2)) return s;
    const double inv = rsqrt(l2);
    fd_quat r = {__dmul_rn(s.q0, inv), __dmul_rn(s.q1, inv), __dmul_rn(s.q2, inv), __dmul_rn(s.q3, inv)};
    return r;
}

__device__ __forceinline__ void drift_body(Body& b, double dt)
{
    b.x = fma3(b.v, dt, b.x);
    b.q = quat_integrate(b.q, b.w, dt);
}

// ---------------------------------------------------------------------------
// hashing and the cell table
// ---------------------------------------------------------------------------
__device__ __forceinline__ void quat_matrix(const fd_quat q, double R[9])
{
    const double q0 = q.q0, q1 = q.q1, q2 = q.q2, q3 = q.q3;
    R[0] = 1.0 - 2.0 * (q2 * q2 + q3 * q3); R[1] = 2.0 * (q1 * q2 - q0 * q3); R[2] = 2.0 * (q1 * q3 + q0 * q2);
    R[3] = 2.0 * (q1 * q2 + q0 * q3); R[4] = 1.0 - 2.0 * (q1 * q1 + q3 * q3); R[5] = 2.0 * (q2 * q3 - q0 * q1);
    R[6] = 2.0 * (q1 * q3 - q0 * q2); R[7] = 2.0 * (q2 * q3 + q0 * q1); R[8] = 1.0 - 2.0 * (q1 * q1 + q2 * q2);
}

// cell hash and single-precision rotation rows of object i at x, q
__device__ __forceinline__ long long hash_one(const ObjDev& O, const FdGrid& g, int i, double3 x, fd_quat q)
{
    const long long h = fd_hash(x, g);
    O.hash[i] = h;
    if (O.rot) {
        double R[9];
        quat_matrix(q, R);
        O.rot[3 * i + 0] = make_float4((float)R[0], (float)R[1], (float)R[2], 0.f);
        O.rot[3 * i + 1] = make_float4((float)R[3], (float)R[4], (float)R[5], 0.f);
        O.rot[3 * i + 2] = make_float4((float)R[6], (float)R[7], (float)R[8], 0.f);
    }
    return h;
}

// new build numbers for a cell table: one for the list generation this step
// writes, a fresh one for the other
__device__ __forceinline__ void bump_build(unsigned int* build, int par)
{
    const unsigned int m = max(build[0], build[1]);
    build[par] = m + 1u;
    build[par ^ 1] = m + 2u;
}

__global__ void k_hash(ObjDev O, FdGrid g, unsigned int* build, int par)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= O.n) return;
    if (i == 0 && build) bump_build(build, par);
    hash_one(O, g, i, O.pos[i], O.q[i]);
}

// ---------------------------------------------------------------------------
// stable LSD radix sort of 64-bit cell keys, 8 bits per pass over the bits a
// key can use: per block a digit histogram, an exclusive scan of the counts
// (digit-major, so equal digits keep block order), then a scatter that ranks
// each key within its block by warp (match of equal digits) and by lane
// ---------------------------------------------------------------------------
constexpr int RS_TPB = 256;
constexpr int RS_RADIX = 256;
constexpr unsigned long long RS_NONE = ~0ull;  // key of an object in no cell

__global__ void k_rs_keys(const long long* hash, int n, long long num, unsigned long long* key, int* idx)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long h = hash[i];
    key[i] = (h >= 0 && h < num) ? (unsigned long long)h : RS_NONE;
    idx[i] = i;
}

__global__ void __launch_bounds__(RS_TPB) k_rs_hist(const unsigned long long* key, int n, int shift, int* bcount,
                                                   int nblk)
{
    __shared__ int h[RS_RADIX];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int i = blockIdx.x * RS_TPB + threadIdx.x;
    if (i < n) atomicAdd(&h[(key[i] >> shift) & (RS_RADIX - 1)], 1);
    __syncthreads();
    bcount[(long long)threadIdx.x * nblk + blockIdx.x] = h[threadIdx.x];
}

__global__ void __launch_bounds__(RS_TPB) k_rs_scatter(const unsigned long long* key, const int* idx, int n, int shift,
                                                      const int* boff, int nblk, unsigned long long* okey, int* oidx)
{
    constexpr int NW = RS_TPB / 32;
    __shared__ int wcnt[NW][RS_RADIX];
    for (int d = threadIdx.x; d < NW * RS_RADIX; d += RS_TPB) (&wcnt[0][0])[d] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blockIdx.x * RS_TPB + threadIdx.x;
    const bool valid = i < n;
    const unsigned long long k = valid ? key[i] : 0ull;
    const int digit = valid ? (int)((k >> shift) & (RS_RADIX - 1)) : RS_RADIX;
    const unsigned int peers = __match_any_sync(0xffffffffu, digit);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (valid && lane == __ffs(peers) - 1) wcnt[w][digit] = __popc(peers);
    __syncthreads();
    if (valid) {
        int pos = boff[(long long)digit * nblk + blockIdx.x] + rank;
        for (int v = 0; v < w; ++v) pos += wcnt[v][digit];
        okey[pos] = k;
        oidx[pos] = idx[i];
    }
}

// the pair cache's gate: the list is built this step, not carried over
__device__ __forceinline__ bool list_built(const StepArgs& a)
{
    return a.gate == nullptr || *a.gate != 0 || (a.gate2 && *a.gate2 != 0);
}
__device__ __forceinline__ double list_skin(const StepArgs& a) { return (a.noskin && *a.noskin) ? 0.0 : a.skin; }

// Cell table: the objects of a cell form a list, head and next.  A counting
// sort took seven launches of 2-4 us each (clear, count, scan, scatter, order;
// 28 with the radix sort of a sparse grid), all waiting on one another; the
// list is one launch of one atomic per object.  The order inside a cell does
// not matter: every search sorts the partners it keeps.  A head carries the
// number of the build that wrote it, so heads of older builds read as empty
// and a dense table is never cleared.
__global__ void k_hkey_clear(unsigned long long* hkey, unsigned long long n, StepArgs a)
{
    const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !list_built(a)) return;
    hkey[i] = RS_NONE;
}

__device__ __forceinline__ unsigned long long cell_slot_hash(unsigned long long k)
{
    // splitmix64 finaliser
    k ^= k >> 30;
    k *= 0xbf58476d1ce4e5b9ull;
    k ^= k >> 27;
    k *= 0x94d049bb133111ebull;
    k ^= k >> 31;
    return k;
}

// put object i into the list of head slot `slot`
__device__ __forceinline__ void cell_push(const CellTableDev& T, unsigned long long slot, unsigned int build, int i)
{
    const unsigned long long old =
        atomicExch(&T.head[slot], ((unsigned long long)build << 32) | (unsigned int)i);
    T.next[i] = (unsigned int)(old >> 32) == build ? (int)(unsigned int)old : -1;
}

// object i, of cell hash h, into the table
__device__ __forceinline__ void cell_link(const CellTableDev& T, long long h, unsigned int build, int i)
{
    if (h < 0 || h >= T.g.num) return;
    if (!T.hashed) {
        cell_push(T, (unsigned long long)h, build, i);
        return;
    }
    const unsigned long long k = (unsigned long long)h;
    unsigned long long slot = cell_slot_hash(k) & T.hmask;
    // the table holds at least twice as many slots as there are objects, so
    // an empty slot is always found; the probe count is bounded all the same
    for (unsigned long long probe = 0; probe <= T.hmask; ++probe) {
        const unsigned long long prev = atomicCAS(&T.hkey[slot], RS_NONE, k);
        if (prev == RS_NONE || prev == k) {
            cell_push(T, slot, build, i);
            return;
        }
        slot = (slot + 1) & T.hmask;
    }
}

// first object of cell h in the build of that number, -1 when it holds none
__device__ __forceinline__ int cell_first(const CellTableDev& T, long long h, unsigned int build)
{
    unsigned long long slot = (unsigned long long)h;
    if (T.hashed) {
        slot = cell_slot_hash((unsigned long long)h) & T.hmask;
        for (unsigned long long probe = 0;; ++probe) {
            const unsigned long long kk = T.hkey[slot];
            if (kk == (unsigned long long)h) break;
            if (kk == RS_NONE || probe >= T.hmask) return -1;
            slot = (slot + 1) & T.hmask;
        }
    }
    const unsigned long long e = T.head[slot];
    return (unsigned int)(e >> 32) == build ? (int)(unsigned int)e : -1;
}

// ---------------------------------------------------------------------------
// periodic wrap and ghosts, mySpatialGrid.cu:28-56, 87-152, 214-240
// ---------------------------------------------------------------------------
__device__ __forceinline__ double3 wrap_x(double3 p, const FdGrid& g)
{
    const double3 off = mk3(g.maxb.x - g.minb.x, 0., 0.);
    if (p.x < g.minb.x) p = p + off;
    else if (p.x >= g.maxb.x) p = p - off;
    return p;
}
__device__ __forceinline__ double3 wrap_y(double3 p, const FdGrid& g)
{
    const double3 off = mk3(0., g.maxb.y - g.minb.y, 0.);
    if (p.y < g.minb.y) p = p + off;
    else if (p.y >= g.maxb.y) p = p - off;
    return p;
}

// periodic shifts of the force-side centres ri, rj against the detection-side
// cA, cB (-1, 0 or 1 period per axis), as one code for the adjoint's record
__device__ __forceinline__ int wrap_code(double3 cA, double3 ri, double3 cB, double3 rj, const FdGrid& g)
{
    const double Lx = g.maxb.x - g.minb.x, Ly = g.maxb.y - g.minb.y;
    auto sh = [](double d, double L) { return d > 0.5 * L ? 1 : (d < -0.5 * L ? -1 : 0); };
    return (sh(ri.x - cA.x, Lx) + 1) + 3 * (sh(ri.y - cA.y, Ly) + 1) + 9 * (sh(rj.x - cB.x, Lx) + 1) +
           27 * (sh(rj.y - cB.y, Ly) + 1);
}

// calculateGhostHashKernel, including its z test against maxBound.y (:236):
// an image outside the domain is hashed into the clamped boundary cell, an
// image inside it is not a ghost
// Returns the directions (bit 0 x, 1 y, 2 z) in which the image lies
// outside the domain.
__device__ __forceinline__ int image_hash(const GhostDev& Gh, int i, double3 r)
{
    const FdGrid& g = Gh.cells.g;
    int3 gc = fd_cell_of(r, g);
    int outm = 0;
    if (r.x < g.minb.x) { gc.x = 0; outm |= 1; }
    else if (r.x >= g.maxb.x) { gc.x = g.size.x - 1; outm |= 1; }
    if (r.y < g.minb.y) { gc.y = 0; outm |= 2; }
    else if (r.y >= g.maxb.y) { gc.y = g.size.y - 1; outm |= 2; }
    if (r.z < g.minb.z) { gc.z = 0; outm |= 4; }
    else if (r.z >= g.maxb.y) { gc.z = g.size.z - 1; outm |= 4; }
    const bool out = outm != 0;
    const long long h = out ? fd_lin3(gc.x, gc.y, gc.z, g.size) : -1;
    Gh.hash[i] = h;
    if (h >= 0 && h < g.num) {
        atomicMin(&Gh.occ[0], gc.x); atomicMin(&Gh.occ[1], gc.y); atomicMin(&Gh.occ[2], gc.z);
        atomicMax(&Gh.occ[3], gc.x); atomicMax(&Gh.occ[4], gc.y); atomicMax(&Gh.occ[5], gc.z);
    }
    return outm;
}

// The image of a particle in the first cell column (row, or both) sits one
// period beyond the domain; every other particle keeps its own position.  A
// particle enters the image table when that position lies outside the
// domain, tested as the reference tests it (z against max y): the shifted
// ones, and unshifted ones above max y.  Gh.live marks these entries.
// Under the pair cache (ctrl non-null) particles without an entry that lie
// within ext_skin of the image band get a shifted entry too, so that a
// rebuild lists the pairs of every particle that can gain an image before
// the next rebuild.
__device__ __forceinline__ int image_out_mask(double3 r, const FdGrid& g)
{
    int m = 0;
    if (r.x < g.minb.x || r.x >= g.maxb.x) m |= 1;
    if (r.y < g.minb.y || r.y >= g.maxb.y) m |= 2;
    if (r.z < g.minb.z || r.z >= g.maxb.y) m |= 4;
    return m;
}
__device__ __forceinline__ void image_build(const GhostDev& Gh, int kind, int i, double3 p, double ext_skin, int* ctrl)
{
    const FdGrid& g = Gh.cells.g;
    const double3 ox = mk3(g.maxb.x - g.minb.x, 0., 0.), oy = mk3(0., g.maxb.y - g.minb.y, 0.);
    const double3 shift = kind == FD_GX ? ox : kind == FD_GY ? oy : ox + oy;
    const int3 c = fd_cell_of(p, g);
    bool shifted = false;
    if (kind == FD_GX) shifted = c.x == 0;
    if (kind == FD_GY) shifted = c.y == 0;
    if (kind == FD_GXY) shifted = c.x == 0 && c.y == 0;
    const double3 ru = shifted ? p + shift : p;
    const bool live = image_out_mask(ru, g) != 0;
    bool band = false;
    if (ctrl && !live) {
        const bool bx = (p.x - g.minb.x) * g.inv.x < 1.0 + ext_skin * g.inv.x * 1.01;
        const bool by = (p.y - g.minb.y) * g.inv.y < 1.0 + ext_skin * g.inv.y * 1.01;
        if (kind == FD_GX) band = bx;
        if (kind == FD_GY) band = by;
        if (kind == FD_GXY) band = bx && by;
    }
    const double3 r = live ? ru : band ? p + shift : p;
    Gh.pos[i] = r;
    if (Gh.live) Gh.live[i] = live ? 1 : 0;
    const int outm = image_hash(Gh, i, r);
    if (ctrl && (live || band)) {
        // outside the domain across the translation only: its cell is the
        // natural one in the other directions, and candidacy follows the
        // geometry; otherwise (a clamped cell) this step is built uncached
        const int along = kind == FD_GX ? 1 : kind == FD_GY ? 2 : 3;
        if (outm & ~along) {
            ctrl[4] = 1;
            ctrl[7] = 1;
        }
    }
}

// the periodic wraps (into dst, which may be P.pos) and the translated images:
// x wraps, x images, y wraps, y and xy images (PeriodicBoundaryXY2D,
// LSSolver.h:780-784).  One pass over the positions in place of five launches.
struct ImageArgs {
    ObjDev P;
    double3* dst;
    GhostDev gh[3];   // X, Y, XY
    int on[3];
    double ext_skin;
    int* ctrl;        // the pair cache's, or null
};
__global__ void k_images(ImageArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.P.n) return;
    if (i == 0)
        for (int d = 0; d < 3; ++d)
            if (a.on[d]) bump_build(a.gh[d].cells.build, a.gh[d].cells.par);
    const double3 p0 = a.P.pos[i];
    double3 p = p0;
    if (a.on[0]) {
        p = wrap_x(p, a.gh[0].cells.g);
        image_build(a.gh[0], FD_GX, i, p, a.ext_skin, a.ctrl);
    }
    if (a.on[1]) {
        p = wrap_y(p, a.gh[1].cells.g);
        image_build(a.gh[1], FD_GY, i, p, a.ext_skin, a.ctrl);
    }
    if (a.on[2]) image_build(a.gh[2], FD_GXY, i, p, a.ext_skin, a.ctrl);
    a.dst[i] = p;
    // under the pair cache a wrap changes which particles have images: the
    // ghost lists of this step are built afresh, and every list at the next
    if (a.ctrl && (p.x != p0.x || p.y != p0.y)) {
        a.ctrl[4] = 1;
        a.ctrl[7] = 1;
    }
}

// ---------------------------------------------------------------------------
// sector periodicity, mySpatialGrid.cu:58-85, 154-213 (PeriodicBoundary.h:
// 319-425): the quarter sector x >= min.x, y >= min.y repeats under quarter
// turns about the z axis through the domain's min corner
// ---------------------------------------------------------------------------
// rotateVector, myVec.h:143-182 (device branch): v turned by the angle |om|
// about om, v + (sin t / t) om x v + ((1 - cos t) / t^2) om x (om x v)
__device__ __forceinline__ double3 turn_vec(double3 v, double3 om)
{
    const double th2 = dot3(om, om);
    if (fd_is_zero(th2)) {
        const double3 oxv = cross3(om, v), oo = cross3(om, oxv);
        return v + oxv + 0.5 * oo;
    }
    const double inv = rsqrt(th2);
    const double th = th2 * inv;
    double sn, cs;
    sincos(th, &sn, &cs);
    const double A = sn * inv, B = (1.0 - cs) * (inv * inv);
    const double3 oxv = cross3(om, v), oo = cross3(om, oxv);
    return v + A * oxv + B * oo;
}
// rotateQuaternion, myQua.h:131-180: the turn about om times q, normalised
__device__ __forceinline__ fd_quat turn_quat(fd_quat q, double3 om)
{
    const double th2 = om.x * om.x + om.y * om.y + om.z * om.z;
    if (fd_is_zero(th2)) return q;
    const double th = sqrt(th2);
    const double inv = 1.0 / th;
    const double ux = om.x * inv, uy = om.y * inv, uz = om.z * inv;
    const double half = 0.5 * th;
    const double c = cos(half), sn = sin(half);
    const double r0 = c, r1 = sn * ux, r2 = sn * uy, r3 = sn * uz;
    fd_quat o;
    o.q0 = r0 * q.q0 - r1 * q.q1 - r2 * q.q2 - r3 * q.q3;
    o.q1 = r0 * q.q1 + r1 * q.q0 + r2 * q.q3 - r3 * q.q2;
    o.q2 = r0 * q.q2 - r1 * q.q3 + r2 * q.q0 + r3 * q.q1;
    o.q3 = r0 * q.q3 + r1 * q.q2 - r2 * q.q1 + r3 * q.q0;
    return fd_normalize_q(o);
}
// velocity, position about the min corner and orientation turned by a about z
__device__ __forceinline__ void sector_turn(double3& v, double3& p, fd_quat& q, double3 mn, double a)
{
    const double3 om = mk3(0., 0., a);
    v = turn_vec(v, om);
    p = mn + turn_vec(p - mn, om);
    q = turn_quat(q, om);
}

// position and velocity of a body as the sector wrap of this step leaves
// them: the reference computes particle and wall contact forces after that
// wrap from contacts detected before it, so the force side of those contacts
// sees the turned body
__device__ __forceinline__ void sector_fold(double3& p, double3& v, double3 mn)
{
    if (p.x < mn.x && p.y >= mn.y) {
        const double3 om = mk3(0., 0., -0.5 * PI_D);
        v = turn_vec(v, om);
        p = mn + turn_vec(p - mn, om);
    }
    if (p.y < mn.y && p.x >= mn.x) {
        const double3 om = mk3(0., 0., 0.5 * PI_D);
        v = turn_vec(v, om);
        p = mn + turn_vec(p - mn, om);
    }
}

// a body that left through the x face comes back through the y face turned
// by -90 degrees, and one that left through the y face by +90 degrees
__global__ void k_sector_wrap(ObjDev P, double3 mn)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    double3 v = P.vel[i], p = P.pos[i];
    fd_quat q = P.q[i];
    bool turned = false;
    if (p.x < mn.x && p.y >= mn.y) { sector_turn(v, p, q, mn, -0.5 * PI_D); turned = true; }
    if (p.y < mn.y && p.x >= mn.x) { sector_turn(v, p, q, mn, 0.5 * PI_D); turned = true; }
    P.vel[i] = v;
    P.pos[i] = p;
    P.q[i] = q;
    if (turned && P.rot) {
        // the single-precision rotation rows of this step follow the turn
        double R[9];
        quat_matrix(q, R);
        P.rot[3 * i + 0] = make_float4((float)R[0], (float)R[1], (float)R[2], 0.f);
        P.rot[3 * i + 1] = make_float4((float)R[3], (float)R[4], (float)R[5], 0.f);
        P.rot[3 * i + 2] = make_float4((float)R[6], (float)R[7], (float)R[8], 0.f);
    }
}

__device__ __forceinline__ void image_store(GhostDev& Gh, int i, double3 p, double3 v, fd_quat q)
{
    Gh.pos[i] = p;
    Gh.vel[i] = v;
    Gh.q[i] = q;
    double R[9];
    quat_matrix(q, R);
    Gh.rot[3 * i + 0] = make_float4((float)R[0], (float)R[1], (float)R[2], 0.f);
    Gh.rot[3 * i + 1] = make_float4((float)R[3], (float)R[4], (float)R[5], 0.f);
    Gh.rot[3 * i + 2] = make_float4((float)R[6], (float)R[7], (float)R[8], 0.f);
    image_hash(Gh, i, p);
}

// images turned by +90 degrees (bodies in the first cell row in y), -90
// degrees (first cell column in x) and 180 degrees (the corner cell); every
// other image is a copy of its body
__global__ void k_sector_images(ObjDev P, GhostDev R90, GhostDev R180, GhostDev R270)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    if (i == 0) {
        bump_build(R90.cells.build, R90.cells.par);
        bump_build(R180.cells.build, R180.cells.par);
        bump_build(R270.cells.build, R270.cells.par);
    }
    const FdGrid& g = R90.cells.g;
    const double3 p = P.pos[i], v = P.vel[i];
    const fd_quat q = P.q[i];
    const int3 c = fd_cell_of(p, g);
    const bool row0 = c.y == 0, col0 = c.x == 0;
    double3 pa = p, va = v;
    fd_quat qa = q;
    if (row0) sector_turn(va, pa, qa, g.minb, 0.5 * PI_D);
    image_store(R90, i, pa, va, qa);
    pa = p; va = v; qa = q;
    if (row0 && col0) sector_turn(va, pa, qa, g.minb, PI_D);
    image_store(R180, i, pa, va, qa);
    pa = p; va = v; qa = q;
    if (col0) sector_turn(va, pa, qa, g.minb, -0.5 * PI_D);
    image_store(R270, i, pa, va, qa);
}

// ---------------------------------------------------------------------------
// broad phase
// ---------------------------------------------------------------------------
__device__ __forceinline__ int cell_index_clamped(double x, double mn, double inv, int size)
{
    double v = (x - mn) * inv;
    v = fmin(fmax(v, -1.0), (double)size);
    int c = (int)v;
    return c < 0 ? 0 : (c > size - 1 ? size - 1 : c);
}

// cells the nodes of a body of radius r centred at c can search, in grid g
__device__ __forceinline__ void body_search_range(double3 c, double r, const FdGrid& g, int3& lo, int3& hi)
{
    lo.x = max(cell_index_clamped(c.x - r, g.minb.x, g.inv.x, g.size.x) - 1, 0);
    lo.y = max(cell_index_clamped(c.y - r, g.minb.y, g.inv.y, g.size.y) - 1, 0);
    lo.z = max(cell_index_clamped(c.z - r, g.minb.z, g.inv.z, g.size.z) - 1, 0);
    hi.x = min(cell_index_clamped(c.x + r, g.minb.x, g.inv.x, g.size.x) + 1, g.size.x - 1);
    hi.y = min(cell_index_clamped(c.y + r, g.minb.y, g.inv.y, g.size.y) + 1, g.size.y - 1);
    hi.z = min(cell_index_clamped(c.z + r, g.minb.z, g.inv.z, g.size.z) + 1, g.size.z - 1);
}

__device__ __forceinline__ void decode_cell(long long h, int3 s, int3& c)
{
    if ((unsigned long long)h < (1ull << 31) && (long long)s.x * s.y < (1ll << 31)) {
        // grids of fewer than 2^31 cells: 32-bit divisions
        const unsigned int u = (unsigned int)h, row = u / (unsigned int)s.x;
        c.x = (int)(u - row * (unsigned int)s.x);
        c.z = (int)(row / (unsigned int)s.y);
        c.y = (int)(row - (unsigned int)c.z * (unsigned int)s.y);
        return;
    }
    c.x = (int)(h % s.x);
    c.y = (int)((h / s.x) % s.y);
    c.z = (int)(h / ((long long)s.x * s.y));
}

__device__ void emit_pairs(int A, int* buf, int cnt, int total, const PairListDev& L, unsigned int* flags)
{
    if (total > MAX_CAND) set_flag(flags, FD_FLAG_NEIGHBOR_OVERFLOW);
    // insertion sort by partner id: deterministic pair order
    for (int a = 1; a < cnt; ++a) {
        const int v = buf[a];
        int b = a - 1;
        while (b >= 0 && buf[b] > v) { buf[b + 1] = buf[b]; --b; }
        buf[b + 1] = v;
    }
    int base = 0;
    if (cnt > 0) base = atomicAdd(L.n_pairs, cnt);
    if (cnt > 0 && base + cnt > L.cap_pairs) {
        set_flag(flags, FD_FLAG_PAIR_OVERFLOW);
        L.seg_off[A] = 0;
        L.seg_cnt[A] = 0;
        return;
    }
    L.seg_off[A] = base;
    L.seg_cnt[A] = cnt;
    for (int k = 0; k < cnt; ++k) {
        L.pairA[base + k] = A;
        L.pairB[base + k] = buf[k];
    }
}

constexpr double BOUND_REL = 1e-9;

// The predicate and contact passes read about 27 numbers a slot at addresses
// that differ from lane to lane, and the L1 serves a warp's addresses one line
// at a time: 79% of its rate at 65,003 particles.  Orientations and the
// interpolation's corners come in 32-byte loads instead (4 to 1 and 8 to 2).
__device__ __forceinline__ double4 load_quad(const double4* p)
{
    double4 v;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}
// The corner values of the cell at point i of a set's grids, of the planes z
// (s0) and z + 1 (s1): from the table of faces, or one by one where the set's
// table would take too much memory (see GeoSetHost::faces).  FACES: the table is
// there; the way without it costs the small steps' pair kernel registers that it
// has not got (ten steps of 4,096 particles 639 us with it, 625 without).
template <bool FACES>
__device__ __forceinline__ void load_corners(const GeoSetDev& S, long long i, long long sx, long long sxy, double4& s0,
                                             double4& s1)
{
    if (FACES || S.sdf_quad) {
        s0 = load_quad(S.sdf_quad + i);
        s1 = load_quad(S.sdf_quad + i + sxy);
        return;
    }
    const double *g = S.sdf + i, *h = g + sxy;
    s0 = make_double4(__ldg(g), __ldg(g + 1), __ldg(g + sx), __ldg(g + sx + 1));
    s1 = make_double4(__ldg(h), __ldg(h + 1), __ldg(h + sx), __ldg(h + sx + 1));
}
template <bool FACES>
__device__ __forceinline__ void load_corners(const GeoSetDev& S, long long i, long long sx, long long sxy, float4& s0,
                                             float4& s1)
{
    if (FACES || S.sdf32_quad) {
        s0 = __ldg(S.sdf32_quad + i);
        s1 = __ldg(S.sdf32_quad + i + sxy);
        return;
    }
    const float *g = S.sdf32 + i, *h = g + sxy;
    s0 = make_float4(__ldg(g), __ldg(g + 1), __ldg(g + sx), __ldg(g + sx + 1));
    s1 = make_float4(__ldg(h), __ldg(h + 1), __ldg(h + sx), __ldg(h + sx + 1));
}

// True when no point within `radius` of p (a position in B's body frame, in
// single precision) can pass the node predicate against B (or, with probe >
// 0, come within `probe` of B).  Conservative: single-precision evaluation
// with relative margins far above its rounding (about 1e-7 relative), bounds
// that hold in exact arithmetic:
//   * B's bounding sphere (particle pairs: the reference's radius test),
//   * B's SDF grid box (nodes outside it are never contacts),
//   * D(v): lower bound on the distance from grid node v to any cell whose
//     corner minimum is <= 0, 1-Lipschitz in the position,
//   * the Lipschitz bound of the trilinear SDF (distance-like fields).
template <bool FACES = false>
__device__ __forceinline__ bool sphere_culled(float px, float py, float pz, float radius, bool radius_test,
                                              const FdGeo32& GB, const GeoSetDev& SB, float probe)
{
    const float scale = GB.radius + radius + GB.spacing;
    const float margin = 2e-5f * scale;
    const float rho = radius + margin;
    if (radius_test) {
        const float lim = GB.radius + rho;
        if (px * px + py * py + pz * pz > lim * lim) return true;
    }
    const float is = GB.is;
    const float gx = (px - GB.ox) * is, gy = (py - GB.oy) * is, gz = (pz - GB.oz) * is;
    const float rg = rho * is + 1e-4f;
    if (gx < -rg || gy < -rg || gz < -rg) return true;
    if (gx > GB.size.x - 1 + rg || gy > GB.size.y - 1 + rg || gz > GB.size.z - 1 + rg) return true;
    if (probe == 0.f) {
        const int vx = min(max(__float2int_rn(gx), 0), GB.size.x - 1);
        const int vy = min(max(__float2int_rn(gy), 0), GB.size.y - 1);
        const int vz = min(max(__float2int_rn(gz), 0), GB.size.z - 1);
        const float D = __ldg(SB.dist + GB.dist_off + fd_lin3(vx, vy, vz, GB.size));
        const float sp = GB.spacing;
        const float dx = (gx - vx) * sp, dy = (gy - vy) * sp, dz = (gz - vz) * sp;
        if (D - sqrtf(dx * dx + dy * dy + dz * dz) > rho) return true;
    }
    // the Lipschitz bound only helps where the field is distance-like
    if (GB.tight && gx >= 0.f && gy >= 0.f && gz >= 0.f && gx < GB.size.x - 1 && gy < GB.size.y - 1 &&
        gz < GB.size.z - 1) {
        const int i0 = (int)gx, j0 = (int)gy, k0 = (int)gz;
        const long long sx = GB.size.x, sxy = (long long)GB.size.x * GB.size.y;
        float4 s0, s1;
        load_corners<FACES>(SB, GB.sdf_off + (long long)k0 * sxy + (long long)j0 * sx + i0, sx, sxy, s0, s1);
        const float fx = gx - i0, fy = gy - j0, fz = gz - k0;
        const float c00 = s0.x * (1.f - fx) + s0.y * fx;
        const float c10 = s0.z * (1.f - fx) + s0.w * fx;
        const float c01 = s1.x * (1.f - fx) + s1.y * fx;
        const float c11 = s1.z * (1.f - fx) + s1.w * fx;
        const float phi = (c00 * (1.f - fy) + c10 * fy) * (1.f - fz) + (c01 * (1.f - fy) + c11 * fy) * fz;
        const float bound = GB.lip * rho + probe;
        if (phi - bound > 1e-5f * (fabsf(phi) + bound + GB.spacing)) return true;
    }
    return false;
}

// Body-level cull of a candidate pair in single precision: A's bounding
// sphere (radius rA about cA) against B, through B's rotation rows
template <bool FACES = false>
__device__ __forceinline__ bool body_culled32(const double3 cA, double rA, const double3 cB, const float4* RB,
                                              bool radius_test, const FdGeo32& GB, const GeoSetDev& SB, double probe)
{
    const float4 b0 = RB[0], b1 = RB[1], b2 = RB[2];
    const float dx = (float)(cA.x - cB.x), dy = (float)(cA.y - cB.y), dz = (float)(cA.z - cB.z);
    const float px = fmaf(b0.x, dx, fmaf(b1.x, dy, b2.x * dz));
    const float py = fmaf(b0.y, dx, fmaf(b1.y, dy, b2.y * dz));
    const float pz = fmaf(b0.z, dx, fmaf(b1.z, dy, b2.z * dz));
    return sphere_culled<FACES>(px, py, pz, (float)rA, radius_test, GB, SB, (float)probe);
}

// cells that can hold the centre of a partner of a body of radius r centred
// at c, when partners have radius at most rp: every partner centre within
// r + rp of c lies in a cell overlapping [c - r - rp, c + r + rp]
__device__ __forceinline__ void partner_search_range(double3 c, double reach, const FdGrid& g, int3& lo, int3& hi)
{
    lo.x = cell_index_clamped(c.x - reach, g.minb.x, g.inv.x, g.size.x);
    lo.y = cell_index_clamped(c.y - reach, g.minb.y, g.inv.y, g.size.y);
    lo.z = cell_index_clamped(c.z - reach, g.minb.z, g.inv.z, g.size.z);
    hi.x = cell_index_clamped(c.x + reach, g.minb.x, g.inv.x, g.size.x);
    hi.y = cell_index_clamped(c.y + reach, g.minb.y, g.inv.y, g.size.y);
    hi.z = cell_index_clamped(c.z + reach, g.minb.z, g.inv.z, g.size.z);
}

// The cells a body's ghost search covers: those within `reach` of its
// centre, and every cell next to a cell its nodes (within rA of the centre)
// can occupy.  The predicate takes an image as a candidate of a node when the
// image's cell is next to the node's (LSParticleContactDetectionKernel.cu:
// 431-607); an image outside the domain in y or z sits in a clamped cell
// (mySpatialGrid.cu:214-240) that its position does not reach, and only the
// node neighbourhoods find it.
__device__ __forceinline__ void ghost_search_range(double3 c, double rA, double reach, const FdGrid& g, int3& lo,
                                                   int3& hi)
{
    partner_search_range(c, reach, g, lo, hi);
    int3 blo, bhi;
    body_search_range(c, rA, g, blo, bhi);
    lo = make_int3(min(lo.x, blo.x), min(lo.y, blo.y), min(lo.z, blo.z));
    hi = make_int3(max(hi.x, bhi.x), max(hi.y, bhi.y), max(hi.z, bhi.z));
}

#ifndef FD_BROAD_LANES
#define FD_BROAD_LANES 8
#endif
constexpr int BROAD_LANES = FD_BROAD_LANES;  // lanes per particle in the cell-table broad phases

// d with its periodic components taken to the nearest image
__device__ __forceinline__ double3 nl_min_image(double3 d, const NlDev& nl, const FdGrid& g)
{
    if (nl.periodic_x) {
        const double L = g.maxb.x - g.minb.x;
        d.x -= L * rint(d.x / L);
    }
    if (nl.periodic_y) {
        const double L = g.maxb.y - g.minb.y;
        d.y -= L * rint(d.y / L);
    }
    return d;
}

// Cell-table broad phase, BROAD_LANES lanes per particle A: each lane walks the
// lists of its share of the cells around A and tests the objects (partner
// order B > A for particle pairs, bounding spheres, body-level cull) and
// emit A's pairs sorted by partner id.  GHOST: partners are the ghost images
// of a cell table built from ghost positions (no B > A rule; the reach is the
// partner's SDF grid radius, since ghost pairs have no radius test).
//
// NLB: build the neighbour list instead of the pairs (only when a rebuild
// was requested): the sphere test is widened by the skin, the body-level
// cull is left to the per-step filter, and each particle's partners go to its
// fixed slice of the list.
//
// skin (pair cache): partners within rA + rB + skin are listed and the
// body-level cull treats A's sphere as skin larger.
template <bool GHOST, bool NLB>
__device__ __forceinline__ void broad_cells(const ObjDev& P, const GeoSetDev& G, const CellTableDev& T,
                                            const double3* gpos, const float4* grot, const int* occ,
                                            const PairListDev& L, const NlDev& nl, unsigned int* flags, double probe,
                                            double skin, int block, int nblocks, int (*s_list)[MAX_CAND])
{
    const unsigned int full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int gl = lane & (BROAD_LANES - 1);
    const int gbase = lane & ~(BROAD_LANES - 1);
    const int gb = threadIdx.x / BROAD_LANES;
    constexpr int GPW = 32 / BROAD_LANES;           // lane groups per warp
    constexpr int GPB = TPB / BROAD_LANES;          // lane groups per block
    const int total = P.n;
    const unsigned int build = T.build[T.par];
    // warp-uniform loop over the warp's groups
    for (int gw = block * GPB + (gb & ~(GPW - 1)); gw < total; gw += nblocks * GPB) {
    const int gidx = gw + (gb & (GPW - 1));
    const bool valid = gidx < total;
    const int A = valid ? gidx : 0;
    double3 cA = mk3(0., 0., 0.);
    double rA = 0.;
    int3 lo = make_int3(0, 0, 0), hi = make_int3(-1, -1, -1);
    if (valid) {
        cA = P.pos[A];
        rA = G.geo[P.geo[A]].radius;
        // above the sphere test's own tolerance (rs * (1 + 2 BOUND_REL))
        const double reach = (rA + (GHOST ? G.grid_rmax : G.rmax)) * (1.0 + 8.0 * BOUND_REL) + (NLB ? nl.skin : skin);
        if (NLB && gl == 0) {
            nl.ref[A] = cA;
            nl.vis[A] = P.hash[A] >= 0;
        }
        if (GHOST) {
            ghost_search_range(cA, rA * (1.0 + 8.0 * BOUND_REL) + skin, reach, T.g, lo, hi);
        } else {
            partner_search_range(cA, reach, T.g, lo, hi);
        }
        if (occ) {
            // only the cells that hold ghost images
            lo.x = max(lo.x, occ[0]); lo.y = max(lo.y, occ[1]); lo.z = max(lo.z, occ[2]);
            hi.x = min(hi.x, occ[3]); hi.y = min(hi.y, occ[4]); hi.z = min(hi.z, occ[5]);
        }
    }
    const int nx = max(hi.x - lo.x + 1, 0), ny = max(hi.y - lo.y + 1, 0), nz = max(hi.z - lo.z + 1, 0);
    const int ncell = nx * ny * nz;
    const int ncell_max = __reduce_max_sync(full, ncell);
    int cnt = 0;  // partners that passed (uniform over the lane group)
    for (int c0 = 0; c0 < ncell_max; c0 += BROAD_LANES) {
        int B = -1;
        const int ci = c0 + gl;
        if (ci < ncell) {
            const int x = lo.x + ci % nx, y = lo.y + (ci / nx) % ny;
            const int z = lo.z + ci / (nx * ny);
            B = cell_first(T, fd_lin3(x, y, z, T.g.size), build);
        }
        // each lane walks the list of its cell
        while (__any_sync(full, B >= 0)) {
            bool pass = false;
            if (B >= 0 && (GHOST || B > A)) {
                const FdGeo& GB = G.geo[P.geo[B]];
                const double3 cB = GHOST ? gpos[B] : P.pos[B];
                if (NLB) {
                    const double rs = (rA + GB.radius) * (1.0 + 8.0 * BOUND_REL) + nl.skin;
                    pass = lengthSq3(nl_min_image(cA - cB, nl, T.g)) <= rs * rs;
                } else {
                    const double rs = rA + (GHOST ? GB.grid_radius : GB.radius) + skin;
                    if (lengthSq3(cA - cB) <= rs * rs * (1.0 + 4.0 * BOUND_REL))
                        pass = !body_culled32(cA, rA + skin, cB, (GHOST && grot ? grot : P.rot) + 3ll * B, !GHOST,
                                              G.geo32[P.geo[B]], G, probe);
                }
            }
            const unsigned int gm = (__ballot_sync(full, pass) >> gbase) & ((1u << BROAD_LANES) - 1u);
            if (pass) {
                const int pos = cnt + __popc(gm & ((1u << gl) - 1u));
                if (pos < MAX_CAND) s_list[gb][pos] = B;
            }
            cnt += __popc(gm);
            if (B >= 0) B = T.next[B];
        }
    }
    __syncwarp();
    if (valid && cnt > MAX_CAND && gl == 0) set_flag(flags, FD_FLAG_NEIGHBOR_OVERFLOW);
    const int n = min(cnt, MAX_CAND);
    if (NLB) {
        static_assert(NL_MAX >= MAX_CAND, "a list slice holds every partner");
        if (valid) {
            for (int e = gl; e < n; e += BROAD_LANES) {
                const int v = s_list[gb][e];
                int r = 0;
                for (int j = 0; j < n; ++j) r += (s_list[gb][j] < v);
                nl.list[(long long)A * NL_MAX + r] = v;
            }
            if (gl == 0) nl.cnt[A] = n;
        }
        __syncwarp();
        continue;
    }
    int base = 0;
    if (valid && gl == 0 && n > 0) base = atomicAdd(L.n_pairs, n);
    base = __shfl_sync(full, base, 0, BROAD_LANES);
    const bool ok = base + n <= L.cap_pairs;
    if (valid && n > 0 && !ok && gl == 0) set_flag(flags, FD_FLAG_PAIR_OVERFLOW);
    if (valid && gl == 0) {
        L.seg_off[A] = (ok && n > 0) ? base : 0;
        L.seg_cnt[A] = ok ? n : 0;
    }
    // pairs of A in ascending partner order (partners are distinct)
    if (valid && ok) {
        for (int e = gl; e < n; e += BROAD_LANES) {
            const int v = s_list[gb][e];
            int r = 0;
            for (int j = 0; j < n; ++j) r += (s_list[gb][j] < v);
            L.pairA[base + r] = A;
            L.pairB[base + r] = v;
        }
    }
    __syncwarp();
    }
}

// the neighbour list, when a rebuild of it was requested
__global__ void __launch_bounds__(TPB) k_broad_nl(ObjDev P, GeoSetDev G, CellTableDev T, NlDev nl, unsigned int* flags)
{
    __shared__ int s_list[TPB / BROAD_LANES][MAX_CAND];
    if (nl.ctrl[0] == 0) return;
    broad_cells<false, true>(P, G, T, nullptr, nullptr, nullptr, PairListDev{}, nl, flags, 0.0, 0.0, blockIdx.x,
                             gridDim.x, s_list);
}

// neighbour list: request a rebuild when a particle moved more than skin / 2
// since the last build or changed visibility
__global__ void k_nl_check(ObjDev P, NlDev nl, FdGrid g)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const double h = 0.5 * nl.skin;
    const bool moved = lengthSq3(nl_min_image(P.pos[i] - nl.ref[i], nl, g)) > h * h;
    const bool vis = P.hash[i] >= 0;
    if (moved || vis != (nl.vis[i] != 0)) nl.ctrl[0] = 1;
}

// the pairs from the neighbour list: the exact sphere test and the
// body-level cull of the cell search, on the listed partners (ascending, so
// each particle's pairs come out in partner order)
__global__ void __launch_bounds__(TPB) k_nl_filter(ObjDev P, GeoSetDev G, PairListDev L, NlDev nl,
                                                   unsigned int* flags, double probe)
{
    constexpr int LN = 8;  // lanes per particle
    const unsigned int full = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & (LN - 1), gbase = lane & ~(LN - 1);
    const int A = (blockIdx.x * blockDim.x + threadIdx.x) / LN;
    const bool valid = A < P.n;
    double3 cA = mk3(0., 0., 0.);
    double rA = 0.;
    int cnt = 0;
    if (valid) {
        cA = P.pos[A];
        rA = G.geo[P.geo[A]].radius;
        cnt = nl.cnt[A];
    }
    const int cmax = __reduce_max_sync(full, cnt);
    // two passes: count the partners that pass, then write them in order
    unsigned long long passed = 0ull;  // bit e: entry e passed (entries < NL_MAX)
    for (int e0 = 0; e0 < cmax; e0 += LN) {
        const int e = e0 + gl;
        bool pass = false;
        if (valid && e < cnt) {
            const int B = nl.list[(long long)A * NL_MAX + e];
            if (P.hash[B] >= 0) {
                const FdGeo& GB = G.geo[P.geo[B]];
                const double3 cB = P.pos[B];
                const double rs = rA + GB.radius;
                if (lengthSq3(cA - cB) <= rs * rs * (1.0 + 4.0 * BOUND_REL))
                    pass = !body_culled32(cA, rA, cB, P.rot + 3ll * B, true, G.geo32[P.geo[B]], G, probe);
            }
        }
        const unsigned int gm = (__ballot_sync(full, pass) >> gbase) & ((1u << LN) - 1u);
        passed |= (unsigned long long)gm << e0;
    }
    const int n = __popcll(passed);
    int base = 0;
    if (valid && gl == 0 && n > 0) base = atomicAdd(L.n_pairs, n);
    base = __shfl_sync(full, base, 0, LN);
    const bool ok = base + n <= L.cap_pairs;
    if (valid && n > 0 && !ok && gl == 0) set_flag(flags, FD_FLAG_PAIR_OVERFLOW);
    if (valid && gl == 0) {
        L.seg_off[A] = (ok && n > 0) ? base : 0;
        L.seg_cnt[A] = ok ? n : 0;
    }
    if (valid && ok) {
        for (int e = gl; e < cnt; e += LN) {
            if (!((passed >> e) & 1ull)) continue;
            const int r = __popcll(passed & ((1ull << e) - 1ull));
            L.pairA[base + r] = A;
            L.pairB[base + r] = nl.list[(long long)A * NL_MAX + e];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) nl.ctrl[0] = 0;
}

// ---------------------------------------------------------------------------
// pair cache of the particle-particle list (see PairCacheDev)
// ---------------------------------------------------------------------------
// 2 sin(theta / 2) = 2 |vector part of q conj(r)|: the chord a unit lever arm
// sweeps under the rotation from r to q
__device__ __forceinline__ double turn_chord(fd_quat q, fd_quat r)
{
    const double vx = r.q0 * q.q1 - q.q0 * r.q1 - (q.q2 * r.q3 - q.q3 * r.q2);
    const double vy = r.q0 * q.q2 - q.q0 * r.q2 - (q.q3 * r.q1 - q.q1 * r.q3);
    const double vz = r.q0 * q.q3 - q.q0 * r.q3 - (q.q1 * r.q2 - q.q2 * r.q1);
    return 2.0 * sqrt(vx * vx + vy * vy + vz * vz);
}
// the drift bound of particle i since the last build, and a rebuild when it
// exceeds skin / 2 or the particle changed visibility
__device__ __forceinline__ void cache_check(const PairCacheDev& c, int i, double3 x, fd_quat q, bool vis)
{
    const double3 d = x - c.ref_pos[i];
    const double chord = turn_chord(q, c.ref_q[i]);
    const double drift = sqrt(lengthSq3(d)) + c.reach * chord;
    // every particle's bound, for the slot test of the predicate pass
    c.drift[i] = __double2float_ru(drift);
    c.disp[i] = make_float4((float)d.x, (float)d.y, (float)d.z, __double2float_ru(c.reach * chord));
    if (c.ctrl[0] != 0) return;
    if (c.ctrl[2] != 0 || c.ctrl[3] != 0) {
        // the last build overflowed its lists, or the last step asked for a
        // rebuild: build again
        c.ctrl[0] = 1;
        return;
    }
    // a little below skin / 2, so that the two drifts of a pair stay below
    // the single-precision skin the culling stages use
    if (!(drift <= 0.5 * c.skin * (1.0 - 1e-6)) || vis != (c.ref_vis[i] != 0)) c.ctrl[0] = 1;
}
// walls: the drift bound of each wall since the last build (rotation lever
// arm: its SDF-grid radius, the farthest a node inside its grid can be), and
// a rebuild when it exceeds skin / 2 or the wall's cell changed (the
// particle-wall candidates follow the wall's cell)
__device__ __forceinline__ void cache_check_wall(const PairCacheDev& c, int w, double3 x, fd_quat q, long long hash,
                                                 double grid_radius)
{
    const double3 d = x - c.wref_pos[w];
    const double rot = grid_radius * turn_chord(q, c.wref_q[w]);
    const double drift = sqrt(lengthSq3(d)) + rot;
    c.wdrift[w] = __double2float_ru(drift);
    c.wdisp[w] = make_float4((float)d.x, (float)d.y, (float)d.z, __double2float_ru(rot));
    if (c.ctrl[0] != 0) return;
    if (!(drift <= 0.5 * c.skin * (1.0 - 1e-6)) || hash != c.wref_hash[w]) c.ctrl[0] = 1;
}

// The slot bound of a carried pair (see k_slot_filter): lip_B times how far a
// node can have moved in B's frame since the build, plus a margin in units of
// B's grid spacing (the single-precision predicate's rounding).  The node's
// offset from B's centre moved by at most |dc_A - dc_B| + the two rotation
// parts (lever arms up to the reach); the displacements are stored in single
// precision, whose rounding (1e-7 of each) the term 1e-6 (drift_A + drift_B)
// covers; never more than the sum of the two drift bounds.
__device__ __forceinline__ float pair_bound(float driftA, float4 a, float driftB, float4 b, const FdGeo& GB,
                                            float spacing_margin)
{
    const float lip = __double2float_ru(GB.lip);
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    const float dab = __fadd_ru(driftA, driftB);
    const float rel = __fadd_ru(__fadd_ru(__fsqrt_ru(__fadd_ru(__fadd_ru(__fmul_ru(dx, dx), __fmul_ru(dy, dy)),
                                                               __fmul_ru(dz, dz))),
                                          __fadd_ru(a.w, b.w)),
                                __fmul_ru(1e-6f, dab));
    float bound = __fmul_ru(lip, fminf(rel, dab));
    if (spacing_margin > 0.f)
        bound = __fadd_ru(__fmul_ru(bound, 1.000001f), __fmul_ru(spacing_margin, __double2float_ru(GB.spacing)));
    return bound;
}

// wall_range (null: every wall): per particle, the first wall and the number
// of walls it can meet (the walls of its own simulation in a batch of
// simulations tiled into one)
__device__ __forceinline__ void broad_walls(const ObjDev& P, const GeoSetDev& G, const ObjDev& W, const GeoSetDev& GW,
                                            const FdGrid& wg, const PairListDev& L, unsigned int* flags, double probe,
                                            const int2* wall_range, double skin, int A)
{
    const double3 cA = P.pos[A];
    const double rA = G.geo[P.geo[A]].radius;
    int3 lo, hi;
    body_search_range(cA, rA * (1.0 + BOUND_REL) + skin, wg, lo, hi);
    int buf[MAX_CAND];
    int cnt = 0, total = 0;
    const int2 wr = wall_range ? wall_range[A] : make_int2(0, W.n);
    const int wend = min(wr.x + wr.y, W.n);
    for (int w = max(wr.x, 0); w < wend; ++w) {
        const long long h = W.hash[w];
        if (h < 0 || h >= wg.num) continue;
        int3 c;
        decode_cell(h, wg.size, c);
        if (c.x < lo.x || c.x > hi.x || c.y < lo.y || c.y > hi.y || c.z < lo.z || c.z > hi.z) continue;
        const FdGeo& GB = GW.geo[W.geo[w]];
        const double rs = rA + GB.grid_radius + skin;
        const double3 cW = W.pos[w];
        if (lengthSq3(cA - cW) > rs * rs * (1.0 + 4.0 * BOUND_REL)) continue;
        if (body_culled32(cA, rA + skin, cW, W.rot + 3ll * w, false, GW.geo32[W.geo[w]], GW, probe)) continue;
        if (cnt < MAX_CAND) buf[cnt++] = w;
        ++total;
    }
    emit_pairs(A, buf, cnt, total, L, flags);
}

// ---------------------------------------------------------------------------
// contact law, contactKernel.cuh:4-77
// ---------------------------------------------------------------------------
// The contact law runs in kernels of several forms and must give each the same
// bits.  Left plain, its sums of products were contracted one way in one kernel
// and another way in the next, so they are explicit, in the form nvcc gave the
// contact pass.
__device__ __forceinline__ double dot3e(double3 a, double3 b) { return dot3f(a.x, a.y, a.z, b.x, b.y, b.z); }
__device__ __forceinline__ double length3e(double3 v) { return sqrt(dot3e(v, v)); }
__device__ __forceinline__ double3 scale3e(double s, double3 a)
{
    return mk3(__dmul_rn(s, a.x), __dmul_rn(s, a.y), __dmul_rn(s, a.z));
}
// s * a + b
__device__ __forceinline__ double3 axpy3e(double s, double3 a, double3 b)
{
    return mk3(__fma_rn(s, a.x, b.x), __fma_rn(s, a.y, b.y), __fma_rn(s, a.z, b.z));
}
// s * a + t * b
__device__ __forceinline__ double3 sum3e(double s, double3 a, double t, double3 b)
{
    return axpy3e(s, a, scale3e(t, b));
}
__device__ __forceinline__ double3 cross3e(double3 a, double3 b)
{
    return mk3(__fma_rn(a.y, b.z, -__dmul_rn(a.z, b.y)), __fma_rn(a.z, b.x, -__dmul_rn(a.x, b.z)),
               __fma_rn(a.x, b.y, -__dmul_rn(a.y, b.x)));
}

// (the recorded tangential energy's)
__device__ __forceinline__ double spring_sq(double3 v) 
{
    return __fma_rn(v.z, v.z, __fma_rn(v.y, v.y, __dmul_rn(v.x, v.x)));
}

__device__ __forceinline__ double3 sliding_spring(double3 prev, double3 sv, double3 n, double3 fn, double mu,
                                                  double k, double c, double dt)
{
    double3 spring = mk3(0., 0., 0.);
    if (mu > 0. && k > 0.) {
        double3 p1 = axpy3e(-dot3e(prev, n), n, prev);
        const double ap1 = length3e(p1);
        if (!fd_is_zero(ap1)) p1 = scale3e(length3e(prev) / ap1, p1);
        spring = axpy3e(dt, sv, p1);
        double3 sf = sum3e(-k, spring, -c, sv);
        const double asf = length3e(sf);
        const double afn = length3e(fn);
        if (!fd_is_zero(asf) && asf > mu * afn) {
            spring = scale3e(-(1.0 / k), sum3e(mu * afn / asf, sf, c, sv));
        }
    }
    return spring;
}

__device__ __forceinline__ void linear_contact(double3& F, double3& spring, double3 vc, double3 n, double delta,
                                               double dt, double kn, double ks, double mu, double res, double m)
{
    if (delta > 0.) {
        const double lr = log(res);
        const double diss = -lr / (double)sqrtf((float)__fma_rn(lr, lr, PI_D * PI_D));
        const double cn = 2. * diss * (double)sqrtf((float)(m * kn));
        const double vcn = dot3e(vc, n);
        const double3 vn = scale3e(vcn, n);
        const double3 fn = sum3e(kn * delta, n, -cn, vn);
        const double cs = 2. * diss * (double)sqrtf((float)(m * ks));
        const double3 vs = mk3(__dsub_rn(vc.x, vn.x), __dsub_rn(vc.y, vn.y), __dsub_rn(vc.z, vn.z));
        spring = sliding_spring(spring, vs, n, fn, mu, ks, cs, dt);
        const double3 fs = sum3e(-ks, spring, -cs, vs);
        F = mk3(__dadd_rn(fn.x, fs.x), __dadd_rn(fn.y, fs.y), __dadd_rn(fn.z, fs.z));
    } else {
        spring = mk3(0., 0., 0.);
    }
}

// ---------------------------------------------------------------------------
// narrow phase + force, one warp per candidate pair
// ---------------------------------------------------------------------------
struct NarrowArgs {
    ObjDev P;
    GeoSetDev G;
    MatDev M;
    ObjDev W;
    GeoSetDev GW;
    MatDev MW;
    FdGrid pgrid;
    FdGrid wgrid;
    GhostDev gh;
    PairListDev L;
    StepArgs a;
    int with_force;
};

// the slave side of a pair, by kind
template <int KIND> struct Slave;
template <> struct Slave<FD_PP> {
    __device__ static const ObjDev& body(const NarrowArgs& n) { return n.P; }
    __device__ static const double3* pos_of(const NarrowArgs& n) { return n.P.pos; }
    __device__ static const double3* vel_of(const NarrowArgs& n) { return n.P.vel; }
    __device__ static const long long* hash_of(const NarrowArgs& n) { return n.P.hash; }
    __device__ static double3 pos(const NarrowArgs& n, int j) { return n.P.pos[j]; }
    __device__ static const fd_quat* q(const NarrowArgs& n, int j) { return n.P.q + j; }
    __device__ static const float4* rot(const NarrowArgs& n, int j) { return n.P.rot + 3ll * j; }
    __device__ static const FdGeo& geo(const NarrowArgs& n, int j) { return n.G.geo[n.P.geo[j]]; }
    __device__ static const GeoSetDev& set(const NarrowArgs& n) { return n.G; }
    __device__ static long long hash(const NarrowArgs& n, int j) { return n.P.hash[j]; }
    __device__ static const FdGrid& grid(const NarrowArgs& n) { return n.pgrid; }
    static constexpr bool radius_test = true;
};
template <> struct Slave<FD_PW> {
    __device__ static const ObjDev& body(const NarrowArgs& n) { return n.W; }
    __device__ static const double3* pos_of(const NarrowArgs& n) { return n.W.pos; }
    __device__ static const double3* vel_of(const NarrowArgs& n) { return n.W.vel; }
    __device__ static const long long* hash_of(const NarrowArgs& n) { return n.W.hash; }
    __device__ static double3 pos(const NarrowArgs& n, int j) { return n.W.pos[j]; }
    __device__ static const fd_quat* q(const NarrowArgs& n, int j) { return n.W.q + j; }
    __device__ static const float4* rot(const NarrowArgs& n, int j) { return n.W.rot + 3ll * j; }
    __device__ static const FdGeo& geo(const NarrowArgs& n, int j) { return n.GW.geo[n.W.geo[j]]; }
    __device__ static const GeoSetDev& set(const NarrowArgs& n) { return n.GW; }
    __device__ static long long hash(const NarrowArgs& n, int j) { return n.W.hash[j]; }
    __device__ static const FdGrid& grid(const NarrowArgs& n) { return n.wgrid; }
    static constexpr bool radius_test = false;
};
// ghost images: translated images share their body's orientation and
// velocity; sector images carry their own.  The angular velocity is always
// the body's own, as in addGhostLevelSetParticleContactForceTorqueKernel
// (contactKernel.cu:262), which does not turn it with the image.
struct SlaveGhost {
    __device__ static const ObjDev& body(const NarrowArgs& n) { return n.P; }
    __device__ static const double3* pos_of(const NarrowArgs& n) { return n.gh.pos; }
    __device__ static const double3* vel_of(const NarrowArgs& n) { return n.gh.vel ? n.gh.vel : n.P.vel; }
    __device__ static const long long* hash_of(const NarrowArgs& n) { return n.gh.hash; }
    __device__ static double3 pos(const NarrowArgs& n, int j) { return n.gh.pos[j]; }
    __device__ static const fd_quat* q(const NarrowArgs& n, int j) { return (n.gh.q ? n.gh.q : n.P.q) + j; }
    __device__ static const float4* rot(const NarrowArgs& n, int j)
    {
        return (n.gh.rot ? n.gh.rot : n.P.rot) + 3ll * j;
    }
    __device__ static const GeoSetDev& set(const NarrowArgs& n) { return n.G; }
    __device__ static long long hash(const NarrowArgs& n, int j) { return n.gh.hash[j]; }
    __device__ static const FdGrid& grid(const NarrowArgs& n) { return n.pgrid; }
    static constexpr bool radius_test = false;
};
template <> struct Slave<FD_GX> : SlaveGhost {};
template <> struct Slave<FD_GY> : SlaveGhost {};
template <> struct Slave<FD_GXY> : SlaveGhost {};

// The lists of a step share each stage's launch: every stage of every list was
// a launch of its own on one of three streams (75 launches a carried step,
// most of them reading the rebuild flag and returning), and at one or two
// microseconds each they were a third of the step at 65,000 particles.  Each
// list has a range of a launch's blocks.
constexpr int MAX_LISTS = 5;  // of a launch: particle pairs, walls, three image lists
struct ListSet {
    NarrowArgs l[MAX_LISTS];
    int kind[MAX_LISTS];           // FD_PP .. FD_GR270
    int block0[MAX_LISTS + 1];
    int n;
    CellTableDev T;               // the particles' cell table
    const int2* wall_range;       // see broad_walls
    int* rev_total;               // zeroed with the lists' counters (null: no index is built)
    float spacing_margin;         // see pair_bound
};
// the list a block works on, and its place among that list's blocks
__device__ __forceinline__ int list_of(const ListSet& a, int& block, int& nblocks)
{
    int k = 0;
    while (k + 1 < a.n && (int)blockIdx.x >= a.block0[k + 1]) ++k;
    block = (int)blockIdx.x - a.block0[k];
    nblocks = a.block0[k + 1] - a.block0[k];
    return k;
}

// First stage.  A list that is built: its counters cleared, its partners'
// cell table.  A carried one: its pairs and slots are those of the build
// (k_step_end left them in both generations), and each pair gets its slot bound.
__global__ void __launch_bounds__(TPB) k_begin_lists(ListSet a)
{
    int block, nblocks;
    const int li = list_of(a, block, nblocks);
    const NarrowArgs& n = a.l[li];
    const PairListDev& L = n.L;
    const int kind = a.kind[li];
    const bool built = list_built(n.a);
    const int t0 = block * blockDim.x + threadIdx.x, stride = nblocks * blockDim.x;
    if (t0 == 0) {
        *L.n_hits = 0;
        *L.n_test = 0;
        if (built) {
            *L.n_pairs = 0;
            *L.n_slots = 0;
        }
        if (li == 0 && a.rev_total) *a.rev_total = 0;
    }
    if (built) {
        if (kind == FD_PW) return;
        const CellTableDev& T = kind == FD_PP ? a.T : n.gh.cells;
        const long long* hash = kind == FD_PP ? n.P.hash : n.gh.hash;
        const unsigned int build = T.build[T.par];
        for (int i = t0; i < n.P.n; i += stride) cell_link(T, hash[i], build, i);
        return;
    }
    if (!n.a.drift) return;
    const bool wall = kind == FD_PW;
    const float* driftB = n.a.driftB ? n.a.driftB : n.a.drift;
    const float4* dispB = n.a.dispB ? n.a.dispB : n.a.disp;
    const int npairs = min(*L.n_pairs, L.cap_pairs);
    for (int p = t0; p < npairs; p += stride) {
        const int A = L.pairA[p], B = L.pairB[p];
        const FdGeo& GB = wall ? n.GW.geo[n.W.geo[B]] : n.G.geo[n.P.geo[B]];
        L.p_hit[p] = 0;
        L.p_bound[p] = pair_bound(n.a.drift[A], n.a.disp[A], driftB[B], dispB[B], GB, wall ? 0.f : a.spacing_margin);
    }
}

// broad phase of every list that is built
__global__ void __launch_bounds__(TPB) k_broad_lists(ListSet a)
{
    __shared__ int s_list[TPB / BROAD_LANES][MAX_CAND];
    int block, nblocks;
    const int li = list_of(a, block, nblocks);
    const NarrowArgs& n = a.l[li];
    if (!list_built(n.a)) return;
    const double skin = list_skin(n.a);
    if (a.kind[li] == FD_PP) {
        broad_cells<false, false>(n.P, n.G, a.T, nullptr, nullptr, nullptr, n.L, NlDev{}, n.a.flags, n.a.probe, skin,
                                  block, nblocks, s_list);
    } else if (a.kind[li] == FD_PW) {
        for (int A = block * blockDim.x + threadIdx.x; A < n.P.n; A += nblocks * blockDim.x)
            broad_walls(n.P, n.G, n.W, n.GW, n.wgrid, n.L, n.a.flags, n.a.probe, a.wall_range, skin, A);
    } else {
        broad_cells<true, false>(n.P, n.G, n.gh.cells, n.gh.pos, n.gh.rot, n.gh.occ, n.L, NlDev{}, n.a.flags,
                                 n.a.probe, skin, block, nblocks, s_list);
    }
}

// load_quad of what kernels write.  Volatile: without it the asm is a function of
// its address to the compiler, which may then merge two of them or move one
// ahead of a barrier or of step_wait
__device__ __forceinline__ double4 load_four(const double4* p)
{
    double4 v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ fd_quat load_q(const fd_quat* p)
{
    fd_quat v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.q0), "=d"(v.q1), "=d"(v.q2), "=d"(v.q3) : "l"(p));
    return v;
}

// Evaluate node predicate for one node.  Returns true when overlap >= 0 and
// fills the grid fraction and the eight corner values.
template <int KIND, bool FACES>
__device__ __forceinline__ bool node_predicate(const double3 gp, const int3 bcell, const FdGrid& sg, const double3 cB,
                                               const fd_quat qB, const FdGeo& GB, const GeoSetDev& SB, double rB2,
                                               double probe, double& overlap, double& fx, double& fy, double& fz,
                                               double p[8])
{
    int3 lo, hi;
    fd_node_range(gp, sg, lo, hi);
    if (bcell.x < lo.x || bcell.x > hi.x || bcell.y < lo.y || bcell.y > hi.y || bcell.z < lo.z || bcell.z > hi.z)
        return false;
    const double3 rel = mk3(gp.x - cB.x, gp.y - cB.y, gp.z - cB.z);
    if (Slave<KIND>::radius_test) {
        if (xm_len2(rel) > rB2) return false;
    }
    const double3 lp = xm_rrot(rel, qB);
    const double gx = (lp.x - GB.origin.x) * GB.inv_spacing;
    const double gy = (lp.y - GB.origin.y) * GB.inv_spacing;
    const double gz = (lp.z - GB.origin.z) * GB.inv_spacing;
    const int i0 = (int)floor(gx), j0 = (int)floor(gy), k0 = (int)floor(gz);
    if (i0 < 0 || j0 < 0 || k0 < 0) return false;
    if (i0 >= GB.size.x - 1 || j0 >= GB.size.y - 1 || k0 >= GB.size.z - 1) return false;
    fx = gx - (double)i0;
    fy = gy - (double)j0;
    fz = gz - (double)k0;
    const long long sx = GB.size.x, sxy = (long long)GB.size.x * GB.size.y;
    double4 s0, s1;
    load_corners<FACES>(SB, GB.sdf_off + (long long)k0 * sxy + (long long)j0 * sx + i0, sx, sxy, s0, s1);
    p[0] = s0.x; p[1] = s0.y; p[2] = s0.z; p[3] = s0.w;
    p[4] = s1.x; p[5] = s1.y; p[6] = s1.z; p[7] = s1.w;
    overlap = -xm_trilinear(fx, fy, fz, p);
    return overlap >= -probe;
}

// Per-pair rigid transform from A's body frame into B's body frame, in
// FP32, for culling only (the exact predicate stays in FP64):
// p_B = M p_A + t with M = R(qB)^T R(qA), t = R(qB)^T (cA - cB).
struct CullXf {
    float m[9];
    float t[3];
};

// from the single-precision rotation rows of A and B; the product's
// relative error (a few 1e-7) is far below the cull margins
__device__ __forceinline__ CullXf cull_transform(const float4* RA, const float4* RB, const double3 cA,
                                                 const double3 cB)
{
    const float4 a0 = RA[0], a1 = RA[1], a2 = RA[2];
    const float4 b0 = RB[0], b1 = RB[1], b2 = RB[2];
    CullXf x;
    // M = RB^T RA
    x.m[0] = fmaf(b0.x, a0.x, fmaf(b1.x, a1.x, b2.x * a2.x));
    x.m[1] = fmaf(b0.x, a0.y, fmaf(b1.x, a1.y, b2.x * a2.y));
    x.m[2] = fmaf(b0.x, a0.z, fmaf(b1.x, a1.z, b2.x * a2.z));
    x.m[3] = fmaf(b0.y, a0.x, fmaf(b1.y, a1.x, b2.y * a2.x));
    x.m[4] = fmaf(b0.y, a0.y, fmaf(b1.y, a1.y, b2.y * a2.y));
    x.m[5] = fmaf(b0.y, a0.z, fmaf(b1.y, a1.z, b2.y * a2.z));
    x.m[6] = fmaf(b0.z, a0.x, fmaf(b1.z, a1.x, b2.z * a2.x));
    x.m[7] = fmaf(b0.z, a0.y, fmaf(b1.z, a1.y, b2.z * a2.y));
    x.m[8] = fmaf(b0.z, a0.z, fmaf(b1.z, a1.z, b2.z * a2.z));
    const float dx = (float)(cA.x - cB.x), dy = (float)(cA.y - cB.y), dz = (float)(cA.z - cB.z);
    x.t[0] = fmaf(b0.x, dx, fmaf(b1.x, dy, b2.x * dz));
    x.t[1] = fmaf(b0.y, dx, fmaf(b1.y, dy, b2.y * dz));
    x.t[2] = fmaf(b0.z, dx, fmaf(b1.z, dy, b2.z * dz));
    return x;
}

// Cluster culling: true when no node of the cluster can pass the node
// predicate (or, with probe > 0, come within `probe` of B).  Conservative:
// single-precision evaluation with relative margins far above its rounding
// (about 1e-7 relative), bounds that hold in exact arithmetic:
//   * B's bounding sphere (particle pairs: the reference's radius test),
//   * B's SDF grid box (nodes outside it are never contacts),
//   * D(v): lower bound on the distance from grid node v to any cell whose
//     corner minimum is <= 0, 1-Lipschitz in the position,
//   * the Lipschitz bound of the trilinear SDF (coarse grids such as plane
//     walls, where it is tight).
template <int KIND, bool FACES>
__device__ __forceinline__ bool cluster_culled(const float4 cl, const CullXf& x, const FdGeo32& GB,
                                               const GeoSetDev& SB, float probe)
{
    const float cx = cl.x, cy = cl.y, cz = cl.z;
    const float px = fmaf(x.m[0], cx, fmaf(x.m[1], cy, fmaf(x.m[2], cz, x.t[0])));
    const float py = fmaf(x.m[3], cx, fmaf(x.m[4], cy, fmaf(x.m[5], cz, x.t[1])));
    const float pz = fmaf(x.m[6], cx, fmaf(x.m[7], cy, fmaf(x.m[8], cz, x.t[2])));
    return sphere_culled<FACES>(px, py, pz, cl.w, Slave<KIND>::radius_test, GB, SB, probe);
}

// Node filter: true when a node certainly fails the node predicate.  The
// node is mapped into B's frame in single precision (position error below
// perr); it is dropped only when
//   * it lies farther than rB + perr from B's centre (particle pairs), or
//   * it lies outside B's grid box by more than the error, or
//   * (distance-like fields) the single-precision trilinear value exceeds the
//     probe by more than the field's Lipschitz bound times the error, or
//   * it sits inside one cell, away from the cell faces by more than the
//     error, whose eight corner values all exceed the probe (the trilinear
//     value is a convex combination of them).
// Nodes that pass go to the exact double-precision predicate.
//
// NODES nodes at a time (on: the node is there; out: dropped): the chains
// from position to interpolation overlap, and none waits at a branch.
template <int KIND, int NODES, bool FACES>
__device__ __forceinline__ void node_filter(const float4 (&p)[NODES], const bool (&on)[NODES], const CullXf& x,
                                             const FdGeo32& GB, const GeoSetDev& SB, float perr, float probe,
                                             bool (&out)[NODES])
{
    const float is = GB.is;
    const float ge = perr * is + 1e-4f;
    const float hx = (float)(GB.size.x - 1), hy = (float)(GB.size.y - 1), hz = (float)(GB.size.z - 1);
    const float lim = GB.radius + perr;
    float gx[NODES], gy[NODES], gz[NODES];
    bool look[NODES];
#pragma unroll
    for (int u = 0; u < NODES; ++u) {
        const float cx = p[u].x, cy = p[u].y, cz = p[u].z;
        const float px = fmaf(x.m[0], cx, fmaf(x.m[1], cy, fmaf(x.m[2], cz, x.t[0])));
        const float py = fmaf(x.m[3], cx, fmaf(x.m[4], cy, fmaf(x.m[5], cz, x.t[1])));
        const float pz = fmaf(x.m[6], cx, fmaf(x.m[7], cy, fmaf(x.m[8], cz, x.t[2])));
        gx[u] = (px - GB.ox) * is;
        gy[u] = (py - GB.oy) * is;
        gz[u] = (pz - GB.oz) * is;
        out[u] = !on[u] || (Slave<KIND>::radius_test && px * px + py * py + pz * pz > lim * lim) || gx[u] < -ge ||
                 gy[u] < -ge || gz[u] < -ge || gx[u] > hx + ge || gy[u] > hy + ge || gz[u] > hz + ge;
        look[u] = !out[u] && !(gx[u] < ge || gy[u] < ge || gz[u] < ge || gx[u] > hx - ge || gy[u] > hy - ge ||
                               gz[u] > hz - ge);
    }
    if (GB.tight) {
        const long long sx = GB.size.x, sxy = (long long)GB.size.x * GB.size.y;
        float4 s0[NODES], s1[NODES];
#pragma unroll
        for (int u = 0; u < NODES; ++u) {
            // a node that needs no look reads the pool's first point
            const long long i =
                look[u] ? GB.sdf_off + (long long)(int)gz[u] * sxy + (long long)(int)gy[u] * sx + (int)gx[u] : 0ll;
            load_corners<FACES>(SB, i, look[u] ? sx : 0ll, look[u] ? sxy : 0ll, s0[u], s1[u]);
        }
#pragma unroll
        for (int u = 0; u < NODES; ++u) {
            const float fx = gx[u] - (int)gx[u], fy = gy[u] - (int)gy[u], fz = gz[u] - (int)gz[u];
            const float c00 = s0[u].x * (1.f - fx) + s0[u].y * fx;
            const float c10 = s0[u].z * (1.f - fx) + s0[u].w * fx;
            const float c01 = s1[u].x * (1.f - fx) + s1[u].y * fx;
            const float c11 = s1[u].z * (1.f - fx) + s1[u].w * fx;
            const float phi = (c00 * (1.f - fy) + c10 * fy) * (1.f - fz) + (c01 * (1.f - fy) + c11 * fy) * fz;
            const float slack = GB.lip * perr + 1e-5f * (fabsf(phi) + GB.spacing);
            if (look[u]) out[u] = phi - probe > slack;
        }
        return;
    }
    // the trilinear value anywhere the node can be (within ge of its
    // single-precision position, in grid units) is at least the smallest
    // corner minimum over the cells that box touches (one to a few cells:
    // two per axis where the node is within ge of a cell face)
    const long long rx = GB.size.x - 1, rxy = (long long)(GB.size.y - 1) * (GB.size.x - 1);
    const float* CM = SB.cellmin + GB.cellmin_off;
    for (int u = 0; u < NODES; ++u) {
        if (!look[u]) continue;
        const int ilo = max((int)floorf(gx[u] - ge), 0), ihi = min((int)floorf(gx[u] + ge), GB.size.x - 2);
        const int jlo = max((int)floorf(gy[u] - ge), 0), jhi = min((int)floorf(gy[u] + ge), GB.size.y - 2);
        const int klo = max((int)floorf(gz[u] - ge), 0), khi = min((int)floorf(gz[u] + ge), GB.size.z - 2);
        if (ihi - ilo > 2 || jhi - jlo > 2 || khi - klo > 2) continue;  // a margin of more than a cell: keep
        bool above = true;
        for (int k = klo; k <= khi && above; ++k)
            for (int j = jlo; j <= jhi && above; ++j)
                for (int i = ilo; i <= ihi && above; ++i) above = !(__ldg(CM + k * rxy + j * rx + i) <= probe);
        out[u] = above;
    }
}

// The nodes of A that may pass the predicate against B, for one warp:
// cluster culling with one cluster per lane, then the single-precision filter
// over the nodes of the surviving clusters.  Their keys go to queue in
// cluster order; returns how many, and the clusters kept.  NODES: clusters
// filtered at a time.  One where there are warps enough to hide the waits (two
// take the registers of a quarter of them: a rebuild's selection 1.5 against
// 1.4 ms at 262,144 particles), two where a warp has an SM's share to itself
// (a step of 1,000 particles 38.4 against 39.6 us).
template <int KIND, int NODES, bool FACES = false>
__device__ __forceinline__ int cull_pair(const NarrowArgs& n, int A, int B, double skin, int lane,
                                         unsigned short* queue, int& kept)
{
    const unsigned int lt_mask = (1u << lane) - 1u;
    const int gA = n.P.geo[A], gB = Slave<KIND>::body(n).geo[B];
    const double3 cA = n.P.pos[A];
    const double3 cB = Slave<KIND>::pos(n, B);
    const GeoSetDev& SB = Slave<KIND>::set(n);
    const FdGeo32& GA = n.G.geo32[gA];
    const FdGeo32& GB = SB.geo32[gB];
    const float probe = (float)n.a.probe;
    const int ncl = GA.clus_count;
    if (ncl > MAX_CLUSTERS) set_flag(n.a.flags, FD_FLAG_CLUSTER_OVERFLOW);
    unsigned long long keep = 0ull;
    const CullXf xf = cull_transform(n.P.rot + 3ll * A, Slave<KIND>::rot(n, B), cA, cB);
    for (int c0 = 0; c0 < min(ncl, MAX_CLUSTERS); c0 += 32) {
        const int c = c0 + lane;
        bool k = false;
        if (c < ncl) {
            float4 cl = n.G.clus_sphere[GA.clus_off + c];
            cl.w += (float)skin;
            k = !cluster_culled<KIND, FACES>(cl, xf, GB, SB, probe);
        }
        keep |= ((unsigned long long)__ballot_sync(0xffffffffu, k)) << c0;
    }
    kept = __popcll(keep);
    const float perr = 4e-6f * (float)(length3(cA - cB) + n.G.geo[gA].radius + SB.geo[gB].radius + SB.geo[gB].spacing) +
                       (float)skin;
    int ncand = 0;
    // the next clusters' ranges and nodes are loaded while these are filtered:
    // range, node and grid values are three dependent loads a cluster
    int2 r[NODES];
    float4 node[NODES];
    auto fetch = [&] {
#pragma unroll
        for (int u = 0; u < NODES; ++u) {
            r[u] = make_int2(0, 0);
            if (!keep) continue;
            const int c = __ffsll((long long)keep) - 1;
            keep &= keep - 1ull;
            r[u] = n.G.clus_range[GA.clus_off + c];
            if (lane < r[u].y) node[u] = n.G.nodes32[GA.node_off + r[u].x + lane];
        }
    };
#pragma unroll
    for (int u = 0; u < NODES; ++u) node[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    fetch();
    for (int left = kept; left > 0; left -= NODES) {
        int first[NODES];
        float4 p[NODES];
        bool on[NODES], out[NODES];
#pragma unroll
        for (int u = 0; u < NODES; ++u) {
            first[u] = r[u].x;
            p[u] = node[u];
            on[u] = lane < r[u].y;
        }
        if (left > NODES) fetch();
        node_filter<KIND, NODES, FACES>(p, on, xf, GB, SB, perr, probe, out);
#pragma unroll
        for (int u = 0; u < NODES; ++u) {
            const unsigned int m = __ballot_sync(0xffffffffu, !out[u]);
            if (!out[u]) queue[ncand + __popc(m & lt_mask)] = (unsigned short)(first[u] + lane);
            ncand += __popc(m);
        }
    }
    __syncwarp();
    return ncand;
}

// the slots of the pair (A, B) in the previous step's list, for one warp
__device__ __forceinline__ void find_history(const PairListDev& L, int A, int B, int lane, int& off, int& cnt)
{
    off = cnt = 0;
    const int os = L.o_seg_off[A], on = L.o_seg_cnt[A];
    int found = -1;
    for (int k0 = 0; k0 < on && found < 0; k0 += 32) {
        const int k = k0 + lane;
        const bool eq = (k < on) && (L.o_pairB[os + k] == B);
        const unsigned int m = __ballot_sync(0xffffffffu, eq);
        if (m) found = os + k0 + __ffs(m) - 1;
    }
    if (found >= 0) { off = L.o_c_off[found]; cnt = L.o_c_cnt[found]; }
}

// ---------------------------------------------------------------------------
// narrow phase, stage 1: one warp per candidate pair.  The clusters of A's
// surface nodes are culled against B, the nodes of the surviving clusters are
// filtered in single precision, and the nodes that may pass the exact
// predicate become the pair's contact slots (contiguous, in cluster order).
// The warp also finds the pair in the previous step's list, the history
// source of its contacts.
// ---------------------------------------------------------------------------
//
// With the pair cache it runs only on rebuild steps, and every culling margin
// is widened by the skin: a cluster
// is kept when it may come within reach of B after moves of up to the skin,
// a node is slotted when it may pass the predicate after such moves.
template <int KIND>
__device__ __forceinline__ void select_list(const NarrowArgs& n, int block, int nblocks,
                                            unsigned short (*s_node)[MAX_NODE_QUEUE], unsigned long long* s_stats)
{
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const PairListDev& L = n.L;
    const int npairs = min(*L.n_pairs, L.cap_pairs);
    const int nwarps = nblocks * NARROW_WARPS;
    const double skin = list_skin(n.a);
    for (int p = block * NARROW_WARPS + wib; p < npairs; p += nwarps) {
        const int A = L.pairA[p];
        const int B = L.pairB[p];
        int kept;
        int ncand = cull_pair<KIND, 1>(n, A, B, skin, lane, s_node[wib], kept);
        if (n.a.stats && lane == 0) {
            atomicAdd(&s_stats[0], 1ull);
            atomicAdd(&s_stats[1], (unsigned long long)min(n.G.geo[n.P.geo[A]].clus_count, MAX_CLUSTERS));
            atomicAdd(&s_stats[2], (unsigned long long)kept);
            atomicAdd(&s_stats[3], (unsigned long long)ncand);
        }
        // ---- contact slots of the pair
        int base = 0;
        if (ncand > 0) {
            if (lane == 0) base = atomicAdd(L.n_slots, ncand);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base + ncand > L.cap_contacts) {
                if (lane == 0) set_flag(n.a.flags, FD_FLAG_CONTACT_OVERFLOW);
                base = 0;
                ncand = 0;
            }
        }
        if (ncand > 0) {
            // history: the same pair in the previous step's list
            int oc_off, oc_cnt;
            find_history(L, A, B, lane, oc_off, oc_cnt);
            for (int i = lane; i < ncand; i += 32) {
                L.c_pair[base + i] = p;
                L.c_k[base + i] = s_node[wib][i];
            }
            if (lane == 0) {
                int3 bcell;
                decode_cell(Slave<KIND>::hash(n, B), Slave<KIND>::grid(n).size, bcell);
                L.p_aux[p] = make_int4(bcell.x, bcell.y, bcell.z, oc_off);
                L.p_hist_cnt[p] = oc_cnt;
            }
        }
        if (lane == 0) {
            L.c_off[p] = base;
            L.c_cnt[p] = ncand;
            L.p_hit[p] = 0;
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(NARROW_WARPS * 32, FD_SELECT_MIN_BLOCKS) k_select_lists(ListSet a)
{
    __shared__ unsigned short s_node[NARROW_WARPS][MAX_NODE_QUEUE];
    // work counters, summed per block and added to the global ones once
    __shared__ unsigned long long s_stats[4];
    int block, nblocks;
    const int li = list_of(a, block, nblocks);
    const NarrowArgs& n = a.l[li];
    if (!list_built(n.a)) return;
    if (n.a.stats && threadIdx.x < 4) s_stats[threadIdx.x] = 0ull;
    __syncthreads();
    // the sector images differ from the translated ones only in the state the
    // ghost traits read: one instance serves every image list
    if (a.kind[li] == FD_PP) select_list<FD_PP>(n, block, nblocks, s_node, s_stats);
    else if (a.kind[li] == FD_PW) select_list<FD_PW>(n, block, nblocks, s_node, s_stats);
    else select_list<FD_GX>(n, block, nblocks, s_node, s_stats);
    if (n.a.stats) {
        __syncthreads();
        if (threadIdx.x < 4 && s_stats[threadIdx.x]) {
            // pairs, clusters, clusters kept, nodes given the exact predicate
            const int slot[4] = {0, 1, 2, 4};
            atomicAdd(&n.a.stats[slot[threadIdx.x]], s_stats[threadIdx.x]);
        }
    }
}

// ---------------------------------------------------------------------------
// pair cache, particle-particle list, carried steps: the slots the predicate
// pass must test.  A slot is skipped when its node was outside B at the
// rebuild by more than the SDF can change under the pair's relative motion
// since (|grad phi| <= lip, the trilinear bound; k_begin_lists stored the
// pair's bound); the others are listed, so that the predicate pass runs full warps.
// The wall and image lists are short: there the extra pass cost more than
// the idle lanes, and the predicate pass tests the bound itself.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(TPB) k_slot_filter(NarrowArgs n)
{
    const PairListDev& L = n.L;
    if (list_built(n.a)) return;
    const int nitems = min(*L.n_slots, L.cap_contacts);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // a block's pass covers SF_UNROLL * TPB slots (slot s0 + u * TPB + tid
    // for u = 0 .. SF_UNROLL - 1), listed in slot order with one atomic: one
    // slot per thread and pass spent a third of its issue slots waiting at
    // the pass's barriers
    constexpr int SF_UNROLL = 4;
    constexpr int NW = TPB / 32;
    const long long stride = (long long)gridDim.x * blockDim.x * SF_UNROLL;
    __shared__ int w_count[SF_UNROLL * NW];
    __shared__ int b_base;
    int tested = 0, skipped = 0;
    for (long long s0 = (long long)blockIdx.x * blockDim.x * SF_UNROLL; s0 < nitems; s0 += stride) {
        int sl[SF_UNROLL], pr[SF_UNROLL];
        bool in[SF_UNROLL];
        float phi0[SF_UNROLL];
#pragma unroll
        for (int u = 0; u < SF_UNROLL; ++u) {
            const long long t = s0 + u * TPB + threadIdx.x;
            in[u] = t < nitems;
            sl[u] = in[u] ? (int)t : 0;
            pr[u] = in[u] ? L.c_pair[sl[u]] : 0;
            phi0[u] = in[u] ? L.c_phi0[sl[u]] : 0.f;
        }
        unsigned int m[SF_UNROLL];
#pragma unroll
        for (int u = 0; u < SF_UNROLL; ++u) {
            bool keep = false;
            if (in[u]) {
                keep = !(phi0[u] > __fadd_ru(L.p_bound[pr[u]], 1e-12f));
                if (!keep) L.c_node[sl[u]] = -1;
            }
            m[u] = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) w_count[u * NW + warp] = __popc(m[u]);
            tested += __popc(m[u]);
            skipped += __popc(__ballot_sync(0xffffffffu, in[u])) - __popc(m[u]);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int total = 0;
            for (int w = 0; w < SF_UNROLL * NW; ++w) {
                const int c = w_count[w];
                w_count[w] = total;
                total += c;
            }
            b_base = total ? atomicAdd(L.n_test, total) : 0;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < SF_UNROLL; ++u)
            if ((m[u] >> lane) & 1u)
                L.c_test[b_base + w_count[u * NW + warp] + __popc(m[u] & ((1u << lane) - 1u))] = sl[u];
        __syncthreads();
    }
    if (n.a.stats && lane == 0) {
        if (tested) atomicAdd(&n.a.stats[5], (unsigned long long)tested);
        if (skipped) atomicAdd(&n.a.stats[6], (unsigned long long)skipped);
    }
}

// ---------------------------------------------------------------------------
// narrow phase, stage 2, in two passes: one thread per contact slot runs the
// exact double-precision node predicate (LSParticleContactDetectionKernel.cu:
// 37-119); one thread per contact the normal, the contact point, the history
// carried over from the previous step (first match on the node, :288-297) and
// the contact law (contactKernel.cu:46-291).  A slot whose node is not in
// contact keeps node id -1.  Force and torques go to the contact's record;
// stage 3 sums them per pair.
// ---------------------------------------------------------------------------
// What the predicate reads of a slot's two bodies, and with law what the
// contact law does.  All of it is independent, and the asm keeps it in one
// place: left to itself the compiler places each load near its use, some
// thirty waits of a microsecond one after the other in the contact pass.
struct PairState {
    double3 xA, xB, vA, vB, wA, wB;
    fd_quat qA, qB;
    long long hB;
    int gA, gB, mA, mB, nodes;
    int hnode, hat;  // a carried slot: its previous self's node id and place (see contact_list)
    bool carried;
};
__device__ __forceinline__ double load_now(const double* p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int load_now(const int* p)
{
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ long long load_now(const long long* p)
{
    long long v;
    asm volatile("ld.global.s64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double3 load_now(const double3* p)
{
    return make_double3(load_now(&p->x), load_now(&p->y), load_now(&p->z));
}
__device__ __forceinline__ fd_quat load_now(const fd_quat* p)
{
    fd_quat v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.q0), "=d"(v.q1), "=d"(v.q2), "=d"(v.q3) : "l"(p));
    return v;
}
template <int KIND, bool LAW>
__device__ __forceinline__ PairState load_pair(const NarrowArgs& n, int A, int B)
{
    const ObjDev& O = Slave<KIND>::body(n);
    PairState st;
    st.carried = false;
    if (!LAW) {
        // the predicate pass: more warps hide the waits, and more registers
        // would cost them
        st.gA = n.P.geo[A];
        st.gB = O.geo[B];
        st.hB = Slave<KIND>::hash_of(n)[B];
        st.xA = n.P.pos[A];
        st.qA = load_q(n.P.q + A);
        st.xB = Slave<KIND>::pos_of(n)[B];
        st.qB = load_q(Slave<KIND>::q(n, B));
        return st;
    }
    st.gA = load_now(n.P.geo + A);
    st.gB = load_now(O.geo + B);
    st.hB = load_now(Slave<KIND>::hash_of(n) + B);
    st.xA = load_now(n.P.pos + A);
    st.qA = load_now(n.P.q + A);
    st.xB = load_now(Slave<KIND>::pos_of(n) + B);
    st.qB = load_now(Slave<KIND>::q(n, B));
    st.mA = load_now(n.P.mat + A);
    st.mB = load_now(O.mat + B);
    st.nodes = load_now(n.P.node_base + A);
    st.vA = load_now(n.P.vel + A);
    st.wA = load_now(n.P.angvel + A);
    st.vB = load_now(Slave<KIND>::vel_of(n) + B);
    st.wB = load_now(O.angvel + B);
    return st;
}

// one slot's node against its partner
struct SlotEval {
    double3 cA, cB, r, gp;  // centres, node offset from A's centre, node
    fd_quat qB;
    int pool;               // the node in the node pools
    double ov, fx, fy, fz, pv[8];
};

// the exact predicate of node k (relative to the geometry) of A against B (st);
// e.ov keeps ov0 when the predicate stops before the distance
template <int KIND, bool FACES = false>
__device__ __forceinline__ bool slot_predicate(const NarrowArgs& n, const PairState& st, int k, int3 bcell, double ov0,
                                               SlotEval& e)
{
    const FdGeo& GA = n.G.geo[st.gA];
    e.cA = st.xA;
    const fd_quat qA = st.qA;
    e.cB = st.xB;
    e.qB = st.qB;
    const GeoSetDev& SB = Slave<KIND>::set(n);
    const FdGeo& GB = SB.geo[st.gB];
    const FdGrid& sg = Slave<KIND>::grid(n);
    const double rB2 = GB.radius * GB.radius;
    e.pool = GA.node_off + k;
    const double3 node = n.G.nodes[e.pool];
    e.r = xm_rot(qA, node);
    e.gp = mk3(e.r.x + e.cA.x, e.r.y + e.cA.y, e.r.z + e.cA.z);
    e.ov = ov0;
    return node_predicate<KIND, FACES>(e.gp, bcell, sg, e.cB, e.qB, GB, SB, rB2, n.a.probe, e.ov, e.fx, e.fy, e.fz, e.pv);
}

// A contact's results go out in 16-byte stores to six whole sectors, side by
// side with the next contact's (at place t of c_hist and c_rec).  As nine
// arrays with an entry per slot they were 22 stores to some fifteen part-written
// sectors, spread over 2.5 GB for 262,144 particles, and the sums read them
// back from there.  That took the contact pass
// from 112 to 88 us, the sums from 65 to 57.
__device__ __forceinline__ void store_hist(const PairListDev& L, int t, double3 spring, int B)
{
    double2* o = reinterpret_cast<double2*>(L.c_hist + t);
    o[0] = make_double2(spring.x, spring.y);
    o[1] = make_double2(spring.z, __hiloint2double(0, B));
}
__device__ __forceinline__ void store_record(const PairListDev& L, int t, double3 pt, double3 nrm, double ov,
                                             double en, double es)
{
    double2* o = reinterpret_cast<double2*>(L.c_rec + (long long)CONTACT_REC * t + CONTACT_POINT);
    o[0] = make_double2(pt.x, pt.y);
    o[1] = make_double2(pt.z, nrm.x);
    o[2] = make_double2(nrm.y, nrm.z);
    o[3] = make_double2(ov, en);
    reinterpret_cast<double*>(o)[8] = es;
}
__device__ __forceinline__ void store_force(const PairListDev& L, int t, const double f[9])
{
    double2* o = reinterpret_cast<double2*>(L.c_rec + (long long)CONTACT_REC * t);
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = make_double2(f[2 * k], f[2 * k + 1]);
    reinterpret_cast<double*>(o)[8] = f[8];
}
__device__ __forceinline__ void store_force(const PairListDev& L, int t, const float f[9])
{
    float4* o = reinterpret_cast<float4*>(L.c_rec + (long long)CONTACT_REC * t);
    o[0] = make_float4(f[0], f[1], f[2], f[3]);
    o[1] = make_float4(f[4], f[5], f[6], f[7]);
    reinterpret_cast<float*>(o)[8] = f[8];
}

// Slot s of list L, a contact by the predicate e: normal, contact point,
// history (the pair's previous slots are oc_off .. oc_off + oc_cnt - 1),
// records, and with forces the contact law, whose force and torques on A and B
// go to o.  Returns the global boundary-node id.
template <int KIND>
__device__ __forceinline__ int contact_law(const NarrowArgs& n, const PairListDev& L, const AdjRec& R, int s, int t, int A,
                                           int B, const PairState& st, int k, int oc_off, int oc_cnt,
                                           const SlotEval& e, double o[9])
{
    const bool periodic = (KIND == FD_PP || KIND == FD_PW) && (n.a.periodic_x || n.a.periodic_y);
    const FdGeo& GA = n.G.geo[st.gA];
    const FdGeo& GB = Slave<KIND>::set(n).geo[st.gB];
    const double3 cA = e.cA, cB = e.cB, r = e.r, gp = e.gp;
    const fd_quat qB = e.qB;
    const double ov = e.ov;
    const int pool = e.pool;
    double3 nrm = fd_gradient_q(e.fx, e.fy, e.fz, e.pv);
    nrm = fd_rot(qB, nrm);
    nrm = fd_normalize(nrm);
    const double3 pt = gp + (0.5 * ov) * nrm;
    const int nid = st.nodes + n.G.node_lid[pool];
    double3 spring = mk3(0., 0., 0.);
    int hist = -1;
    if (st.carried) {
        // a carried layout keeps each slot's previous self at its index
        if (st.hnode == nid) hist = s;
        if (hist >= 0) {
            const double4 h = load_four(L.o_c_hist + st.hat);
            spring = mk3(h.x, h.y, h.z);
        }
    } else {
        // the previous slots of the pair are ascending in node
        // key; a node appears at most once per pair.
        const int oc_end = oc_off + oc_cnt;
        int lo = oc_off, hi = oc_end;
        if (s >= oc_off && s < oc_end && L.o_c_k[s] == k) lo = hi = s;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (L.o_c_k[mid] < k) lo = mid + 1; else hi = mid;
        }
        if (lo < oc_end && L.o_c_k[lo] == k) {
            const int at = L.o_c_at[lo];
            if (L.o_c_node[lo] == nid) {
                const double4 h = load_four(L.o_c_hist + at);
                spring = mk3(h.x, h.y, h.z);
                hist = lo;
            }
        }
    }
    if (R.hit && s < R.cap) {
        R.A[s] = A;
        R.B[s] = B;
        R.Bp[s] = KIND == FD_PW ? -1 : B;
        R.geoB[s] = KIND == FD_PW ? n.W.geo[B] : n.P.geo[B];
        R.matB[s] = KIND == FD_PW ? n.W.mat[B] : n.P.mat[B];
        R.nid[s] = nid;
        R.hist[s] = hist;
        R.rel[3 * s + 0] = gp.x - cB.x;
        R.rel[3 * s + 1] = gp.y - cB.y;
        R.rel[3 * s + 2] = gp.z - cB.z;
        R.sprev[3 * s + 0] = spring.x;
        R.sprev[3 * s + 1] = spring.y;
        R.sprev[3 * s + 2] = spring.z;
        R.qB[4 * s + 0] = qB.q0;
        R.qB[4 * s + 1] = qB.q1;
        R.qB[4 * s + 2] = qB.q2;
        R.qB[4 * s + 3] = qB.q3;
        R.arm[3 * s + 0] = r.x;
        R.arm[3 * s + 1] = r.y;
        R.arm[3 * s + 2] = r.z;
        R.wrap[s] = 13 + 27;  // no shift unless the force side records one
    }
    double kn = 0., ks = 0.;
    if (n.with_force) {
        // force-side state (positions after the periodic wrap,
        // LSSolver.h:1175-1190)
        double3 ri = cA, rj = cB;
        if (periodic) {
            if (n.a.periodic_x) { ri = wrap_x(ri, n.pgrid); if (KIND == FD_PP) rj = wrap_x(rj, n.pgrid); }
            if (n.a.periodic_y) { ri = wrap_y(ri, n.pgrid); if (KIND == FD_PP) rj = wrap_y(rj, n.pgrid); }
        }
        double3 vi = st.vA, vjs = st.vB;
        const double3 wi = st.wA, wj = st.wB;
        if ((KIND == FD_PP || KIND == FD_PW) && n.a.sector) {
            sector_fold(ri, vi, n.pgrid.minb);
            if (KIND == FD_PP) sector_fold(rj, vjs, n.pgrid.minb);
        }
        const int mi = st.mA;
        const double invMi = GA.inv_mass;
        const double kni = n.M.kn[mi], ksi = n.M.ks[mi], mui = n.M.mu[mi], ei = n.M.e[mi];
        double3 vj;
        double effM = 0., mu, res;
        if (KIND == FD_PW) {
            vj = vjs;
            const int mj = st.mB;
            mu = fmin(mui, n.MW.mu[mj]);
            res = fmin(ei, n.MW.e[mj]);
            if (invMi > 0.) effM = 1. / invMi;
            kn = kni;
            ks = ksi;
        } else {
            vj = vjs;
            const double invMj = GB.inv_mass;
            const int mj = st.mB;
            const double knj = n.M.kn[mj], ksj = n.M.ks[mj];
            if (kni > 0. && knj > 0.) kn = kni * knj / (kni + knj);
            if (ksi > 0. && ksj > 0.) ks = ksi * ksj / (ksi + ksj);
            if (invMi > 0. || invMj > 0.) effM = 1. / (invMi + invMj);
            res = fmin(ei, n.M.e[mj]);
            mu = fmin(mui, n.M.mu[mj]);
        }
        const double3 vc = (vi + cross3e(wi, pt - ri)) - (vj + cross3e(wj, pt - rj));
        if (R.hit && s < R.cap) {
            R.vc[3 * s + 0] = vc.x;
            R.vc[3 * s + 1] = vc.y;
            R.vc[3 * s + 2] = vc.z;
            R.wrap[s] = wrap_code(cA, ri, cB, rj, n.pgrid);
        }
        double3 F = mk3(0., 0., 0.);
        linear_contact(F, spring, vc, nrm, ov, n.a.dt, kn, ks, mu, res, effM);
        const double3 TA = cross3e(pt - ri, F);
        const double3 TB = cross3e(F, pt - rj);
        o[0] = F.x; o[1] = F.y; o[2] = F.z;
        o[3] = TA.x; o[4] = TA.y; o[5] = TA.z;
        o[6] = TB.x; o[7] = TB.y; o[8] = TB.z;
    }
    L.c_at[s] = t;
    store_hist(L, t, spring, B);
    if (n.a.records) {
        if (!n.with_force) {
            const int mi = st.mA;
            kn = n.M.kn[mi];
            ks = n.M.ks[mi];
            if (KIND != FD_PW) {
                const int mj = st.mB;
                const double knj = n.M.kn[mj], ksj = n.M.ks[mj];
                kn = (kn > 0. && knj > 0.) ? kn * knj / (kn + knj) : 0.;
                ks = (ks > 0. && ksj > 0.) ? ks * ksj / (ks + ksj) : 0.;
            }
        }
        store_record(L, t, pt, nrm, ov, 0.5 * ov * ov * kn, 0.5 * spring_sq(spring) * ks);
    }
    return nid;
}

template <int KIND, int PASS>
__device__ __forceinline__ void contact_list(const NarrowArgs& n, int block, int nblocks)
{
    const PairListDev& L = n.L;
    // pair cache (particle-particle, particle-wall and translated image
    // lists, predicate pass): a rebuild step tests every slot and stores its
    // bound; a carried step tests the slots k_slot_filter listed (the
    // particle-particle list) or tests the slot bound here (the others).  An
    // image list under the cache also holds the pairs of particles that have
    // no image entry this step: their slots hold no contact.
    constexpr bool IMAGE = KIND != FD_PP && KIND != FD_PW;
    const bool cache = n.a.gate != nullptr;
    const bool carried = !list_built(n.a);
    const bool listed = KIND == FD_PP && PASS == 0 && carried;
    const bool slot_test = PASS == 0 && carried && !listed;
    const bool phi0_store = PASS == 0 && cache && !carried;
    const bool live_test = IMAGE && PASS == 0 && n.gh.live != nullptr;
    // pass 0: every slot (or the listed ones); pass 1: the slots pass 0
    // listed as contacts
    const int nitems = PASS == 0 ? min(listed ? *L.n_test : *L.n_slots, L.cap_contacts)
                                 : min(*L.n_hits, L.cap_contacts);
    const int lane = threadIdx.x & 31;
    const int stride = nblocks * blockDim.x;
    int hits = 0;
    for (int s0 = block * blockDim.x + (threadIdx.x & ~31); s0 < nitems; s0 += stride) {
        const int t = s0 + lane;
        bool continue_slot = false;
        const int s = t < nitems ? (PASS == 1 ? L.c_hit[t] : listed ? L.c_test[t] : t) : t;
        bool hit = false;
        if ((slot_test || live_test) && t < nitems) {
            const int p = L.c_pair[s];
            if (live_test && !n.gh.live[L.pairB[p]]) {
                L.c_node[s] = -1;
                if (phi0_store) L.c_phi0[s] = __int_as_float(0xff800000);  // -inf: never skipped
                continue_slot = true;
            } else if (slot_test && L.c_phi0[s] > __fadd_ru(L.p_bound[p], 1e-12f)) {
                // the bound k_slot_filter tests for the particle-particle list
                L.c_node[s] = -1;
                continue_slot = true;
            }
        }
        if (t < nitems && !continue_slot) {
            const int p = L.c_pair[s];
            const int k = L.c_k[s];
            const int A = L.pairA[p];
            const int B = L.pairB[p];
            // a carried slot's history is its previous self, and its partner's
            // cell this step's
            PairState st = load_pair<KIND, PASS == 1>(n, A, B);
            if (PASS == 1 && carried) {
                st.carried = true;
                st.hnode = load_now(L.o_c_node + s);
                st.hat = load_now(L.o_c_at + s);
            }
            int4 aux = make_int4(0, 0, 0, s);
            int hist = 1;
            if (carried) {
                int3 bc;
                decode_cell(st.hB, Slave<KIND>::grid(n).size, bc);
                aux.x = bc.x; aux.y = bc.y; aux.z = bc.z;
            } else {
                aux = L.p_aux[p];
                hist = L.p_hist_cnt[p];
            }
            SlotEval e;
            // an overlap the predicate did not reach stays +inf (a slot that
            // is never skipped)
            hit = slot_predicate<KIND>(n, st, k, make_int3(aux.x, aux.y, aux.z),
                                       PASS == 0 ? __longlong_as_double(0x7ff0000000000000ll) : 0., e);
            if (phi0_store) L.c_phi0[s] = __double2float_rd(-e.ov);
            int nid = -1;
            if (PASS == 1 && hit) {
                double o[9];
                nid = contact_law<KIND>(n, L, n.a.rec, s, t, A, B, st, k, aux.w, hist, e, o);
                if (n.with_force) store_force(L, t, o);
            }
            if (PASS == 1) {
                L.c_node[s] = nid;
            } else {
                if (hit) L.p_hit[p] = 1;
                else L.c_node[s] = -1;
                if (n.a.rec.hit && s < n.a.rec.cap) n.a.rec.hit[s] = hit ? 1 : 0;
            }
        }
        if (PASS == 0 && cache && !listed && n.a.stats) {
            // slots given the exact predicate, slots skipped (k_slot_filter
            // counts the listed steps)
            const unsigned int tested = __ballot_sync(0xffffffffu, t < nitems && !continue_slot);
            const unsigned int skipped = __ballot_sync(0xffffffffu, continue_slot);
            if (lane == 0 && tested) atomicAdd(&n.a.stats[5], (unsigned long long)__popc(tested));
            if (lane == 0 && skipped) atomicAdd(&n.a.stats[6], (unsigned long long)__popc(skipped));
        }
        if (PASS == 0) {
            // contacts are listed for pass 1, one atomic per warp
            const unsigned int m = __ballot_sync(0xffffffffu, hit);
            if (m) {
                int base = 0;
                if (lane == 0) base = atomicAdd(L.n_hits, __popc(m));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (hit) L.c_hit[base + __popc(m & ((1u << lane) - 1u))] = s;
                hits += __popc(m);
            }
        }
    }
    if (PASS == 0 && n.a.stats && lane == 0 && hits) atomicAdd(&n.a.stats[3], (unsigned long long)hits);
}

// ---------------------------------------------------------------------------
// narrow phase, stage 3: the force and torques of each pair that holds a
// contact, summed over its contacts in slot order (ascending node keys), eight
// lanes per pair.  The order is the contacts' own: slots without one, of which
// a cached list holds more, do not change the sum.
//
// Bound by the latency of pair, slots, node ids and forces, loads that wait for
// one another.  Three pairs in four hold no contact (a settled bed: 8 slots and
// a quarter of a contact per pair), so a warp takes several pairs' flags in one
// load, the next ones' meanwhile, and passes on to those that hold one; with
// eight lanes looking at each pair the sums took 105 us for 262,144 particles,
// this way 57 (cold caches; 28 to 38 in a run of steps).  A pair of bodies
// pressed into one another holds hundreds of contacts: their forces are loaded
// three at a time, the next slots' ids meanwhile, and a short list is shared out
// over all warps.  With a load per contact and 32 pairs a warp whatever their
// number, 40,000 pairs of such bodies took 2,660 us, this way 195.  Four or eight
// at a time take 150 and 127, but registers of the other warps: a settled bed
// of 262,144 then 40 and 48 us, not 38.
// ---------------------------------------------------------------------------
// the forces of the first COUNT contacts that m still names (bit u: slot u of
// the lane's group of eight; at: the place of the lane's own slot), in slot
// order: component l of each onto acc, the ninth onto lane 0's acc8.  For whole
// warps.
template <int COUNT, typename Real>
__device__ __forceinline__ void add_some(const double* rec, unsigned int& m, int at, int l, Real& acc, Real& acc8)
{
    Real v[COUNT], v8[COUNT];
    bool on[COUNT];
#pragma unroll
    for (int u = 0; u < COUNT; ++u) {
        on[u] = m != 0u;
        const int t = __shfl_sync(0xffffffffu, at, on[u] ? __ffs(m) - 1 : 0, 8);
        m &= m - 1u;
        const Real* f = reinterpret_cast<const Real*>(rec + (long long)CONTACT_REC * t);
        v[u] = on[u] ? f[l] : Real(0);
        v8[u] = on[u] && l == 0 ? f[8] : Real(0);
    }
#pragma unroll
    for (int u = 0; u < COUNT; ++u)
        if (on[u]) {
            acc += v[u];
            acc8 += v8[u];
        }
}
template <typename Real>
__device__ __forceinline__ void add_contacts(const double* rec, unsigned int m, int at, int l, Real& acc, Real& acc8)
{
    if (!__any_sync(0xffffffffu, __popc(m) > 1)) {
        add_some<1>(rec, m, at, l, acc, acc8);
        return;
    }
    while (__any_sync(0xffffffffu, m != 0u)) add_some<3>(rec, m, at, l, acc, acc8);
}

constexpr int SUM_TPB = 512;  // four such blocks fill an SM's warps

template <typename Real>
__device__ __forceinline__ void sum_list(const PairListDev& L, int kind, int block, int nblocks, bool link,
                                         const RevDev& R, int n_obj, int3* list)
{
    Real* pf = reinterpret_cast<Real*>(L.pf);
    const unsigned int full = 0xffffffffu;
    const int lane = threadIdx.x & 31, grp = lane >> 3, l = lane & 7;
    const int thread = block * blockDim.x + threadIdx.x, nthreads = nblocks * blockDim.x;
    const int npairs = min(*L.n_pairs, L.cap_pairs);
    if (link) {
        // a list that is built: each pair joins its partner's list of the
        // reverse index (only pairs with contact slots carry a force)
        const unsigned int build = *R.build;
        for (int p = thread; p < npairs; p += nthreads) {
            if (L.c_cnt[p] <= 0) continue;
            const int B = L.pairB[p];
            if (B < 0 || B >= n_obj) continue;
            const unsigned int code = (unsigned int)(p * 8 + kind);  // pair counts stay below 2^28
            const unsigned long long old = atomicExch(&R.head[B], ((unsigned long long)build << 32) | code);
            L.r_next[p] = (unsigned int)(old >> 32) == build ? (int)(unsigned int)old : -1;
        }
    }
    // a warp takes `take` pairs at a time: as many as it has lanes, or what
    // gives every warp its share of a short list, four for its four groups at
    // least
    const int warp = thread >> 5, nwarps = nthreads >> 5;
    const int take = min(max((npairs + 4 * nwarps - 1) / (4 * nwarps) * 4, 4), 32);
    auto flag = [&](int p0) { return lane < take && p0 + lane < npairs && L.p_hit[p0 + lane] != 0; };
    bool next = flag(warp * take);
    for (int p0 = warp * take; p0 < npairs; p0 += nwarps * take) {
        const bool hit = next;
        const unsigned int m = __ballot_sync(full, hit);
        const int p = p0 + lane;
        if (hit) list[__popc(m & ((1u << lane) - 1u))] = make_int3(p, L.c_off[p], L.c_cnt[p]);
        const int count = __popc(m);
        next = flag(p0 + nwarps * take);  // the next pairs' flags, meanwhile
        __syncwarp();
        for (int i0 = 0; i0 < count; i0 += 4) {
            const bool on = i0 + grp < count;
            const int3 q = on ? list[i0 + grp] : make_int3(0, 0, 0);
            const int o = q.y, c = q.z;
            Real acc = 0, acc8 = 0;
            // eight slots at a time: lane l looks at slot l of the next ones
            // while the forces of these are added
            const int cmax = __reduce_max_sync(full, c);
            int at = l < c ? L.c_at[o + l] : 0;
            int node = l < c ? L.c_node[o + l] : -1;
            for (int j0 = 0; j0 < cmax; j0 += 8) {
                const unsigned int any = __ballot_sync(full, node >= 0);
                const int here = at, j = j0 + 8 + l;
                at = j < c ? L.c_at[o + j] : 0;
                node = j < c ? L.c_node[o + j] : -1;
                if (any) add_contacts(L.c_rec, (any >> (8 * grp)) & 0xffu, here, l, acc, acc8);
            }
            if (on) {
                Real* out = pf + (long long)RESULT * q.x;
                out[l / 3 * 4 + l % 3] = acc;
                if (l == 0) out[10] = acc8;
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Mixed precision (FUNDEM_FP32_MIXED).  The node predicate, the SDF
// gradient, the contact law, the bond law and the force sums run in single
// precision with single-precision accumulation; positions, orientations and
// their integration, and the tangential-spring history, stay in double
// precision.  Node positions are formed relative to the body centres, so the
// single-precision quantities are millimetre-scale offsets, never absolute
// coordinates.
// ---------------------------------------------------------------------------
struct v3f {
    float x, y, z;
};
__device__ __forceinline__ v3f mkf(float x, float y, float z) { return v3f{x, y, z}; }
__device__ __forceinline__ v3f tof(double3 a) { return v3f{(float)a.x, (float)a.y, (float)a.z}; }
__device__ __forceinline__ double3 tod(v3f a) { return mk3((double)a.x, (double)a.y, (double)a.z); }
__device__ __forceinline__ v3f operator+(v3f a, v3f b) { return v3f{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ v3f operator-(v3f a, v3f b) { return v3f{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ v3f operator-(v3f a) { return v3f{-a.x, -a.y, -a.z}; }
__device__ __forceinline__ v3f operator*(float s, v3f a) { return v3f{s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ float dotf(v3f a, v3f b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }
__device__ __forceinline__ float lenf(v3f a) { return sqrtf(dotf(a, a)); }
__device__ __forceinline__ v3f crossf(v3f a, v3f b)
{
    return v3f{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
// R v and R^T v from the rotation rows
__device__ __forceinline__ v3f rowsf(float4 r0, float4 r1, float4 r2, v3f v)
{
    return v3f{fmaf(r0.x, v.x, fmaf(r0.y, v.y, r0.z * v.z)), fmaf(r1.x, v.x, fmaf(r1.y, v.y, r1.z * v.z)),
               fmaf(r2.x, v.x, fmaf(r2.y, v.y, r2.z * v.z))};
}
constexpr float PI_F = 3.14159265358979f;

// the linear contact law (contactKernel.cuh:4-77) in single precision, with
// the spring history accumulated in double precision
__device__ __forceinline__ v3f linear_contact32(double3& spring, v3f vc, v3f n, float delta, float dt, float kn,
                                                float ks, float mu, float res, float m)
{
    if (!(delta > 0.f)) {
        spring = mk3(0., 0., 0.);
        return mkf(0.f, 0.f, 0.f);
    }
    const float lr = logf(res);
    const float diss = -lr / sqrtf(lr * lr + PI_F * PI_F);
    const float cn = 2.f * diss * sqrtf(m * kn);
    const v3f vn = dotf(vc, n) * n;
    const v3f fn = (kn * delta) * n - cn * vn;
    const float cs = 2.f * diss * sqrtf(m * ks);
    const v3f vs = vc - vn;
    if (mu > 0.f && ks > 0.f) {
        // the history itself is kept in double precision: projection onto
        // the tangent plane, accumulation and the Coulomb rescaling
        const double3 nd = tod(n), vsd = tod(vs);
        double3 p1 = spring - dot3(spring, nd) * nd;
        const double ap1 = length3(p1);
        if (!fd_is_zero(ap1)) p1 = p1 * (length3(spring) / ap1);
        spring = p1 + (double)dt * vsd;
        const v3f sf = -ks * tof(spring) - cs * vs;
        const float asf = lenf(sf), afn = lenf(fn);
        if (asf > 1e-20f && asf > mu * afn) {
            const double scale = (double)(mu * afn) / (double)asf;
            const double3 sfd = -(double)ks * spring - (double)cs * vsd;
            spring = (-1.0 / (double)ks) * (scale * sfd + (double)cs * vsd);
        }
    } else {
        spring = mk3(0., 0., 0.);
    }
    return fn + (-ks * tof(spring) - cs * vs);
}

// explicit fused multiply-adds, as in the contact law: the predicate pass, the
// law pass, the image lists' and the small steps must give a node the same
// overlap
__device__ __forceinline__ float lerp32(float a, float b, float t) { return fmaf(a, 1.f - t, __fmul_rn(b, t)); }
__device__ __forceinline__ float trilinear32(const float* p, float x, float y, float z)
{
    return lerp32(lerp32(lerp32(p[0], p[1], x), lerp32(p[2], p[3], x), y),
                  lerp32(lerp32(p[4], p[5], x), lerp32(p[6], p[7], x), y), z);
}

// one slot's node against its partner, single-precision SDF
struct SlotEval32 {
    double3 cA, cB, rd, gp;  // centres, node offset from A's centre, node
    int pool;
    float ov, phi0, fx, fy, fz, pv[8];
};

// as slot_predicate
template <int KIND, bool FACES = false>
__device__ __forceinline__ bool slot_predicate32(const NarrowArgs& n, const PairState& st, int k, int3 bcell, float ov0,
                                                 SlotEval32& e)
{
    const FdGeo& GA = n.G.geo[st.gA];
    const double3 cA = st.xA;
    const double3 cB = st.xB;
    const GeoSetDev& SB = Slave<KIND>::set(n);
    const FdGeo& GB = SB.geo[st.gB];
    const FdGrid& sg = Slave<KIND>::grid(n);
    // the rigid transforms in double precision (as in FP64 mode), the
    // position inside the cell and the SDF interpolation in single
    e.cA = cA;
    e.cB = cB;
    e.pool = GA.node_off + k;
    e.rd = xm_rot(st.qA, n.G.nodes[e.pool]);
    const double3 gp = mk3(e.rd.x + cA.x, e.rd.y + cA.y, e.rd.z + cA.z);
    e.gp = gp;
    int3 lo, hi;
    fd_node_range(gp, sg, lo, hi);
    float fx = 0.f, fy = 0.f, fz = 0.f;
    float* pv = e.pv;
    bool hit = false;
    e.ov = ov0;
    e.phi0 = __int_as_float(0xff800000);  // the slot bound to store (-inf: never skipped)
    if (bcell.x >= lo.x && bcell.x <= hi.x && bcell.y >= lo.y && bcell.y <= hi.y && bcell.z >= lo.z && bcell.z <= hi.z) {
        const double3 rel = mk3(gp.x - cB.x, gp.y - cB.y, gp.z - cB.z);
        if (!Slave<KIND>::radius_test || xm_len2(rel) <= GB.radius * GB.radius) {
            const double3 lp = xm_rrot(rel, st.qB);
            const double gx = (lp.x - GB.origin.x) * GB.inv_spacing;
            const double gy = (lp.y - GB.origin.y) * GB.inv_spacing;
            const double gz = (lp.z - GB.origin.z) * GB.inv_spacing;
            const int i0 = (int)floor(gx), j0 = (int)floor(gy), k0 = (int)floor(gz);
            if (i0 >= 0 && j0 >= 0 && k0 >= 0 && i0 < GB.size.x - 1 && j0 < GB.size.y - 1 &&
                k0 < GB.size.z - 1) {
                fx = (float)(gx - (double)i0);
                fy = (float)(gy - (double)j0);
                fz = (float)(gz - (double)k0);
                const long long sx = GB.size.x, sxy = (long long)GB.size.x * GB.size.y;
                const long long c0 = GB.sdf_off + (long long)k0 * sxy + (long long)j0 * sx + i0;
                if (KIND == FD_PW) {
                    // wall grids are coarse (a plane wall is one cell
                    // the size of the domain, corner values of tenths
                    // of a metre): single-precision interpolation
                    // there would carry errors of 1e-8 m, so the
                    // (few) wall contacts interpolate in double
                    double4 s0, s1;
                    load_corners<FACES>(SB, c0, sx, sxy, s0, s1);
                    double pd[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
                    const double ovd = -xm_trilinear(gx - (double)i0, gy - (double)j0, gz - (double)k0, pd);
#pragma unroll
                    for (int c = 0; c < 8; ++c) pv[c] = (float)pd[c];
                    e.ov = (float)ovd;
                    e.phi0 = __double2float_rd(-ovd);
                    hit = ovd >= -n.a.probe;
                } else {
                    float4 s0, s1;
                    load_corners<FACES>(SB, c0, sx, sxy, s0, s1);
                    pv[0] = s0.x; pv[1] = s0.y; pv[2] = s0.z; pv[3] = s0.w;
                    pv[4] = s1.x; pv[5] = s1.y; pv[6] = s1.z; pv[7] = s1.w;
                    e.ov = -trilinear32(pv, fx, fy, fz);
                    e.phi0 = -e.ov;
                    hit = e.ov >= -(float)n.a.probe;
                }
            }
        }
    }
    e.fx = fx;
    e.fy = fy;
    e.fz = fz;
    return hit;
}

// as contact_law
template <int KIND>
__device__ __forceinline__ int contact_law32(const NarrowArgs& n, const PairListDev& L, const AdjRec& R, int s, int t, int A,
                                             int B, const PairState& st, int k, int oc_off, int oc_cnt,
                                             const SlotEval32& e, float o[9])
{
    const bool periodic = (KIND == FD_PP || KIND == FD_PW) && (n.a.periodic_x || n.a.periodic_y);
    const FdGeo& GA = n.G.geo[st.gA];
    const FdGeo& GB = Slave<KIND>::set(n).geo[st.gB];
    const float4* RB = Slave<KIND>::rot(n, B);
    const float4 b0 = RB[0], b1 = RB[1], b2 = RB[2];
    const double3 cA = e.cA, cB = e.cB, rd = e.rd, gp = e.gp;
    const v3f r = tof(rd);  // node offset from A's centre
    const float ov = e.ov, fy = e.fy, fz = e.fz;
    const float* pv = e.pv;
    const int pool = e.pool;
    // gradient with the x weight truncated as the reference does
    // (LSParticleContactDetectionKernel.cuh:34)
    const float wy0 = 1.f - fy, wy1 = fy, wz0 = 1.f - fz, wz1 = fz;
    const v3f gB =
        mkf(fmaf(__fmul_rn(pv[7] - pv[6], wy1), wz1,
                 fmaf(__fmul_rn(pv[5] - pv[4], wy0), wz1,
                      fmaf(__fmul_rn(pv[1] - pv[0], wy0), wz0, __fmul_rn(__fmul_rn(pv[3] - pv[2], wy1), wz0)))),
            fmaf(pv[2] - pv[0], wz0, __fmul_rn(pv[6] - pv[4], wz1)),
            fmaf(pv[4] - pv[0], wy0, __fmul_rn(pv[6] - pv[2], wy1)));
    v3f nrm = rowsf(b0, b1, b2, gB);
    const float l2 = dotf(nrm, nrm);
    nrm = l2 > 1e-20f ? rsqrtf(l2) * nrm : mkf(0.f, 0.f, 0.f);
    const v3f arm = r + (0.5f * ov) * nrm;  // contact point relative to A's centre
    const int nid = st.nodes + n.G.node_lid[pool];
    double3 spring = mk3(0., 0., 0.);
    int hist = -1;
    if (st.carried) {
        if (st.hnode == nid) hist = s;
        if (hist >= 0) {
            const double4 h = load_four(L.o_c_hist + st.hat);
            spring = mk3(h.x, h.y, h.z);
        }
    } else {
        const int oc_end = oc_off + oc_cnt;
        int lo2 = oc_off, hi2 = oc_end;
        if (s >= oc_off && s < oc_end && L.o_c_k[s] == k) lo2 = hi2 = s;
        while (lo2 < hi2) {
            const int mid = (lo2 + hi2) >> 1;
            if (L.o_c_k[mid] < k) lo2 = mid + 1; else hi2 = mid;
        }
        if (lo2 < oc_end && L.o_c_k[lo2] == k) {
            const int at = L.o_c_at[lo2];
            if (L.o_c_node[lo2] == nid) {
                const double4 h = load_four(L.o_c_hist + at);
                spring = mk3(h.x, h.y, h.z);
                hist = lo2;
            }
        }
    }
    if (R.hit && s < R.cap) {
        const fd_quat qB = st.qB;
        R.A[s] = A;
        R.B[s] = B;
        R.Bp[s] = KIND == FD_PW ? -1 : B;
        R.geoB[s] = KIND == FD_PW ? n.W.geo[B] : n.P.geo[B];
        R.matB[s] = KIND == FD_PW ? n.W.mat[B] : n.P.mat[B];
        R.nid[s] = nid;
        R.hist[s] = hist;
        R.rel[3 * s + 0] = gp.x - cB.x;
        R.rel[3 * s + 1] = gp.y - cB.y;
        R.rel[3 * s + 2] = gp.z - cB.z;
        R.sprev[3 * s + 0] = spring.x;
        R.sprev[3 * s + 1] = spring.y;
        R.sprev[3 * s + 2] = spring.z;
        R.qB[4 * s + 0] = qB.q0;
        R.qB[4 * s + 1] = qB.q1;
        R.qB[4 * s + 2] = qB.q2;
        R.qB[4 * s + 3] = qB.q3;
        R.arm[3 * s + 0] = rd.x;
        R.arm[3 * s + 1] = rd.y;
        R.arm[3 * s + 2] = rd.z;
        R.wrap[s] = 13 + 27;  // no shift unless the force side records one
    }
    const int mi = st.mA;
    float kn = 0.f, ks = 0.f;
    float mu, res, effM = 0.f;
    const double kni = n.M.kn[mi], ksi = n.M.ks[mi];
    const double invMi = GA.inv_mass;
    if (KIND == FD_PW) {
        const int mj = st.mB;
        mu = (float)fmin(n.M.mu[mi], n.MW.mu[mj]);
        res = (float)fmin(n.M.e[mi], n.MW.e[mj]);
        if (invMi > 0.) effM = (float)(1. / invMi);
        kn = (float)kni;
        ks = (float)ksi;
    } else {
        const int mj = st.mB;
        const double knj = n.M.kn[mj], ksj = n.M.ks[mj], invMj = GB.inv_mass;
        if (kni > 0. && knj > 0.) kn = (float)(kni * knj / (kni + knj));
        if (ksi > 0. && ksj > 0.) ks = (float)(ksi * ksj / (ksi + ksj));
        if (invMi > 0. || invMj > 0.) effM = (float)(1. / (invMi + invMj));
        res = (float)fmin(n.M.e[mi], n.M.e[mj]);
        mu = (float)fmin(n.M.mu[mi], n.M.mu[mj]);
    }
    if (n.with_force) {
        double3 ri = cA, rj = cB;
        if (periodic) {
            if (n.a.periodic_x) { ri = wrap_x(ri, n.pgrid); if (KIND == FD_PP) rj = wrap_x(rj, n.pgrid); }
            if (n.a.periodic_y) { ri = wrap_y(ri, n.pgrid); if (KIND == FD_PP) rj = wrap_y(rj, n.pgrid); }
        }
        double3 vid = st.vA, vjd = st.vB;
        if ((KIND == FD_PP || KIND == FD_PW) && n.a.sector) {
            sector_fold(ri, vid, n.pgrid.minb);
            if (KIND == FD_PP) sector_fold(rj, vjd, n.pgrid.minb);
        }
        const v3f armA = tof(cA - ri) + arm;
        const v3f armB = tof(cA - rj) + arm;
        const v3f vi = tof(vid), wi = tof(st.wA);
        const v3f vj = tof(vjd);
        const v3f wj = tof(st.wB);
        const v3f vc = (vi + crossf(wi, armA)) - (vj + crossf(wj, armB));
        if (R.hit && s < R.cap) {
            R.vc[3 * s + 0] = vc.x;
            R.vc[3 * s + 1] = vc.y;
            R.vc[3 * s + 2] = vc.z;
            R.wrap[s] = wrap_code(cA, ri, cB, rj, n.pgrid);
        }
        const v3f F = linear_contact32(spring, vc, nrm, ov, (float)n.a.dt, kn, ks, mu, res, effM);
        const v3f TA = crossf(armA, F);
        const v3f TB = crossf(armB, -F);
        o[0] = F.x; o[1] = F.y; o[2] = F.z;
        o[3] = TA.x; o[4] = TA.y; o[5] = TA.z;
        o[6] = TB.x; o[7] = TB.y; o[8] = TB.z;
    }
    L.c_at[s] = t;
    store_hist(L, t, spring, B);
    if (n.a.records) {
        store_record(L, t, mk3(cA.x + arm.x, cA.y + arm.y, cA.z + arm.z), mk3(nrm.x, nrm.y, nrm.z), ov,
                     0.5 * (double)ov * (double)ov * (double)kn, 0.5 * spring_sq(spring) * (double)ks);
    }
    return nid;
}

template <int KIND, int PASS>
__device__ __forceinline__ void contact_list32(const NarrowArgs& n, int block, int nblocks)
{
    const PairListDev& L = n.L;
    // pass 0: every slot; pass 1: the slots pass 0 listed as contacts
    const int nitems = PASS == 0 ? min(*L.n_slots, L.cap_contacts) : min(*L.n_hits, L.cap_contacts);
    const int lane = threadIdx.x & 31;
    const int stride = nblocks * blockDim.x;
    // pair cache, as in k_contact; the single-precision predicate's own
    // rounding (a few 1e-7 of the SDF values) is covered by a margin of
    // 1e-4 of B's grid spacing in the pair bound
    constexpr bool IMAGE = KIND != FD_PP && KIND != FD_PW;
    const bool cache = n.a.gate != nullptr;
    const bool carried = !list_built(n.a);
    const bool listed = KIND == FD_PP && PASS == 0 && carried;
    const bool slot_test = PASS == 0 && carried && !listed;
    const bool phi0_store = PASS == 0 && cache && !carried;
    const bool live_test = IMAGE && PASS == 0 && n.gh.live != nullptr;
    const int nitems_c = PASS == 0 && listed ? min(*L.n_test, L.cap_contacts) : nitems;
    int hits = 0;
    for (int s0 = block * blockDim.x + (threadIdx.x & ~31); s0 < nitems_c; s0 += stride) {
        const int t = s0 + lane;
        const int s = t < nitems_c ? (PASS == 1 ? L.c_hit[t] : listed ? L.c_test[t] : t) : t;
        bool hit = false;
        bool continue_slot = false;
        if ((slot_test || live_test) && t < nitems_c) {
            const int p = L.c_pair[s];
            if (live_test && !n.gh.live[L.pairB[p]]) {
                L.c_node[s] = -1;
                if (phi0_store) L.c_phi0[s] = __int_as_float(0xff800000);  // -inf: never skipped
                continue_slot = true;
            } else if (slot_test && L.c_phi0[s] > __fadd_ru(L.p_bound[p], 1e-12f)) {
                // pair_bound carries the margin of 1e-4 of B's grid spacing in
                // this precision
                L.c_node[s] = -1;
                continue_slot = true;
            }
        }
        if (t < nitems_c && !continue_slot) {
            const int p = L.c_pair[s];
            const int k = L.c_k[s];
            const int A = L.pairA[p];
            const int B = L.pairB[p];
            // a carried slot's history is its previous self, and its partner's
            // cell this step's
            PairState st = load_pair<KIND, PASS == 1>(n, A, B);
            if (PASS == 1 && carried) {
                st.carried = true;
                st.hnode = load_now(L.o_c_node + s);
                st.hat = load_now(L.o_c_at + s);
            }
            int4 aux = make_int4(0, 0, 0, s);
            int hist = 1;
            if (carried) {
                int3 bc;
                decode_cell(st.hB, Slave<KIND>::grid(n).size, bc);
                aux.x = bc.x; aux.y = bc.y; aux.z = bc.z;
            } else {
                aux = L.p_aux[p];
                hist = L.p_hist_cnt[p];
            }
            SlotEval32 e;
            // an overlap the predicate did not reach stays +inf (a slot that
            // is never skipped)
            hit = slot_predicate32<KIND>(n, st, k, make_int3(aux.x, aux.y, aux.z),
                                         PASS == 0 ? __int_as_float(0x7f800000) : 0.f, e);
            if (phi0_store) L.c_phi0[s] = e.phi0;
            int nid = -1;
            if (PASS == 1 && hit) {
                float o[9];
                nid = contact_law32<KIND>(n, L, n.a.rec, s, t, A, B, st, k, aux.w, hist, e, o);
                if (n.with_force) store_force(L, t, o);
            }
            if (PASS == 1) {
                L.c_node[s] = nid;
            } else {
                if (hit) L.p_hit[p] = 1;
                else L.c_node[s] = -1;
                if (n.a.rec.hit && s < n.a.rec.cap) n.a.rec.hit[s] = hit ? 1 : 0;
            }
        }
        if (PASS == 0) {
            // contacts are listed for pass 1, one atomic per warp
            const unsigned int m = __ballot_sync(0xffffffffu, hit);
            if (m) {
                int base = 0;
                if (lane == 0) base = atomicAdd(L.n_hits, __popc(m));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (hit) L.c_hit[base + __popc(m & ((1u << lane) - 1u))] = s;
                hits += __popc(m);
            }
        }
    }
    if (PASS == 0 && n.a.stats && lane == 0 && hits) atomicAdd(&n.a.stats[3], (unsigned long long)hits);
}

// The two contact passes of every list, bound by the waits of their gathers
// (16-22 stalls for a load per issue).  262,144 bodies on a carried step, 2.4
// million slots tested, 340,000 contacts: predicate 106 us (111 with 8-byte
// loads of the corners), law 80 us (126 with a result per slot and each load
// at its use).
template <bool MIXED, int PASS>
__global__ void __launch_bounds__(TPB, PASS == 0 ? FD_PROBE_MIN_BLOCKS : FD_CONTACT_MIN_BLOCKS) k_contact_lists(ListSet a)
{
    int block, nblocks;
    const int li = list_of(a, block, nblocks);
    const NarrowArgs& n = a.l[li];
    if (MIXED) {
        if (a.kind[li] == FD_PP) contact_list32<FD_PP, PASS>(n, block, nblocks);
        else if (a.kind[li] == FD_PW) contact_list32<FD_PW, PASS>(n, block, nblocks);
        else contact_list32<FD_GX, PASS>(n, block, nblocks);
    } else {
        if (a.kind[li] == FD_PP) contact_list<FD_PP, PASS>(n, block, nblocks);
        else if (a.kind[li] == FD_PW) contact_list<FD_PW, PASS>(n, block, nblocks);
        else contact_list<FD_GX, PASS>(n, block, nblocks);
    }
}

// ---------------------------------------------------------------------------
// reverse index: pairs grouped by partner B, sorted by A
// ---------------------------------------------------------------------------
// (with the image lists): every pair with contact slots joins the list of its
// partner in the pair sums (heads tagged with the step's build number, as the
// cell table's, so nothing is cleared), and at the step's end each particle
// walks its list into a segment of codes and sorts it.  Counting, scanning,
// filling and sorting were seven launches.
static_assert(FD_NKIND <= 8, "a reverse-index code keeps the kind in 3 bits");

// the index is built: always (gate null), or on the steps that build a list
__device__ __forceinline__ bool rev_built(const RevDev& R)
{
    return R.gate == nullptr || *R.gate != 0 || (R.gate2 && *R.gate2 != 0);
}

template <typename Real>
__global__ void __launch_bounds__(SUM_TPB, FD_SUM_MIN_BLOCKS) k_sum_lists(ListSet a, RevDev R)
{
    int block, nblocks;
    const int li = list_of(a, block, nblocks);
    const NarrowArgs& n = a.l[li];
    __shared__ int3 s_list[SUM_TPB / 32][32];
    sum_list<Real>(n.L, a.kind[li], block, nblocks, a.kind[li] != FD_PW && rev_built(R), R, n.P.n,
                   s_list[threadIdx.x >> 5]);
}

// End of a step.  The reverse index, where a list was built; under the pair
// cache the layout of each list that was built goes to the other generation
// too (a carried step then finds it in place), the bodies' state becomes the
// new reference, and the last block renews the flags: a list that overflowed
// asks for a rebuild, this step's requests become the next step's.
// the bodies' state as the pair cache's reference
__device__ __forceinline__ void cache_refs(const PairCacheDev& pc, const ObjDev& P, const ObjDev& W, int i0, int stride)
{
    for (int i = i0; i < P.n; i += stride) {
        pc.ref_pos[i] = P.pos[i];
        pc.ref_q[i] = P.q[i];
        pc.ref_vis[i] = P.hash[i] >= 0;
    }
    for (int w = i0; w < W.n; w += stride) {
        pc.wref_pos[w] = W.pos[w];
        pc.wref_q[w] = W.q[w];
        pc.wref_hash[w] = W.hash[w];
    }
}
// where the wraps that follow the detection of particles and walls move bodies
// in place, the references are taken before them: a body moved since its pairs
// were listed has drifted
__global__ void __launch_bounds__(TPB) k_cache_refs(PairCacheDev pc, ObjDev P, ObjDev W)
{
    if (pc.ctrl[0] != 0) cache_refs(pc, P, W, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

struct EndArgs {
    ObjDev P, W;
    PairListDev L[FD_NKIND];  // by kind
    int active[FD_NKIND];
    RevDev R;
    PairCacheDev pc;
    int cached;               // the pair cache is on; ghosts: so are the translated image lists
    int cached_ghosts;
    int refs;                 // the bodies' state is the reference of a build (see k_cache_refs)
    unsigned int* done;       // blocks finished (returns to 0)
    unsigned int* flags;
};
__global__ void __launch_bounds__(TPB) k_step_end(EndArgs a)
{
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (rev_built(a.R)) {
        const unsigned int build = *a.R.build;
        for (int i = i0; i < a.P.n; i += stride) {
            const unsigned long long h = a.R.head[i];
            int cnt = 0;
            if ((unsigned int)(h >> 32) == build)
                for (int code = (int)(unsigned int)h; code >= 0 && cnt <= a.R.cap; code = a.L[code & 7].r_next[code >> 3])
                    ++cnt;
            if (cnt > a.R.cap) {  // more links than the lists have pairs: not a list
                set_flag(a.flags, FD_FLAG_INDEX);
                cnt = 0;
            }
            const int o = cnt ? atomicAdd(a.R.total, cnt) : 0;
            cnt = min(cnt, a.R.cap - o);
            a.R.off[i] = o;
            a.R.cnt[i] = cnt;
            // by owner, then kind (an owner has one pair per kind with a given
            // partner)
            int* seg = a.R.code + o;
            auto key = [&](int code) { return (long long)a.L[code & 7].pairA[code >> 3] * 8 + (code & 7); };
            int code = (int)(unsigned int)h;
            for (int n = 0; n < cnt; ++n) {
                const long long kv = key(code);
                int b = n - 1;
                while (b >= 0 && key(seg[b]) > kv) { seg[b + 1] = seg[b]; --b; }
                seg[b + 1] = code;
                code = a.L[code & 7].r_next[code >> 3];
            }
        }
    }
    if (!a.cached) return;
    const bool built = a.pc.ctrl[0] != 0, ghosts_built = built || a.pc.ctrl[4] != 0;
    for (int k = 0; k < FD_NKIND; ++k) {
        if (!a.active[k] || !(k <= FD_PW ? built : ghosts_built && a.cached_ghosts)) continue;
        const PairListDev& L = a.L[k];
        const int np = min(*L.n_pairs, L.cap_pairs), ns = min(*L.n_slots, L.cap_contacts);
        if (i0 == 0) {
            L.o_counters[0] = *L.n_pairs;
            L.o_counters[1] = *L.n_slots;
        }
        for (int i = i0; i < a.P.n; i += stride) {
            L.o_seg_off[i] = L.seg_off[i];
            L.o_seg_cnt[i] = L.seg_cnt[i];
        }
        for (int p = i0; p < np; p += stride) {
            L.o_pairA[p] = L.pairA[p];
            L.o_pairB[p] = L.pairB[p];
            L.o_c_off[p] = L.c_off[p];
            L.o_c_cnt[p] = L.c_cnt[p];
        }
        for (int s = i0; s < ns; s += stride) L.o_c_k[s] = L.c_k[s];
    }
    if (built && a.refs) cache_refs(a.pc, a.P, a.W, i0, stride);
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicInc(a.done, gridDim.x - 1) != gridDim.x - 1) return;
    // the last block: every other one has read the flags
    int* ctrl = a.pc.ctrl;
    auto overflowed = [&](int k) {
        return *a.L[k].n_pairs > a.L[k].cap_pairs || *a.L[k].n_slots > a.L[k].cap_contacts;
    };
    if (built) {
        ctrl[1] += 1;
        // a build whose pairs or slots did not fit is not kept: the next step
        // builds again (the host grows the lists at its next check)
        ctrl[2] = overflowed(FD_PP) ? 1 : 0;
    }
    int request = ctrl[7];
    for (int k = FD_PW; k < FD_NKIND; ++k)
        if (a.active[k] && (k == FD_PW || a.cached_ghosts) && overflowed(k)) request = 1;
    ctrl[3] = request;
    ctrl[7] = 0;
    ctrl[0] = 0;
    ctrl[4] = 0;
}

__device__ __forceinline__ double4 load_vec(const double* p) { return load_four(reinterpret_cast<const double4*>(p)); }
__device__ __forceinline__ float4 load_vec(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void store_vec(double* p, double x, double y, double z)
{
    reinterpret_cast<double2*>(p)[0] = make_double2(x, y);
    reinterpret_cast<double2*>(p)[1] = make_double2(z, 0.);
}
__device__ __forceinline__ void store_vec(float* p, float x, float y, float z)
{
    *reinterpret_cast<float4*>(p) = make_float4(x, y, z, 0.f);
}
// a bond's eight frame vectors, 192 bytes in six loads: with 24 loads at a
// stride of 192 bytes (and six orientations' and nine results' worth more) the
// bond kernels spent their time in the L1
__device__ __forceinline__ void load_frames(const double3* p, double3 (&f)[8])
{
    const double4* q = reinterpret_cast<const double4*>(p);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const double4 a = load_quad(q + 3 * h), b = load_quad(q + 3 * h + 1), c = load_quad(q + 3 * h + 2);
        f[4 * h] = make_double3(a.x, a.y, a.z);
        f[4 * h + 1] = make_double3(a.w, b.x, b.y);
        f[4 * h + 2] = make_double3(b.z, b.w, c.x);
        f[4 * h + 3] = make_double3(c.y, c.z, c.w);
    }
}

// ---------------------------------------------------------------------------
// bonds, contactKernel.cuh:138-199 and contactKernel.cu:293-371
// ---------------------------------------------------------------------------
__global__ void k_bonds(ObjDev P, BondDev Bd)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Bd.n) return;
    double2* E2 = reinterpret_cast<double2*>(Bd.energy + 6ll * k);
    double* O = reinterpret_cast<double*>(Bd.out) + (long long)RESULT * k;
    if (Bd.rec_active) Bd.rec_active[k] = Bd.active[k] != 0;
    if (Bd.active[k] == 0) {
        for (int t = 0; t < 3; ++t) E2[t] = make_double2(0., 0.);
        for (int t = 0; t < 3; ++t) store_vec(O + 4 * t, 0, 0, 0);
        return;
    }
    const int i = Bd.master[k], j = Bd.slave[k];
    const fd_quat qi = load_q(P.q + i), qj = load_q(P.q + j);
    double3 f[8];
    load_frames(Bd.frames + 8ll * k, f);
    const double3 n1i = fd_rot(qi, f[0]), n2i = fd_rot(qi, f[1]), n3i = fd_rot(qi, f[2]);
    const double3 n1j = fd_rot(qj, f[4]), n2j = fd_rot(qj, f[5]), n3j = fd_rot(qj, f[6]);
    const double3 ri = P.pos[i], rj = P.pos[j];
    const double3 rbi = fd_rot(qi, f[3]) + ri;
    const double3 rbj = fd_rot(qj, f[7]) + rj;
    Bd.point[k] = 0.5 * (rbi + rbj);
    double3 F = mk3(0., 0., 0.), Mij = mk3(0., 0., 0.), Mji = mk3(0., 0., 0.);
    int act = 1;
    const double3 rij = rbi - rbj;
    if (Bd.rec_rij) {
        Bd.rec_rij[3 * k + 0] = rij.x;
        Bd.rec_rij[3 * k + 1] = rij.y;
        Bd.rec_rij[3 * k + 2] = rij.z;
        Bd.rec_dn[3 * k + 0] = n1j.x - n1i.x;
        Bd.rec_dn[3 * k + 1] = n1j.y - n1i.y;
        Bd.rec_dn[3 * k + 2] = n1j.z - n1i.z;
    }
    const double D = length3(rij);
    if (!fd_is_zero(D)) {
        const double4 b = load_vec(Bd.B + 4ll * k);
        const double B1 = b.x, B2 = b.y, B3 = b.z, B4 = b.w;
        double E[6];
        const double R = Bd.radius[k], D0 = Bd.L0[k];
        const double3 nij = fd_normalize(rij);
        const double3 e = -nij;
        E[0] = 0.5 * B1 * (D - D0) * (D - D0);
        E[1] = B2 * (0.5 * dot3(n1j - n1i, e) - 0.25 * dot3(n1i, n1j) + 0.75);
        E[2] = (0.25 * B2 + B3 + 0.5 * B4) * (dot3(n1i, n1j) + 1.);
        E[3] = -0.5 * B4 * (dot3(n1i, n1j) + dot3(n2i, n2j) + dot3(n3i, n3j) - 1);
        const double3 dn = n1j - n1i;
        F = B1 * (D - D0) * e + B2 / (2 * D) * (dn - dot3(dn, e) * e);
        const double3 MTB = B3 * cross3(n1j, n1i) - 0.5 * B4 * (cross3(n2j, n2i) + cross3(n3j, n3i));
        Mij = -0.5 * B2 * cross3(e, n1i) + MTB;
        Mji = 0.5 * B2 * cross3(e, n1j) - MTB;
        const double bnf = dot3(F, nij);
        const double3 bsf = F - bnf * nij;
        const double btt = dot3(MTB, nij);
        const double3 bbt = MTB - btt * nij;
        const double Ab = R * R * PI_D;
        const double Ib = Ab * R * R / 4.;
        const double Jb = 2 * Ib;
        E[4] = -bnf / Ab + length3(bbt) / Ib * R;
        E[5] = length3(bsf) / Ab + fabs(btt) / Jb * R;
        if (Bd.ts[k] > 0. && E[4] > Bd.ts[k]) act = 0;
        else if (Bd.coh[k] > 0. && E[5] > Bd.coh[k] - Bd.mu[k] * E[4]) act = 0;
        for (int t = 0; t < 3; ++t) E2[t] = make_double2(E[2 * t], E[2 * t + 1]);
    }
    Bd.active[k] = act;
    const double3 Ti = Mij + cross3(rbi - ri, F);
    const double3 Tj = Mji + cross3(rbj - rj, -F);
    store_vec(O, F.x, F.y, F.z);
    store_vec(O + 4, Ti.x, Ti.y, Ti.z);
    store_vec(O + 8, Tj.x, Tj.y, Tj.z);
}

// the V-bond (contactKernel.cuh:138-199) in single precision; the frames are
// rotated with the single-precision rotation rows, the bond vector is formed
// from the double-precision centre difference plus the rotated offsets
__global__ void k_bonds32(ObjDev P, BondDev Bd)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Bd.n) return;
    double2* E2 = reinterpret_cast<double2*>(Bd.energy + 6ll * k);
    float* O = reinterpret_cast<float*>(Bd.out) + (long long)RESULT * k;
    if (Bd.rec_active) Bd.rec_active[k] = Bd.active[k] != 0;
    if (Bd.active[k] == 0) {
        for (int t = 0; t < 3; ++t) E2[t] = make_double2(0., 0.);
        for (int t = 0; t < 3; ++t) store_vec(O + 4 * t, 0, 0, 0);
        return;
    }
    const int i = Bd.master[k], j = Bd.slave[k];
    const float4 a0 = P.rot[3ll * i], a1 = P.rot[3ll * i + 1], a2 = P.rot[3ll * i + 2];
    const float4 b0 = P.rot[3ll * j], b1 = P.rot[3ll * j + 1], b2 = P.rot[3ll * j + 2];
    double3 f[8];
    load_frames(Bd.frames + 8ll * k, f);
    const v3f n1i = rowsf(a0, a1, a2, tof(f[0])), n2i = rowsf(a0, a1, a2, tof(f[1])), n3i = rowsf(a0, a1, a2, tof(f[2]));
    const v3f n1j = rowsf(b0, b1, b2, tof(f[4])), n2j = rowsf(b0, b1, b2, tof(f[5])), n3j = rowsf(b0, b1, b2, tof(f[6]));
    const double3 ri = P.pos[i], rj = P.pos[j];
    const v3f oi = rowsf(a0, a1, a2, tof(f[3])), oj = rowsf(b0, b1, b2, tof(f[7]));
    Bd.point[k] = 0.5 * (ri + rj) + 0.5 * tod(oi + oj);
    v3f F = mkf(0.f, 0.f, 0.f), Mij = mkf(0.f, 0.f, 0.f), Mji = mkf(0.f, 0.f, 0.f);
    int act = 1;
    const v3f rij = tof(ri - rj) + (oi - oj);
    if (Bd.rec_rij) {
        Bd.rec_rij[3 * k + 0] = rij.x;
        Bd.rec_rij[3 * k + 1] = rij.y;
        Bd.rec_rij[3 * k + 2] = rij.z;
        Bd.rec_dn[3 * k + 0] = n1j.x - n1i.x;
        Bd.rec_dn[3 * k + 1] = n1j.y - n1i.y;
        Bd.rec_dn[3 * k + 2] = n1j.z - n1i.z;
    }
    const float D = lenf(rij);
    if (D > 1e-20f) {
        const double4 b = load_vec(Bd.B + 4ll * k);
        const float B1 = (float)b.x, B2 = (float)b.y, B3 = (float)b.z, B4 = (float)b.w;
        double E[6];
        const float R = (float)Bd.radius[k], D0 = (float)Bd.L0[k];
        const v3f nij = rsqrtf(dotf(rij, rij)) * rij;
        const v3f e = -nij;
        const float c11 = dotf(n1i, n1j);
        E[0] = 0.5 * (double)B1 * (double)(D - D0) * (double)(D - D0);
        E[1] = (double)(B2 * (0.5f * dotf(n1j - n1i, e) - 0.25f * c11 + 0.75f));
        E[2] = (double)((0.25f * B2 + B3 + 0.5f * B4) * (c11 + 1.f));
        E[3] = (double)(-0.5f * B4 * (c11 + dotf(n2i, n2j) + dotf(n3i, n3j) - 1.f));
        const v3f dn = n1j - n1i;
        F = (B1 * (D - D0)) * e + (B2 / (2.f * D)) * (dn - dotf(dn, e) * e);
        const v3f MTB = B3 * crossf(n1j, n1i) - (0.5f * B4) * (crossf(n2j, n2i) + crossf(n3j, n3i));
        Mij = (-0.5f * B2) * crossf(e, n1i) + MTB;
        Mji = (0.5f * B2) * crossf(e, n1j) - MTB;
        const float bnf = dotf(F, nij);
        const v3f bsf = F - bnf * nij;
        const float btt = dotf(MTB, nij);
        const v3f bbt = MTB - btt * nij;
        const float Ab = R * R * PI_F;
        const float Ib = Ab * R * R / 4.f;
        const float Jb = 2.f * Ib;
        const float sn = -bnf / Ab + lenf(bbt) / Ib * R;
        const float ss = lenf(bsf) / Ab + fabsf(btt) / Jb * R;
        E[4] = sn;
        E[5] = ss;
        if (Bd.ts[k] > 0. && sn > (float)Bd.ts[k]) act = 0;
        else if (Bd.coh[k] > 0. && ss > (float)(Bd.coh[k] - Bd.mu[k] * (double)sn)) act = 0;
        for (int t = 0; t < 3; ++t) E2[t] = make_double2(E[2 * t], E[2 * t + 1]);
    }
    Bd.active[k] = act;
    const v3f Ti = Mij + crossf(oi, F);
    const v3f Tj = Mji + crossf(oj, -F);
    store_vec(O, F.x, F.y, F.z);
    store_vec(O + 4, Ti.x, Ti.y, Ti.z);
    store_vec(O + 8, Tj.x, Tj.y, Tj.z);
}

// ---------------------------------------------------------------------------
// per-particle reduction, fixed order
// ---------------------------------------------------------------------------
struct ReduceArgs {
    ObjDev P;
    PairListDev L[FD_NKIND];
    int active[FD_NKIND];
    RevDev R;
    BondDev B;
};

// Real = double: FP64 mode; Real = float: mixed mode (pair and bond results
// stored and summed in single precision)
template <typename Real> struct ForceSum {
    Real F[3] = {0, 0, 0}, T[3] = {0, 0, 0};
    // one pair or bond result, as the body's own (F, torque) or as the partner's
    // (k: its number; torque 1: on A, 2: on B)
    __device__ __forceinline__ void add(const Real* results, long long k, Real sgn, int torque)
    {
        const Real* r = results + RESULT * k;
        const auto f = load_vec(r), t = load_vec(r + 4 * torque);
        F[0] += sgn * f.x;
        F[1] += sgn * f.y;
        F[2] += sgn * f.z;
        T[0] += t.x;
        T[1] += t.y;
        T[2] += t.z;
    }
    // the pairs the particle owns in one list (s: first, c: count; no contact,
    // no sum kept), four hit flags loaded ahead
    __device__ __forceinline__ void own(const PairListDev& L, int s, int c)
    {
        for (int k = s; k < s + c; k += 4) {
            int h[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) h[u] = k + u < s + c ? L.p_hit[k + u] : 0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (h[u]) add(reinterpret_cast<const Real*>(L.pf), k + u, Real(1), 1);
        }
    }
    __device__ __forceinline__ void bonds(const BondDev& B, int i)
    {
        const Real* out = reinterpret_cast<const Real*>(B.out);
        for (int e = B.plist_off[i]; e < B.plist_off[i + 1]; ++e) {
            const int code = B.plist[e];
            if ((code & 1) == 0) add(out, code >> 1, Real(1), 1);
            else add(out, code >> 1, Real(-1), 2);
        }
    }
};

// What surrounds a step's detection: the force sums of one step (SUM), its
// second half kick (BACK), and the next step's first half kick, drift, hash
// and pair-cache check, walls too (FRONT).  Between two steps all of it is one
// pass over the bodies; the sums, the copy of the wrapped positions, two
// kicks, two drifts, two hashes and two checks were a launch each.  Bound by
// the waits of range, flag and result, a thread a body; 262,144 bodies take
// 54 us (162 MB from and to memory: 25 us at the measured copy rate), 72 with
// the results as single numbers and no load ahead.
struct AdvanceArgs {
    ObjDev P, W;
    GeoSetDev G, GW;
    FdGrid pgrid, wgrid;
    ReduceArgs r;             // SUM
    const double3* wrapped;   // the positions after the periodic wraps (null: P.pos)
    double3 gravity;
    double h, dt;
    unsigned int* build;      // FRONT: the cell table's build numbers, renewed for
    int par;                  // a step of this list generation
    PairCacheDev pc;
    int cached;
    int* occ[6];              // occupied-cell boxes of the image tables, reset
};
template <typename Real, bool SUM, bool BACK, bool FRONT>
__global__ void __launch_bounds__(128) k_advance(AdvanceArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (FRONT && i < 36 && a.occ[i / 6]) a.occ[i / 6][i % 6] = i % 6 < 3 ? 0x7f7f7f7f : -1;
    if (FRONT && i == 0) bump_build(a.build, a.par);
    if (i < a.P.n) {
        double3 F, T;
        if (SUM) {
            const ReduceArgs& r = a.r;
            ForceSum<Real> f;
            // pairs the particle owns, kind by kind, then those in which it is
            // the partner, by owner.  Ranges, codes, flags and sums are loads
            // that wait for one another: those of all kinds, and of four
            // codes, are under way together
            int so[FD_NKIND], sc[FD_NKIND];
#pragma unroll
            for (int kind = 0; kind < FD_NKIND; ++kind) {
                so[kind] = r.active[kind] ? r.L[kind].seg_off[i] : 0;
                sc[kind] = r.active[kind] ? r.L[kind].seg_cnt[i] : 0;
            }
            const int rs = r.R.off[i], re = rs + min(r.R.cnt[i], r.R.cap - rs);
#pragma unroll
            for (int kind = 0; kind < FD_NKIND; ++kind) f.own(r.L[kind], so[kind], sc[kind]);
            for (int e = rs; e < re; e += 4) {
                int code[4], h[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) code[u] = e + u < re ? r.R.code[e + u] : -1;
#pragma unroll
                for (int u = 0; u < 4; ++u) h[u] = code[u] >= 0 ? r.L[code[u] & 7].p_hit[code[u] >> 3] : 0;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (!h[u]) continue;
                    const int kind = code[u] & 7, k = code[u] >> 3;
                    const PairListDev& L = r.L[kind];
                    if (kind != FD_PP && L.pairA[k] == i) continue;  // a particle against its own ghost
                    f.add(reinterpret_cast<const Real*>(L.pf), k, Real(-1), 2);
                }
            }
            if (r.B.n > 0) f.bonds(r.B, i);
            F = mk3((double)f.F[0], (double)f.F[1], (double)f.F[2]);
            T = mk3((double)f.T[0], (double)f.T[1], (double)f.T[2]);
            a.P.force[i] = F;
            a.P.torque[i] = T;
            if (!FRONT && a.wrapped) a.P.pos[i] = a.wrapped[i];
        } else {
            F = a.P.force[i];
            T = a.P.torque[i];
        }
        if (!BACK && !FRONT) return;
        Body b;
        b.v = a.P.vel[i];
        b.w = a.P.angvel[i];
        b.q = a.P.q[i];
        const FdGeo& geo = a.G.geo[a.P.geo[i]];
        if (BACK) kick_body(b, geo, F, T, a.gravity, a.h);
        if (FRONT) {
            b.x = SUM && a.wrapped ? a.wrapped[i] : a.P.pos[i];
            kick_body(b, geo, F, T, a.gravity, a.h);
            drift_body(b, a.dt);
            a.P.pos[i] = b.x;
            a.P.q[i] = b.q;
            const long long hash = hash_one(a.P, a.pgrid, i, b.x, b.q);
            if (a.cached) cache_check(a.pc, i, b.x, b.q, hash >= 0);
        }
        a.P.vel[i] = b.v;
        a.P.angvel[i] = b.w;
    } else if (FRONT && i - a.P.n < a.W.n) {
        const int w = i - a.P.n;
        Body b{a.W.pos[w], a.W.vel[w], a.W.angvel[w], a.W.q[w]};
        drift_body(b, a.dt);
        a.W.pos[w] = b.x;
        a.W.q[w] = b.q;
        const long long hash = hash_one(a.W, a.wgrid, w, b.x, b.q);
        if (a.cached) cache_check_wall(a.pc, w, b.x, b.q, hash, a.GW.geo[a.W.geo[w]].grid_radius);
    }
}

// ---------------------------------------------------------------------------
// Small sets (no neighbour list, no pair cache, no images).  A step of the
// staged kernels is a dozen dependent launches, each a few microseconds of
// latency and next to no work at these sizes: 73 us a step for 1,000 particles
// in a graph replay.  Here a step is two launches.  k_small_pairs takes each
// particle's partners and walls from the cell lists, culls each candidate pair
// in one warp, takes the block's slots through predicate and contact law one
// thread each, and sums its pairs with eight lanes each; k_small_advance sums
// each particle's pairs and runs the half kicks, the drift, the hash and the
// cell lists of the next step.  The sums run in the staged kernels' order, so
// the results are theirs.  A block's few slots leave most of its threads idle
// in the contact law, so large sets stay with the staged kernels.
//
// Bound by the chain of one block: about 9,400 cycles of search, 13,000 of
// culling (two pairs a warp), 8,000 of predicate and law, 4,000 of sums.  A
// step of 1,000 particles takes 38 us (50 with a pair's slots in its own warp),
// of 4,096 65 us (81).  Where the staged kernels take over: SMALL_PARTICLES.
// ---------------------------------------------------------------------------
constexpr int SMALL_BODIES = 4;               // particles per block
constexpr int SMALL_WARPS = 2 * SMALL_BODIES;  // a warp for each one's partners, one for its walls
constexpr int SMALL_TASKS = SMALL_BODIES * MAX_CAND;  // pairs of a block, per kind
constexpr int MAX_FOUND = 512;                // objects of the cells around a particle, staged for the test

struct SmallArgs {
    NarrowArgs n;          // n.L, n.a.rec: the particle-particle list
    PairListDev Lw;        // the particle-wall list
    AdjRec recw;
    CellTableDev T;
    const int2* wall_range;
    int* r_head;           // per particle: the last pair with a contact it is the partner of
    void* own;             // per particle: force and torque of its own pairs (6 Real)
};

// one pair of list L, one warp: its slots, written to L.c_k.  Returns the first
// slot, their count, and the slots of the pair's history.
template <int KIND, int NODES>
__device__ __forceinline__ int4 small_slots(const NarrowArgs& n, const PairListDev& L, int p, int A, int B, int lane,
                                            unsigned short* queue, unsigned long long* stats)
{
    int kept;
    int ncand = cull_pair<KIND, NODES, true>(n, A, B, 0.0, lane, queue, kept);
    if (n.a.stats && lane == 0) {
        atomicAdd(&stats[0], 1ull);
        atomicAdd(&stats[1], (unsigned long long)min(n.G.geo[n.P.geo[A]].clus_count, MAX_CLUSTERS));
        atomicAdd(&stats[2], (unsigned long long)kept);
        atomicAdd(&stats[4], (unsigned long long)ncand);
    }
    int4 slot = make_int4(0, 0, 0, 0);
    if (ncand > 0) {
        if (lane == 0) slot.x = atomicAdd(L.n_slots, ncand);
        find_history(L, A, B, lane, slot.z, slot.w);
        slot.x = __shfl_sync(0xffffffffu, slot.x, 0);
        slot.y = ncand;
        if (slot.x + ncand > L.cap_contacts) {
            if (lane == 0) set_flag(n.a.flags, FD_FLAG_CONTACT_OVERFLOW);
            slot.x = slot.y = 0;
        }
    }
    if (lane == 0) {
        L.c_off[p] = slot.x;
        L.c_cnt[p] = slot.y;
    }
    for (int i = lane; i < slot.y; i += 32) L.c_k[slot.x + i] = queue[i];
    return slot;
}

// one slot of pair (A, B) of list L: predicate and contact law; true for a contact
template <int KIND, bool MIXED>
__device__ __forceinline__ bool small_contact(const NarrowArgs& n, const PairListDev& L, const AdjRec& R, int A, int B,
                                              int s, int oc_off, int oc_cnt)
{
    using Real = typename std::conditional<MIXED, float, double>::type;
    const int k = load_now(L.c_k + s);
    const PairState st = load_pair<KIND, true>(n, A, B);
    int3 bcell;
    decode_cell(st.hB, Slave<KIND>::grid(n).size, bcell);
    int nid = -1;
    bool hit;
    Real o[9];
    if constexpr (MIXED) {
        SlotEval32 e;
        hit = slot_predicate32<KIND, true>(n, st, k, bcell, 0.f, e);
        if (hit) nid = contact_law32<KIND>(n, L, R, s, s, A, B, st, k, oc_off, oc_cnt, e, o);
    } else {
        SlotEval e;
        hit = slot_predicate<KIND, true>(n, st, k, bcell, 0., e);
        if (hit) nid = contact_law<KIND>(n, L, R, s, s, A, B, st, k, oc_off, oc_cnt, e, o);
    }
    if (hit) store_force(L, s, o);
    L.c_node[s] = nid;
    if (R.hit && s < R.cap) R.hit[s] = hit ? 1 : 0;
    return hit;
}

// the pairs of particle A with the partners in list[0 .. cnt - 1], one warp:
// ascending partners, and a task for each; range: the tasks' first and count
__device__ __forceinline__ void small_emit(const PairListDev& L, unsigned int* flags, int A, const int* list, int cnt,
                                           int lane, int2* task, int* ntask, int2* range)
{
    const unsigned int full = 0xffffffffu;
    if (cnt > MAX_CAND && lane == 0) set_flag(flags, FD_FLAG_NEIGHBOR_OVERFLOW);
    int n = min(cnt, MAX_CAND);
    int base = 0, t0 = 0;
    if (lane == 0 && n > 0) {
        base = atomicAdd(L.n_pairs, n);
        if (base + n > L.cap_pairs) {
            set_flag(flags, FD_FLAG_PAIR_OVERFLOW);
            n = 0;
        } else {
            t0 = atomicAdd(ntask, n);
        }
    }
    n = __shfl_sync(full, n, 0);
    base = __shfl_sync(full, base, 0);
    t0 = __shfl_sync(full, t0, 0);
    if (lane == 0) {
        L.seg_off[A] = n > 0 ? base : 0;
        L.seg_cnt[A] = n;
        *range = make_int2(t0, n);
    }
    for (int e = lane; e < n; e += 32) {
        const int v = list[e];
        int r = 0;
        for (int j = 0; j < n; ++j) r += (list[j] < v);
        L.pairA[base + r] = A;
        L.pairB[base + r] = v;
        task[t0 + r] = make_int2(v, SMALL_BODIES * (base + r) + A % SMALL_BODIES);
    }
    __syncwarp();
}

// BLOCKS: resident blocks per SM the registers are cut for
template <bool MIXED, int BLOCKS>
__global__ void __launch_bounds__(SMALL_WARPS * 32, BLOCKS) k_small_pairs(SmallArgs a)
{
    step_wait();
    using Real = typename std::conditional<MIXED, float, double>::type;
    constexpr int NODES = BLOCKS > 2 ? 1 : 2;
    // the candidate lists and the node queues are not in use together
    __shared__ union {
        unsigned short queue[SMALL_WARPS][MAX_NODE_QUEUE];
        struct {
            int found[SMALL_BODIES][MAX_FOUND];
            int list[SMALL_WARPS][MAX_CAND];
        } c;
    } q;
    // the block's pairs (partner, SMALL_BODIES * pair + body), partners in the
    // first half, walls in the second; their first slots and those of their
    // histories, and the counts of both; the first slot of each in the block's
    // order, partners then walls, the walls' from a multiple of 32; contacts
    __shared__ int2 s_task[2 * SMALL_TASKS];
    __shared__ int2 s_slot[2 * SMALL_TASKS];
    __shared__ ushort2 s_cnt[2 * SMALL_TASKS];
    __shared__ int s_first[2 * SMALL_TASKS + 1];
    __shared__ int s_hits[2 * SMALL_TASKS];
    __shared__ int2 s_range[SMALL_WARPS];
    __shared__ int s_ntask[2], s_pw;
    __shared__ unsigned long long s_stats[5];
    const NarrowArgs& n = a.n;
    const unsigned int full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int body = wib % SMALL_BODIES;
    if (threadIdx.x < 2) s_ntask[threadIdx.x] = 0;
    for (int t = threadIdx.x; t < 2 * SMALL_TASKS; t += blockDim.x) s_hits[t] = 0;
    if (threadIdx.x < 5) s_stats[threadIdx.x] = 0ull;
    if (threadIdx.x < SMALL_WARPS) s_range[threadIdx.x] = make_int2(0, 0);
    __syncthreads();
    const CellTableDev& T = a.T;
    const unsigned int build = T.build[T.par];
    // the other generation's step needs a number no head can hold
    if (blockIdx.x == 0 && threadIdx.x == 0) T.build[T.par ^ 1] = build + 1u;
    const int A0 = blockIdx.x * SMALL_BODIES, A = A0 + body;
    if (A < n.P.n) {
        const double3 cA = n.P.pos[A];
        const double rA = n.G.geo[n.P.geo[A]].radius;
        int* list = q.c.list[wib];
        int cnt = 0;
        int3 lo, hi;
        if (wib < SMALL_BODIES) {
            // partners: each lane walks the list of a cell, and the objects
            // found are tested side by side (a test is a chain of five loads)
            int* found = q.c.found[body];
            partner_search_range(cA, (rA + n.G.rmax) * (1.0 + 8.0 * BOUND_REL), T.g, lo, hi);
            const int nx = hi.x - lo.x + 1, ny = hi.y - lo.y + 1, nz = hi.z - lo.z + 1;
            const int ncell = nx * ny * nz;
            int nf = 0;
            auto test = [&] {
                __syncwarp();
                for (int f0 = 0; f0 < nf; f0 += 32) {
                    bool pass = false;
                    int B = -1;
                    if (f0 + lane < nf) {
                        B = found[f0 + lane];
                        const FdGeo& GB = n.G.geo[n.P.geo[B]];
                        const double3 cB = n.P.pos[B];
                        const double rs = rA + GB.radius;
                        if (lengthSq3(cA - cB) <= rs * rs * (1.0 + 4.0 * BOUND_REL))
                            pass = !body_culled32<true>(cA, rA, cB, n.P.rot + 3ll * B, true, n.G.geo32[n.P.geo[B]], n.G,
                                                  n.a.probe);
                    }
                    const unsigned int m = __ballot_sync(full, pass);
                    if (pass) {
                        const int at = cnt + __popc(m & ((1u << lane) - 1u));
                        if (at < MAX_CAND) list[at] = B;
                    }
                    cnt += __popc(m);
                }
                nf = 0;
                __syncwarp();
            };
            for (int c0 = 0; c0 < ncell; c0 += 32) {
                const int ci = c0 + lane;
                int B = -1;
                if (ci < ncell)
                    B = cell_first(T, fd_lin3(lo.x + ci % nx, lo.y + (ci / nx) % ny, lo.z + ci / (nx * ny), T.g.size),
                                   build);
                while (__any_sync(full, B >= 0)) {
                    const unsigned int m = __ballot_sync(full, B > A);
                    if (nf + __popc(m) > MAX_FOUND) test();
                    if (B > A) found[nf + __popc(m & ((1u << lane) - 1u))] = B;
                    nf += __popc(m);
                    if (B >= 0) B = T.next[B];
                }
            }
            test();
            small_emit(n.L, n.a.flags, A, list, cnt, lane, s_task, &s_ntask[0], &s_range[wib]);
        } else {
            body_search_range(cA, rA * (1.0 + BOUND_REL), n.wgrid, lo, hi);
            const int2 wr = a.wall_range ? a.wall_range[A] : make_int2(0, n.W.n);
            const int wend = min(wr.x + wr.y, n.W.n);
            for (int w0 = max(wr.x, 0); w0 < wend; w0 += 32) {
                const int w = w0 + lane;
                bool pass = false;
                const long long h = w < wend ? n.W.hash[w] : -1;
                if (h >= 0 && h < n.wgrid.num) {
                    int3 c;
                    decode_cell(h, n.wgrid.size, c);
                    if (c.x >= lo.x && c.x <= hi.x && c.y >= lo.y && c.y <= hi.y && c.z >= lo.z && c.z <= hi.z) {
                        const FdGeo& GB = n.GW.geo[n.W.geo[w]];
                        const double rs = rA + GB.grid_radius;
                        const double3 cW = n.W.pos[w];
                        pass = lengthSq3(cA - cW) <= rs * rs * (1.0 + 4.0 * BOUND_REL) &&
                               !body_culled32<true>(cA, rA, cW, n.W.rot + 3ll * w, false, n.GW.geo32[n.W.geo[w]], n.GW,
                                              n.a.probe);
                    }
                }
                const unsigned int m = __ballot_sync(full, pass);
                if (pass) {
                    const int at = cnt + __popc(m & ((1u << lane) - 1u));
                    if (at < MAX_CAND) list[at] = w;
                }
                cnt += __popc(m);
            }
            __syncwarp();
            small_emit(a.Lw, n.a.flags, A, list, cnt, lane, s_task + SMALL_TASKS, &s_ntask[1], &s_range[wib]);
        }
    }
    __syncthreads();
    // the block's pairs, shared out over its warps
    const int npp = s_ntask[0], ntask = npp + s_ntask[1];
    for (int u = wib; u < ntask; u += SMALL_WARPS) {
        const bool wall = u >= npp;
        const int t = wall ? SMALL_TASKS + u - npp : u;
        const int2 k = s_task[t];
        const int At = A0 + k.y % SMALL_BODIES, p = k.y / SMALL_BODIES;
        const int4 slot = wall ? small_slots<FD_PW, NODES>(n, a.Lw, p, At, k.x, lane, q.queue[wib], s_stats)
                               : small_slots<FD_PP, NODES>(n, n.L, p, At, k.x, lane, q.queue[wib], s_stats);
        if (lane == 0) {
            s_slot[t] = make_int2(slot.x, slot.z);
            s_cnt[t] = make_ushort2((unsigned short)slot.y, (unsigned short)slot.w);
        }
        __syncwarp();
    }
    __syncthreads();
    if (wib == 0) {
        int sum = 0;
        for (int u0 = 0; u0 < ntask; u0 += 32) {
            const int u = u0 + lane;
            const int c = u < ntask ? s_cnt[u >= npp ? SMALL_TASKS + u - npp : u].x : 0;
            int x = c;
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(full, x, d);
                if (lane >= d) x += y;
            }
            if (u < ntask) s_first[u] = sum + x - c;
            sum += __shfl_sync(full, x, 31);
        }
        __syncwarp();
        // the walls' slots start a warp
        const int pw = npp < ntask ? s_first[npp] : sum;
        const int shift = (32 - (pw & 31)) & 31;
        __syncwarp();
        for (int u = npp + lane; u < ntask; u += 32) s_first[u] += shift;
        if (lane == 0) {
            s_first[ntask] = sum + shift;
            s_pw = pw + shift;
        }
    }
    __syncthreads();
    // the block's slots, a thread each
    for (int j = threadIdx.x; j < s_first[ntask]; j += blockDim.x) {
        int lo = 0, hi = ntask;  // the last pair that starts at or before slot j
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_first[mid] <= j) lo = mid; else hi = mid;
        }
        const bool wall = j >= s_pw;
        const int t = wall ? SMALL_TASKS + lo - npp : lo;
        const int2 k = s_task[t], slot = s_slot[t];
        const ushort2 cnt = s_cnt[t];
        const int i = j - s_first[lo], At = A0 + k.y % SMALL_BODIES;
        if (i >= cnt.x) continue;
        const bool hit =
            wall ? small_contact<FD_PW, MIXED>(n, a.Lw, a.recw, At, k.x, slot.x + i, slot.y, cnt.y)
                 : small_contact<FD_PP, MIXED>(n, n.L, n.a.rec, At, k.x, slot.x + i, slot.y, cnt.y);
        if (hit) atomicAdd(&s_hits[t], 1);
    }
    __syncthreads();
    // the sums of the pairs that hold contacts, as sum_list
    const int grp = lane >> 3, l = lane & 7;
    for (int u0 = 4 * wib; u0 < ntask; u0 += 4 * SMALL_WARPS) {
        const int u = u0 + grp;
        const bool wall = u >= npp;
        const int t = u >= ntask ? -1 : wall ? SMALL_TASKS + u - npp : u;
        const int hits = t >= 0 ? s_hits[t] : 0;
        const int base = hits ? s_slot[t].x : 0, c = hits ? s_cnt[t].x : 0;
        const PairListDev& L = wall ? a.Lw : n.L;
        Real acc = 0, acc8 = 0;
        const int cmax = __reduce_max_sync(full, c);
        int node = l < c ? L.c_node[base + l] : -1;
        for (int j0 = 0; j0 < cmax; j0 += 8) {
            const unsigned int any = __ballot_sync(full, node >= 0);
            node = j0 + 8 + l < c ? L.c_node[base + j0 + 8 + l] : -1;
            if (any) add_contacts(L.c_rec, (any >> (8 * grp)) & 0xffu, base + j0 + l, l, acc, acc8);
        }
        if (!hits) continue;
        // a pair without a contact sums to zero: nobody reads it
        const int p = s_task[t].y / SMALL_BODIES;
        Real* out = reinterpret_cast<Real*>(L.pf) + (long long)RESULT * p;
        out[l / 3 * 4 + l % 3] = acc;
        if (l == 0) {
            out[10] = acc8;
            atomicAdd(L.n_hits, hits);
            if (!wall) L.r_next[p] = atomicExch(&a.r_head[s_task[t].x], p);
            if (n.a.stats) atomicAdd(&s_stats[3], (unsigned long long)hits);
        }
    }
    __syncthreads();
    // each particle's own pairs, partners then walls, in order: lane t < 3 sums
    // the force, lane 3 <= t < 6 the torque
    if (wib < SMALL_BODIES && A < n.P.n && lane < 6) {
        Real acc = 0;
        for (int w = 0; w < 2; ++w) {
            const int2 r = s_range[body + w * SMALL_BODIES];
            const Real* pf = reinterpret_cast<const Real*>(w ? a.Lw.pf : n.L.pf);
            for (int t = r.x + w * SMALL_TASKS; t < r.x + w * SMALL_TASKS + r.y; ++t)
                if (s_hits[t]) acc += pf[(long long)RESULT * (s_task[t].y / SMALL_BODIES) + lane / 3 * 4 + lane % 3];
        }
        reinterpret_cast<Real*>(a.own)[6ll * A + lane] = acc;
    }
    if (n.a.stats && threadIdx.x < 5 && s_stats[threadIdx.x])
        atomicAdd(&n.a.stats[threadIdx.x], s_stats[threadIdx.x]);
}

struct SmallAdvanceArgs {
    ObjDev P, W;
    GeoSetDev G;
    FdGrid pgrid, wgrid;
    PairListDev Lp;        // the step's particle-particle list
    BondDev B;
    CellTableDev T;        // the next step's table
    int* r_head;           // see SmallArgs
    const void* own;
    int* zero[2];          // counters of the next step's lists (three each)
    double3 gravity;
    double h, dt;
};

// the particle's pairs as a partner, by owner; its list is emptied.  The list
// is in no order: a pass over it keeps the next LOCAL owners, so a body with
// many takes a pass for each LOCAL of them (a body with 100, 400 and 1,500
// owners: 218, 1,800 and 19,000 us a step; with a pass for each owner 732,
// 10,600 and 147,000, in the staged kernels 360, 4,400 and 54,000).
template <typename Real>
__device__ __forceinline__ void small_partner_sum(const SmallAdvanceArgs& a, int i, ForceSum<Real>& f)
{
    constexpr int LOCAL = 16;
    const PairListDev& L = a.Lp;
    const int head = a.r_head[i];
    if (head < 0) return;
    a.r_head[i] = -1;
    int pair[LOCAL], owner[LOCAL], cnt = 0;
    for (int p = head; p >= 0; p = L.r_next[p], ++cnt) {
        if (cnt >= LOCAL) continue;
        const int own = L.pairA[p];
        int b = cnt - 1;
        while (b >= 0 && owner[b] > own) { owner[b + 1] = owner[b]; pair[b + 1] = pair[b]; --b; }
        owner[b + 1] = own;
        pair[b + 1] = p;
    }
    const Real* pf = reinterpret_cast<const Real*>(L.pf);
    if (cnt <= LOCAL) {
#pragma unroll 4
        for (int e = 0; e < cnt; ++e) f.add(pf, pair[e], Real(-1), 2);
        return;
    }
    int last = -1;
    for (int left = cnt; left > 0; left -= LOCAL) {
        int kept = 0;
        for (int p = head; p >= 0; p = L.r_next[p]) {
            const int own = L.pairA[p];
            if (own <= last || (kept == LOCAL && own > owner[LOCAL - 1])) continue;
            int b = (kept < LOCAL ? kept++ : LOCAL - 1) - 1;
            while (b >= 0 && owner[b] > own) { owner[b + 1] = owner[b]; pair[b + 1] = pair[b]; --b; }
            owner[b + 1] = own;
            pair[b + 1] = p;
        }
        for (int e = 0; e < kept; ++e) f.add(pf, pair[e], Real(-1), 2);
        last = owner[LOCAL - 1];
    }
}

// SUM: the step's forces; BACK: its second half kick; FRONT: the next step's
// first half kick, drift, hash and cell lists
template <typename Real, bool SUM, bool BACK, bool FRONT>
__global__ void __launch_bounds__(64) k_small_advance(SmallAdvanceArgs a)
{
    step_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (FRONT && i < 6) a.zero[i / 3][i % 3] = 0;
    if (i < a.P.n) {
        // one thread a body and a block or less an SM: the kernel is its chain
        // of loads, so the state is on its way before the sums start
        Body b;
        int gi = 0;
        if (BACK || FRONT) {
            gi = load_now(a.P.geo + i);
            b.x = load_now(a.P.pos + i);
            b.v = load_now(a.P.vel + i);
            b.w = load_now(a.P.angvel + i);
            b.q = load_now(a.P.q + i);
        }
        double3 F, T;
        if (SUM) {
            ForceSum<Real> f;
            const Real* own = reinterpret_cast<const Real*>(a.own) + 6ll * i;
            for (int t = 0; t < 3; ++t) {
                f.F[t] = own[t];
                f.T[t] = own[3 + t];
            }
            small_partner_sum(a, i, f);
            if (a.B.n > 0) f.bonds(a.B, i);
            F = mk3((double)f.F[0], (double)f.F[1], (double)f.F[2]);
            T = mk3((double)f.T[0], (double)f.T[1], (double)f.T[2]);
            a.P.force[i] = F;
            a.P.torque[i] = T;
        } else {
            F = a.P.force[i];
            T = a.P.torque[i];
        }
        if (!BACK && !FRONT) return;
        const FdGeo& geo = a.G.geo[gi];
        if (BACK) kick_body(b, geo, F, T, a.gravity, a.h);
        if (FRONT) {
            kick_body(b, geo, F, T, a.gravity, a.h);
            drift_body(b, a.dt);
            a.P.pos[i] = b.x;
            a.P.q[i] = b.q;
            const long long h = hash_one(a.P, a.pgrid, i, b.x, b.q);
            if (h >= 0 && h < a.T.g.num) cell_push(a.T, (unsigned long long)h, a.T.build[a.T.par], i);
        }
        a.P.vel[i] = b.v;
        a.P.angvel[i] = b.w;
    } else if (FRONT && i - a.P.n < a.W.n) {
        const int w = i - a.P.n;
        Body b{a.W.pos[w], a.W.vel[w], a.W.angvel[w], a.W.q[w]};
        drift_body(b, a.dt);
        a.W.pos[w] = b.x;
        a.W.q[w] = b.q;
        hash_one(a.W, a.wgrid, w, b.x, b.q);
    }
}

}  // namespace

// kernel launches are counted into the counter the calling thread set
// (fundem_launch_count); none when it set none
thread_local long long* t_launch_counter = nullptr;
void set_launch_counter(long long* c) { t_launch_counter = c; }
thread_local bool t_launch_ahead = true;
void set_launch_ahead(bool on) { t_launch_ahead = on; }
void count_launch()
{
    if (t_launch_counter) ++*t_launch_counter;
}
static inline void note_launch()
{
    if (t_launch_counter) ++*t_launch_counter;
}
// For kernels that begin with step_wait: the two of a small set's step, plain
// launches.  Not in recorded graphs, whose launches are a microsecond apart as
// it is (4,096 particles: 65.8 us a step against 64.8); a plain step of 777
// particles went from 52.6 to 44.6 us.  The staged kernels have no such wait and
// are launched one after the other; whether they would gain was not measured.
template <typename... P, typename... A>
static void launch_ahead(void (*kernel)(P...), int blocks, int threads, cudaStream_t s, const A&... args)
{
    cudaLaunchAttribute ahead{};
    ahead.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    ahead.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3((unsigned)threads);
    c.stream = s;
    c.attrs = &ahead;
    c.numAttrs = t_launch_ahead ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, P(args)...);
    note_launch();
}
template <typename... P, typename... A>
static void launch_step(void (*kernel)(P...), int blocks, int threads, cudaStream_t s, const A&... args)
{
    kernel<<<blocks, threads, 0, s>>>(args...);
    note_launch();
}

// ---------------------------------------------------------------------------
// contiguous views of a contact list and of the bonds (the device arrays the
// reference's SolidInteraction and VBondedInteraction getters return)
// ---------------------------------------------------------------------------
__global__ void k_view_keys(PairListDev L, long long* key)
{
    const int nslots = min(*L.n_slots, L.cap_contacts);
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < L.cap_contacts; s += gridDim.x * blockDim.x) {
        const int node = s < nslots ? L.c_node[s] : -1;
        key[s] = node >= 0 ? ((long long)node << 32) | (unsigned int)__double2loint(L.c_hist[L.c_at[s]].w) : -1ll;
    }
}
__global__ void k_view_gather(PairListDev L, const int* order, long long n, ContactViewDev v)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int s = order[i];
        v.master[i] = L.c_node[s];
        const int t = L.c_at[s];
        const double4 hist = L.c_hist[t];
        const double* r = L.c_rec + (long long)CONTACT_REC * t;
        for (int d = 0; d < 3; ++d) {
            v.point[3 * i + d] = r[CONTACT_POINT + d];
            v.normal[3 * i + d] = r[CONTACT_NORMAL + d];
            v.spring[3 * i + d] = d == 0 ? hist.x : d == 1 ? hist.y : hist.z;
        }
        v.slave[i] = __double2loint(hist.w);
        v.overlap[i] = r[CONTACT_OVERLAP];
        v.en[i] = r[CONTACT_EN];
        v.es[i] = r[CONTACT_ES];
    }
}
// the contacts of a list packed field by field (count of them, in no order):
// the host reads those back instead of every slot, most of which hold none
__global__ void k_pack_contacts(PairListDev L, ContactPackDev v, int* at, int count)
{
    const int nslots = min(*L.n_slots, L.cap_contacts);
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nslots; s += gridDim.x * blockDim.x) {
        const int node = L.c_node[s];
        if (node < 0) continue;
        const int i = atomicAdd(at, 1);
        if (i >= count) continue;
        const int t = L.c_at[s];
        const double4 hist = L.c_hist[t];
        const double* r = L.c_rec + (long long)CONTACT_REC * t;
        for (int d = 0; d < 3; ++d) {
            if (v.point) v.point[3 * i + d] = r[CONTACT_POINT + d];
            if (v.normal) v.normal[3 * i + d] = r[CONTACT_NORMAL + d];
            if (v.spring) v.spring[3 * i + d] = d == 0 ? hist.x : d == 1 ? hist.y : hist.z;
        }
        v.id[i] = make_int2(node, __double2loint(hist.w));
        if (v.overlap) v.overlap[i] = r[CONTACT_OVERLAP];
        if (v.en) v.en[i] = r[CONTACT_EN];
        if (v.es) v.es[i] = r[CONTACT_ES];
    }
}
__global__ void k_bond_view(BondDev B, BondViewDev v)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= B.n) return;
    for (int t = 0; t < 4; ++t) v.B[t][k] = B.B[4 * k + t];
    for (int t = 0; t < 6; ++t) v.energy[t][k] = B.energy[6 * k + t];
    for (int t = 0; t < 8; ++t) v.frames[t][k] = B.frames[8 * k + t];
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
size_t scan_tmp_size(long long n)
{
    size_t total = 0;
    long long m = n;
    while (m > SCAN_TILE) {
        m = (m + SCAN_TILE - 1) / SCAN_TILE;
        total += (size_t)m;
    }
    return total + 1;
}

void scan_exclusive(const int* in, int* out, long long n, int* tmp, cudaStream_t s)
{
    if (n <= 0) return;
    if (n <= SCAN_TILE) {
        k_scan_tile<false><<<1, SCAN_TPB, 0, s>>>(in, out, n, nullptr); note_launch();
        return;
    }
    const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    int* sums = tmp;
    k_scan_tile<false><<<(unsigned)tiles, SCAN_TPB, 0, s>>>(in, out, n, sums); note_launch();
    scan_exclusive(sums, sums, tiles, tmp + tiles, s);
    k_scan_add<<<(unsigned)tiles, SCAN_TPB, 0, s>>>(out, n, sums); note_launch();
}

void scan_inclusive(const int* in, int* out, long long n, int* tmp, cudaStream_t s)
{
    if (n <= 0) return;
    if (n <= SCAN_TILE) {
        k_scan_tile<true><<<1, SCAN_TPB, 0, s>>>(in, out, n, nullptr); note_launch();
        return;
    }
    const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    int* sums = tmp;
    k_scan_tile<true><<<(unsigned)tiles, SCAN_TPB, 0, s>>>(in, out, n, sums); note_launch();
    scan_exclusive(sums, sums, tiles, tmp + tiles, s);
    k_scan_add<<<(unsigned)tiles, SCAN_TPB, 0, s>>>(out, n, sums); note_launch();
}

__global__ void __launch_bounds__(TPB) k_sdf_quads(const double* sdf, const float* sdf32, double4* quad,
                                                   float4* quad32, int3 size, long long n)
{
    const long long sx = size.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        // points of the last column or row start no cell
        const bool cell = i % sx + 1 < sx && (i / sx) % size.y + 1 < size.y;
        if (quad)
            quad[i] = cell ? make_double4(sdf[i], sdf[i + 1], sdf[i + sx], sdf[i + sx + 1]) : make_double4(0., 0., 0., 0.);
        quad32[i] =
            cell ? make_float4(sdf32[i], sdf32[i + 1], sdf32[i + sx], sdf32[i + sx + 1]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
void launch_sdf_quads(const double* sdf, const float* sdf32, double4* quad, float4* quad32, long long off, int3 size,
                      cudaStream_t s)
{
    const long long n = (long long)size.x * size.y * size.z;
    if (n <= 0) return;
    k_sdf_quads<<<(int)std::min<long long>((n + TPB - 1) / TPB, 148 * 8), TPB, 0, s>>>(sdf + off, sdf32 + off,
                                                                                       quad ? quad + off : nullptr, quad32 + off, size, n);
    note_launch();
}

void launch_hash(const ObjDev& O, const FdGrid& g, cudaStream_t s, unsigned int* build, int par)
{
    if (O.n > 0) { k_hash<<<nblocks(O.n), TPB, 0, s>>>(O, g, build, par); note_launch(); }
}
void radix_sort_scratch(int n, size_t& bcount_ints, size_t& bscan_ints)
{
    const long long nblk = std::max<long long>((n + RS_TPB - 1) / RS_TPB, 1);
    bcount_ints = (size_t)(RS_RADIX * nblk);
    bscan_ints = scan_tmp_size((long long)bcount_ints);
}
void radix_sort_keys(const long long* keys, int n, long long num_keys, unsigned long long* out_key, int* out_idx,
                     unsigned long long* key_b, int* idx_b, int* bcount, int* bscan_tmp, cudaStream_t s)
{
    if (n <= 0) return;
    // bits a key can use; keys of objects in no cell sort after every cell
    int bits = 1;
    while (bits < 64 && ((unsigned long long)num_keys >> bits) != 0ull) ++bits;
    const int passes = (bits + 7) / 8;
    const int nblk = (n + RS_TPB - 1) / RS_TPB;
    // the last pass writes (out_key, out_idx)
    unsigned long long* kb[2] = {out_key, key_b};
    int* ib[2] = {out_idx, idx_b};
    int src = passes & 1;
    k_rs_keys<<<nblocks(n), TPB, 0, s>>>(keys, n, num_keys, kb[src], ib[src]); note_launch();
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        k_rs_hist<<<nblk, RS_TPB, 0, s>>>(kb[src], n, shift, bcount, nblk); note_launch();
        scan_exclusive(bcount, bcount, (long long)RS_RADIX * nblk, bscan_tmp, s);
        k_rs_scatter<<<nblk, RS_TPB, 0, s>>>(kb[src], ib[src], n, shift, bcount, nblk, kb[src ^ 1], ib[src ^ 1]);
        note_launch();
        src ^= 1;
    }
}
void launch_images(const ObjDev& P, double3* dst, const GhostDev* gh, const int* on, double ext_skin, int* ctrl,
                   cudaStream_t s)
{
    if (P.n <= 0) return;
    ImageArgs a{P, dst, {gh[0], gh[1], gh[2]}, {on[0], on[1], on[2]}, ext_skin, ctrl};
    launch_step(k_images, nblocks(P.n), TPB, s, a);
}
void reset_image_box(int* occ, cudaStream_t s)
{
    cudaMemsetAsync(occ, 0x7f, 3 * sizeof(int), s);
    cudaMemsetAsync(occ + 3, 0xff, 3 * sizeof(int), s);
}
void launch_sector_wrap(ObjDev& P, const FdGrid& g, cudaStream_t s)
{
    if (P.n > 0) { k_sector_wrap<<<nblocks(P.n), TPB, 0, s>>>(P, g.minb); note_launch(); }
}
void launch_sector_images(const ObjDev& P, GhostDev* R, cudaStream_t s)
{
    if (P.n > 0) { k_sector_images<<<nblocks(P.n), TPB, 0, s>>>(P, R[0], R[1], R[2]); note_launch(); }
}

namespace {
// kernel arguments of a set of lists, with blocks[k] blocks for list k
ListSet list_set(const ListArgs* lists, int n, const StepShared& c, const int* blocks)
{
    if (n > MAX_LISTS) throw std::logic_error("more contact lists than a launch takes");
    ListSet a;
    a.n = n;
    a.T = c.T;
    a.wall_range = c.wall_range;
    a.rev_total = c.with_force ? c.R.total : nullptr;
    a.spacing_margin = c.mixed ? 1e-4f : 0.f;
    int b = 0;
    for (int k = 0; k < n; ++k) {
        NarrowArgs& m = a.l[k];
        m.P = lists[k].P; m.G = c.G; m.M = c.M; m.W = c.W; m.GW = c.GW; m.MW = c.MW;
        m.pgrid = c.pgrid; m.wgrid = c.wgrid; m.gh = lists[k].gh; m.L = lists[k].L; m.a = lists[k].a;
        m.with_force = c.with_force;
        a.kind[k] = lists[k].kind;
        a.block0[k] = b;
        b += blocks[k];
    }
    a.block0[n] = b;
    return a;
}
}  // namespace

void launch_broad(const ListArgs* lists, int n, const StepShared& c, NlDev* nl, cudaStream_t s)
{
    if (n <= 0 || c.n <= 0) return;
    int blocks[FD_NKIND];
    // sparse tables: the keys of the lists that are built are cleared first
    for (int k = 0; k < n; ++k) {
        if (lists[k].kind == FD_PW) continue;
        const CellTableDev& T = lists[k].kind == FD_PP ? c.T : lists[k].gh.cells;
        if (!T.hashed) continue;
        k_hkey_clear<<<nblocks((long long)T.hmask + 1), TPB, 0, s>>>(T.hkey, T.hmask + 1, lists[k].a);
        note_launch();
    }
    for (int k = 0; k < n; ++k) blocks[k] = std::min(nblocks(c.n), 148 * 8);
    ListSet a = list_set(lists, n, c, blocks);
    launch_step(k_begin_lists, a.block0[n], TPB, s, a);
    if (nl) {
        // the particle-particle list comes from the neighbour list
        for (int k = 0; k < n; ++k) {
            if (lists[k].kind != FD_PP) continue;
            k_nl_check<<<nblocks(c.n), TPB, 0, s>>>(lists[k].P, *nl, c.T.g); note_launch();
            k_broad_nl<<<nblocks((long long)c.n * BROAD_LANES), TPB, 0, s>>>(lists[k].P, c.G, c.T, *nl, lists[k].a.flags);
            note_launch();
            k_nl_filter<<<nblocks((long long)c.n * 8), TPB, 0, s>>>(lists[k].P, c.G, lists[k].L, *nl, lists[k].a.flags,
                                                                   lists[k].a.probe);
            note_launch();
        }
    }
    int total = 0;
    for (int k = 0; k < n; ++k) {
        const bool pp = lists[k].kind == FD_PP;
        blocks[k] = pp && nl ? 0
                    : lists[k].kind == FD_PW ? std::min(nblocks(c.n), 148 * 4)
                                             : std::min(nblocks((long long)c.n * BROAD_LANES), 148 * 4);
        total += blocks[k];
    }
    if (total == 0) return;
    a = list_set(lists, n, c, blocks);
    launch_step(k_broad_lists, total, TPB, s, a);
}

void launch_narrow(const ListArgs* lists, int n, const StepShared& c, cudaStream_t s)
{
    if (n <= 0 || c.n <= 0) return;
    // grid-stride kernels sized in blocks per SM (the pair and slot counts are
    // known only on the device): the particle-particle list's defaults fill
    // one resident wave; the short wall and image lists come first and get a
    // quarter of it each, so that they end before the long list does
    int shape[4];
    for (int k = 0; k < 4; ++k) shape[k] = lists[0].a.shape[k] > 0 ? lists[0].a.shape[k] : DEFAULT_SHAPE[k];
    auto share = [&](int* blocks, int per_sm) {
        for (int k = 0; k < n; ++k) {
            const long long need = ((long long)lists[k].L.cap_pairs + NARROW_WARPS - 1) / NARROW_WARPS;
            const long long most = lists[k].kind == FD_PP || n == 1 ? 148ll * per_sm : 148ll * std::max(per_sm / 4, 1);
            blocks[k] = (int)std::max(1ll, std::min(need, most));
        }
    };
    int blocks[FD_NKIND];
    share(blocks, shape[0]);
    ListSet a = list_set(lists, n, c, blocks);
    launch_step(k_select_lists, a.block0[n], NARROW_WARPS * 32, s, a);
    for (int k = 0; k < n; ++k) {
        if (lists[k].kind != FD_PP || !lists[k].a.gate) continue;
        launch_step(k_slot_filter, 148 * shape[1], TPB, s, a.l[k]);
    }
    share(blocks, shape[1]);
    a = list_set(lists, n, c, blocks);
    launch_step(c.mixed ? k_contact_lists<true, 0> : k_contact_lists<false, 0>, a.block0[n], TPB, s, a);
    share(blocks, shape[2]);
    a = list_set(lists, n, c, blocks);
    launch_step(c.mixed ? k_contact_lists<true, 1> : k_contact_lists<false, 1>, a.block0[n], TPB, s, a);
    if (!c.with_force) return;
    share(blocks, shape[3]);
    a = list_set(lists, n, c, blocks);
    launch_step(c.mixed ? k_sum_lists<float> : k_sum_lists<double>, a.block0[n], SUM_TPB, s, a, c.R);
}

void launch_cache_refs(const ObjDev& P, const ObjDev& W, const PairCacheDev& pc, cudaStream_t s)
{
    if (P.n > 0) launch_step(k_cache_refs, std::min(nblocks(P.n), 148 * 8), TPB, s, pc, P, W);
}

void launch_step_end(const ObjDev& P, const ObjDev& W, const PairListDev* lists, const int* active, const RevDev& R,
                     const PairCacheDev* pc, bool cached_ghosts, bool refs, unsigned int* done, unsigned int* flags,
                     cudaStream_t s)
{
    if (P.n <= 0) return;
    EndArgs a;
    a.P = P;
    a.W = W;
    for (int k = 0; k < FD_NKIND; ++k) { a.L[k] = lists[k]; a.active[k] = active[k]; }
    a.R = R;
    a.cached = pc != nullptr;
    a.cached_ghosts = cached_ghosts;
    a.refs = refs;
    if (pc) a.pc = *pc; else memset(&a.pc, 0, sizeof(a.pc));
    a.done = done;
    a.flags = flags;
    launch_step(k_step_end, std::min(nblocks(P.n), 148 * 8), TPB, s, a);
}

void launch_advance(const StepShared& c, const ObjDev& P, const PairListDev* lists, const int* active, const BondDev& B,
                    const double3* wrapped, double3 gravity, double dt, const PairCacheDev* pc, int* const* occ,
                    int par, int parts, cudaStream_t s)
{
    // without particles there are still walls to move
    if (P.n <= 0 && (!(parts & STEP_FRONT) || c.W.n <= 0)) return;
    AdvanceArgs a;
    a.P = P; a.W = c.W; a.G = c.G; a.GW = c.GW; a.pgrid = c.pgrid; a.wgrid = c.wgrid;
    a.r.R = c.R;
    a.r.B = B;
    for (int k = 0; k < FD_NKIND; ++k) { a.r.L[k] = lists[k]; a.r.active[k] = active[k]; }
    a.wrapped = wrapped;
    a.gravity = gravity;
    a.h = 0.5 * dt;
    a.dt = dt;
    a.build = c.T.build;
    a.par = par;
    a.cached = pc != nullptr;
    if (pc) a.pc = *pc; else memset(&a.pc, 0, sizeof(a.pc));
    for (int d = 0; d < 6; ++d) a.occ[d] = occ[d];
    const int tpb = 128;
    const int blocks = std::max(1, nblocks(P.n + ((parts & STEP_FRONT) ? c.W.n : 0), tpb));
#define FD_ADVANCE(S, K, F)                                                                  \
    case (S ? STEP_SUM : 0) | (K ? STEP_BACK : 0) | (F ? STEP_FRONT : 0):                    \
        launch_step(c.mixed ? k_advance<float, S, K, F> : k_advance<double, S, K, F>, blocks, tpb, s, a); \
        break;
    switch (parts) {
        FD_ADVANCE(false, false, true)
        FD_ADVANCE(false, true, false)
        FD_ADVANCE(false, true, true)
        FD_ADVANCE(true, false, false)
        FD_ADVANCE(true, true, false)
        FD_ADVANCE(true, true, true)
    }
#undef FD_ADVANCE
}

void launch_small_pairs(const ObjDev& P, const GeoSetDev& G, const MatDev& M, const ObjDev& W, const GeoSetDev& GW,
                        const MatDev& MW, const FdGrid& pgrid, const FdGrid& wgrid, const CellTableDev& T,
                        const PairListDev& Lp, const PairListDev& Lw, const StepArgs& a, const AdjRec& recw,
                        const int2* wall_range, int* r_head, void* own, bool mixed, cudaStream_t s)
{
    if (P.n <= 0) return;
    SmallArgs k;
    NarrowArgs& n = k.n;
    n.P = P; n.G = G; n.M = M; n.W = W; n.GW = GW; n.MW = MW; n.pgrid = pgrid; n.wgrid = wgrid;
    memset(&n.gh, 0, sizeof(n.gh));
    n.L = Lp; n.a = a; n.with_force = 1;
    k.Lw = Lw; k.recw = recw; k.T = T; k.wall_range = wall_range; k.r_head = r_head;
    k.own = own;
    const int blocks = (P.n + SMALL_BODIES - 1) / SMALL_BODIES;
    // A block is a chain of some 20 us whatever its neighbours do.  While all
    // blocks are resident at two per SM (1,184 particles) the kernel keeps its
    // registers; more blocks than that go four to an SM with half as many,
    // spilled values and all (4,096 particles: 65 us a step against 76; 1,000
    // particles: 46 against 39).
    const bool many = blocks > 2 * 148;
    launch_ahead(mixed ? (many ? k_small_pairs<true, 4> : k_small_pairs<true, 2>)
                       : (many ? k_small_pairs<false, 4> : k_small_pairs<false, 2>),
                 blocks, SMALL_WARPS * 32, s, k);
}

void launch_small_advance(const ObjDev& P, const GeoSetDev& G, const ObjDev& W, const FdGrid& pgrid,
                          const FdGrid& wgrid, const PairListDev& Lp, const BondDev& B, const CellTableDev& T,
                          int* r_head, const void* own, int* zero_p, int* zero_w, double3 gravity, double dt,
                          bool mixed, int parts, cudaStream_t s)
{
    if (P.n <= 0) return;
    SmallAdvanceArgs a{P, W, G, pgrid, wgrid, Lp, B, T, r_head, own, {zero_p, zero_w}, gravity, 0.5 * dt, dt};
    // small blocks: the work is a chain of dependent loads per particle, so it
    // goes to as many SMs as there are
    const int tpb = 64;
    const int blocks = std::max(1, (P.n + ((parts & STEP_FRONT) ? W.n : 0) + tpb - 1) / tpb);
#define FD_ADVANCE(S, K, F)                                                                                    \
    case (S ? STEP_SUM : 0) | (K ? STEP_BACK : 0) | (F ? STEP_FRONT : 0):                                   \
        launch_ahead(mixed ? k_small_advance<float, S, K, F> : k_small_advance<double, S, K, F>, blocks, tpb, s, a); \
        break;
    switch (parts) {
        FD_ADVANCE(false, false, true)
        FD_ADVANCE(true, false, false)
        FD_ADVANCE(true, true, false)
        FD_ADVANCE(true, true, true)
    }
#undef FD_ADVANCE
}

void launch_bonds(const ObjDev& P, BondDev& B, bool mixed, cudaStream_t s)
{
    if (B.n <= 0) return;
    if (mixed) {
        k_bonds32<<<nblocks(B.n), TPB, 0, s>>>(P, B);
    } else {
        k_bonds<<<nblocks(B.n), TPB, 0, s>>>(P, B);
    }
    note_launch();
}

void launch_contact_view(const PairListDev& L, long long* keys, int* order, unsigned long long* skey,
                         unsigned long long* key_b, int* idx_b, int* bcount, int* bscan, long long n,
                         long long max_key, const ContactViewDev& v, cudaStream_t s)
{
    if (L.cap_contacts <= 0) return;
    k_view_keys<<<148 * 4, TPB, 0, s>>>(L, keys); note_launch();
    radix_sort_keys(keys, L.cap_contacts, max_key, skey, order, key_b, idx_b, bcount, bscan, s);
    if (n > 0) { k_view_gather<<<148 * 4, TPB, 0, s>>>(L, order, n, v); note_launch(); }
}
void launch_pack_contacts(const PairListDev& L, const ContactPackDev& v, int* at, int count, cudaStream_t s)
{
    cudaMemsetAsync(at, 0, sizeof(int), s);
    k_pack_contacts<<<148 * 4, TPB, 0, s>>>(L, v, at, count); note_launch();
}
void launch_bond_view(const BondDev& B, const BondViewDev& v, cudaStream_t s)
{
    if (B.n > 0) { k_bond_view<<<nblocks(B.n), TPB, 0, s>>>(B, v); note_launch(); }
}

}  // namespace fd

// ---------------------------------------------------------------------------
// Prefix sum without allocation.
//
// For callers that cannot allocate device memory when they need the scan:
// code that runs inside a device-memory budget owned by another allocator
// (a framework that has reserved the GPU's memory up front, where a
// cudaMalloc can fail), and code for which cudaMalloc's implicit device-wide
// synchronisation is not acceptable.  The scratch (one int per 4096-element
// tile) lives in a fixed device array of this library instead, so the scan
// is limited to FUNDEM_NOALLOC_SCAN_MAX elements.  Every GPU that loads the
// library keeps the 16 KiB array until the process exits.
//
// The array is shared by all calls on a device and keeps the last call's
// contents.  Nothing in it needs to start at zero: every tile sum the scan
// reads is written earlier in the same call.  Calls that overlap on the GPU
// (concurrent streams) race on the array.
// ---------------------------------------------------------------------------
namespace {
constexpr int NOALLOC_TILES = 4096;
static_assert((long long)NOALLOC_TILES * fd::SCAN_TILE == FUNDEM_NOALLOC_SCAN_MAX, "limit and scratch size differ");
static __device__ __align__(256) int g_noalloc_scan_scratch[NOALLOC_TILES];

constexpr int NOALLOC_MAX_DEVICES = 256;
std::mutex g_noalloc_mutex;
int* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {nullptr};

// device address of the scratch on the current device; looked up once per
// device (host code only sees a stand-in for the array's address)
int noalloc_scratch(int** out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return FUNDEM_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        int* p = nullptr;
        if (cudaGetSymbolAddress((void**)&p, g_noalloc_scan_scratch) != cudaSuccess || !p) return FUNDEM_ERR_CUDA;
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return FUNDEM_OK;
}
}  // namespace

extern "C" int fundem_prefix_sum_noalloc(int* d_prefix, const int* d_count, long long n, void* stream)
{
    if (n < 0 || (n > 0 && (!d_prefix || !d_count))) return FUNDEM_ERR_ARG;
    if (n > FUNDEM_NOALLOC_SCAN_MAX) return FUNDEM_ERR_ARG;
    if (n == 0) return FUNDEM_OK;
    int* scratch = nullptr;
    const int r = noalloc_scratch(&scratch);
    if (r != FUNDEM_OK) return r;
    // n <= NOALLOC_TILES * SCAN_TILE: the tile sums fit the array and their
    // own scan is a single tile, which needs no further scratch
    fd::scan_inclusive(d_count, d_prefix, n, scratch, (cudaStream_t)stream);
    return cudaGetLastError() == cudaSuccess ? FUNDEM_OK : FUNDEM_ERR_CUDA;
}
