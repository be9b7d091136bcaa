// +z ray-parity voxelizer -- bit-identical to the reference's labelPoints.
//
// Restates, per lattice point, the reference's FP64 arithmetic in its exact
// operation order (this translation unit is compiled with --fmad=false, so
// no multiply-add is contracted, matching the reference built with
// -ffp-contract=off):
//   ray construction       ComplexGeometry.cpp:987-1035 (case 0, +z)
//   ray adjustment         ComplexGeometry.cpp:853-884
//   ray/plane test         ComplexGeometry.cpp:803-848 (uses the STL's facet normal)
//   point-in-triangle      ComplexGeometry.cpp:620-674 (recomputed normal, +z projection)
//   parity -> Fluid        ComplexGeometry.cpp:1041-1048
//
// GB300 design: the reference tests every point against every triangle
// (O(N*T)).  Here a triangle meets only the lattice columns within its xy extent
// widened by 4 L E (tri_extent): L its longest edge at vertex 1, E a bound of
// the rounding of the reference's barycentric coordinates (barycentric_bound),
// beyond which the point-in-triangle test fails for every point of the column,
// so that leaving the triangle out changes no count.  Triangles that can never
// pass (zero area, a computed normal with |n_z| < 1e-16 or a file normal whose z
// the plane test rejects) have no columns; those too ill-conditioned for any
// bound (cull_margin) go to a global list tested by every point.
// All points of a column share the ray's x and y, so a (column, triangle)
// pair is decided once for the whole column: whether the line lies inside
// the triangle does not depend on k but for rounding, and the crossing
// counts for the k below the height where the line meets the facet plane.
// Both decisions carry a bound of ~300 times the worst rounding of the
// reference's tests; what lies within it (a line through an edge or a
// vertex, a point on the facet) is left to the reference's own FP64 test of
// that (point, triangle).  The pair flips the parity of a range of k: two
// bits of a difference bit field, whose running XOR along k is the mask.
// (70,040 triangles on a 56 x 54 x 509 lattice: 0.19 ms in these kernels,
// where one FP64 test per point and candidate took 12.3 ms at GB300's two
// FP64 multiply-adds a cycle and SM; k_tri_columns is bound by its ~400 FP64
// operations a triangle.)
#include <cmath>
#include <algorithm>

#include "lbm_internal.cuh"

namespace lbm {
namespace {

struct Ray {
    double px, py, pz, ex, ey, ez;
};

__host__ __device__ inline Ray point_ray(const double* bb, const double* org, double s, int i, int j, int k) {
    double x = org[0] + i * s;
    double y = org[1] + j * s;
    double z = org[2] + k * s;
    const double rayOffset = 0.02;
    double rayLength = bb[5] - bb[4];
    Ray r;
    r.px = x; r.py = y; r.pz = z + s / 2;
    r.ex = x; r.ey = y; r.ez = z + rayLength + 0.1;
    if (r.px == bb[0]) { r.px += rayOffset; r.ex += rayOffset; }
    if (r.px == bb[1]) { r.px -= rayOffset; r.ex -= rayOffset; }
    if (r.py == bb[2]) { r.py += rayOffset; r.ey += rayOffset; }
    if (r.py == bb[3]) { r.py -= rayOffset; r.ey -= rayOffset; }
    if (r.pz == bb[4]) { r.pz += rayOffset; }
    if (r.ez == bb[5]) { r.ez -= rayOffset; }
    return r;
}

__device__ __forceinline__ bool inside_tri(double x, double y, double z, const double* __restrict__ T) {
    double x1 = T[0], y1 = T[1], z1 = T[2];
    double x2 = T[3], y2 = T[4], z2 = T[5];
    double x3 = T[6], y3 = T[7], z3 = T[8];
    double dirX = 0.0, dirY = 0.0, dirZ = 1.0;
    double uX = x2 - x1, uY = y2 - y1, uZ = z2 - z1;
    double vX = x3 - x1, vY = y3 - y1, vZ = z3 - z1;
    double nX = uY * vZ - uZ * vY;
    double nY = uZ * vX - uX * vZ;
    double nZ = uX * vY - uY * vX;
    double nLengthSq = nX * nX + nY * nY + nZ * nZ;
    const double tol = 1e-16;
    if (nLengthSq < tol * tol) return false;
    double w0X = x - x1, w0Y = y - y1, w0Z = z - z1;
    double a = -(nX * w0X + nY * w0Y + nZ * w0Z);
    double b = nX * dirX + nY * dirY + nZ * dirZ;
    if (fabs(b) < tol) return false;
    double pos = a / b;
    double ix = x + pos * dirX;
    double iy = y + pos * dirY;
    double iz = z + pos * dirZ;
    double uu = uX * uX + uY * uY + uZ * uZ;
    double uv = uX * vX + uY * vY + uZ * vZ;
    double vv = vX * vX + vY * vY + vZ * vZ;
    double wX = ix - x1, wY = iy - y1, wZ = iz - z1;
    double wu = wX * uX + wY * uY + wZ * uZ;
    double wv = wX * vX + wY * vY + wZ * vZ;
    double D = uv * uv - uu * vv;
    double sb = (uv * wv - vv * wu) / D;
    if (sb < 0.0 || sb > 1.0) return false;
    double tb = (uv * wu - uu * wv) / D;
    if (tb < 0.0 || (sb + tb) > 1.0) return false;
    return true;
}

__device__ __forceinline__ int ray_hits(const Ray& r, const double* __restrict__ T) {
    const double threshold = 1e-16;
    double dx = r.ex - r.px, dy = r.ey - r.py, dz = r.ez - r.pz;
    double nx = T[9], ny = T[10], nz = T[11];
    double qx = T[0], qy = T[1], qz = T[2];
    double numerator = (qx - r.px) * nx + (qy - r.py) * ny + (qz - r.pz) * nz;
    double denominator = dx * nx + dy * ny + dz * nz;
    if (fabs(denominator) < threshold) return 0;
    double t = numerator / denominator;
    if (t >= 0.0 && t <= 1.0) {
        double ix = r.px + t * dx;
        double iy = r.py + t * dy;
        double iz = r.pz + t * dz;
        return inside_tri(ix, iy, iz, T) ? 1 : 0;
    }
    return 0;
}

// A margin of the xy extent about 1e8 times the rounding of the point-in-triangle
// test; -1: the triangle never counts, 1e30: no margin holds it.  It sorts the
// triangles, bounds the columns where tri_extent's own bound is larger, and gives
// the number of candidate tests that a call reports.
__device__ double cull_margin(const double* T, double zspan) {
    double uX = T[3] - T[0], uY = T[4] - T[1], uZ = T[5] - T[2];
    double vX = T[6] - T[0], vY = T[7] - T[1], vZ = T[8] - T[2];
    double nX = uY * vZ - uZ * vY;
    double nY = uZ * vX - uX * vZ;
    double nZ = uX * vY - uY * vX;
    double nLengthSq = nX * nX + nY * nY + nZ * nZ;
    if (nLengthSq < 1e-16 * 1e-16) return -1.0;
    if (fabs(nZ) < 1e-16) return -1.0;
    double nlen = sqrt(nLengthSq);
    double wX = vX - uX, wY = vY - uY, wZ = vZ - uZ;
    double L = sqrt(fmax(fmax(uX * uX + uY * uY + uZ * uZ, vX * vX + vY * vY + vZ * vZ), wX * wX + wY * wY + wZ * wZ));
    double cabs = 0.0;
    for (int k = 0; k < 9; ++k) cabs = fmax(cabs, fabs(T[k]));
    double shape = (L * L) / nlen;
    double m = 1e-7 * (L + zspan + cabs) * shape * shape * (nlen / fabs(nZ));
    if (!(m < 1e29)) return 1e30;
    return m;
}

// What every kernel of a call needs.
struct VoxParams {
    double bb[6];
    double org[3];
    double s, inv_s;
    double zspan;     // of cull_margin
    double span;      // bound of every coordinate difference of the tests
    double dz;        // ray length of an unadjusted ray
    double zabs;      // bound of |pz|, |ez|
    int nx, ny, nz;
    int kadj[2];      // the k whose ray ends are moved off the bounding box (-1: none)
    int exact_only;   // rays the column decisions do not describe: every pair is tested point by point
    int64_t ncol;
    int64_t ntri;
    int64_t cap;      // entries of the pair list
};

// Counters of one call.
struct VoxCounters {
    unsigned long long fluid, pairs;
    unsigned long long npair;  // pairs left to k_exact_pairs (may exceed the list)
    unsigned long long nglob, nwide;
};

__device__ __forceinline__ double column_x(const VoxParams& P, int i) {
    double x = P.org[0] + i * P.s;
    if (x == P.bb[0]) x += 0.02;
    if (x == P.bb[1]) x -= 0.02;
    return x;
}
__device__ __forceinline__ double column_y(const VoxParams& P, int j) {
    double y = P.org[1] + j * P.s;
    if (y == P.bb[2]) y += 0.02;
    if (y == P.bb[3]) y -= 0.02;
    return y;
}

// Difference bit field [k / 32][column]: point (c, k) is fluid when the XOR
// of bits 0 .. k of its column is 1.
__device__ __forceinline__ void flip(uint32_t* __restrict__ bits, const VoxParams& P, int64_t c, int k) {
    if (k < P.nz) atomicXor(bits + (int64_t)(k >> 5) * P.ncol + c, 1u << (k & 31));
}
__device__ __forceinline__ void flip_range(uint32_t* __restrict__ bits, const VoxParams& P, int64_t c, int k0, int k1) {
    flip(bits, P, c, k0);
    flip(bits, P, c, k1 + 1);
}

__device__ __forceinline__ bool exact_hit(const VoxParams& P, const double* T, int i, int j, int k) {
    return ray_hits(point_ray(P.bb, P.org, P.s, i, j, k), T) != 0;
}

// One triangle's FP64 constants for the column decisions, besides its 12 numbers.
struct TriConst {
    double nX, nY, nZ, inv_nZ;          // computed normal
    double uX, uY, uZ, vX, vY, vZ;      // edges
    double uu, uv, vv, inv_D;
    double E;                           // bound of the barycentric coordinates' rounding; < 0: decide nothing
    double inv_fz;                      // 1 / facet normal z
};

// Bound of the rounding of the barycentric coordinates, as the reference
// computes them, for any point of a column: an error eps * span in w moves
// the point on the computed plane by eps span L^2 / |nZ| along z, and that
// by a factor L / |n| in the coordinates; with shape = L^2 / |n| that is
// eps shape^2 (|n| / |nZ|) (span / L), times a small count of operations
// (< 30); 4e-12 is 36,000 eps.  L2: the larger squared edge at vertex 1
// (the third edge is at most twice as long); n2, nZ: the computed normal.
// In FP32 where nothing can underflow: the bound needs no digits (GB300's
// FP64 rate is 1/64 of FP32's).
__device__ __forceinline__ double barycentric_bound(const VoxParams& P, double L2, double n2, double nZ) {
    const float l2 = (float)L2, m2 = (float)n2;
    if (!(l2 > 1e-8f && l2 < 1e8f && m2 > 1e-20f))
        return 4e-12 * (L2 / n2 * L2) * (sqrt(n2) / fabs(nZ)) * (1.0 + P.span / sqrt(L2));
    return 4e-12f * (l2 * l2 / m2) * (sqrtf(m2) / fabsf((float)nZ)) * (1.0f + (float)P.span * rsqrtf(l2));
}

__device__ __forceinline__ TriConst tri_const(const VoxParams& P, const double* T) {
    TriConst c;
    c.uX = T[3] - T[0]; c.uY = T[4] - T[1]; c.uZ = T[5] - T[2];
    c.vX = T[6] - T[0]; c.vY = T[7] - T[1]; c.vZ = T[8] - T[2];
    c.nX = c.uY * c.vZ - c.uZ * c.vY;
    c.nY = c.uZ * c.vX - c.uX * c.vZ;
    c.nZ = c.uX * c.vY - c.uY * c.vX;
    c.inv_nZ = 1.0 / c.nZ;
    c.uu = c.uX * c.uX + c.uY * c.uY + c.uZ * c.uZ;
    c.uv = c.uX * c.vX + c.uY * c.vY + c.uZ * c.vZ;
    c.vv = c.vX * c.vX + c.vY * c.vY + c.vZ * c.vZ;
    c.inv_D = 1.0 / (c.uv * c.uv - c.uu * c.vv);
    const double n2 = c.nX * c.nX + c.nY * c.nY + c.nZ * c.nZ;
    c.E = barycentric_bound(P, fmax(c.uu, c.vv), n2, c.nZ);
    c.inv_fz = 1.0 / T[11];
    const double den = fabs(P.dz * T[11]);  // the reference rejects |den| < 1e-16
    if (!isfinite(c.E) || !(den > 2e-16) || !isfinite(c.inv_fz) || P.exact_only) c.E = -1.0;
    return c;
}

// Column (i, j) against triangle T: flips the column's parity where the ray
// of point k crosses T.  A pair that no bound decides goes to the pair list,
// tested point by point by k_exact_pairs.
__device__ __forceinline__ void column_pair(const VoxParams& P, const TriConst& t, const double* T, int32_t tri,
                                            int i, int j, double px, double py, uint32_t* __restrict__ bits,
                                            int2* __restrict__ list, VoxCounters* __restrict__ cnt) {
    const int64_t c = (int64_t)j * P.nx + i;
    bool undecided = t.E < 0.0;
    if (!undecided) {
        const double wX = px - T[0], wY = py - T[1];
        const double wZ = -(t.nX * wX + t.nY * wY) * t.inv_nZ;
        const double wu = wX * t.uX + wY * t.uY + wZ * t.uZ;
        const double wv = wX * t.vX + wY * t.vY + wZ * t.vZ;
        const double sb = (t.uv * wv - t.vv * wu) * t.inv_D;
        const double tb = (t.uv * wu - t.uu * wv) * t.inv_D;
        if (sb < -t.E || tb < -t.E || sb + tb > 1.0 + t.E) return;  // outside for every k
        undecided = !(sb > t.E && tb > t.E && sb + tb < 1.0 - t.E);
    }
    if (!undecided) {
        // 0 <= t <= 1 of the ray parameter: z* - dz <= pz(k) <= z*
        const double ax = (T[0] - px) * T[9], ay = (T[1] - py) * T[10];
        const double zs = T[2] + (ax + ay) * t.inv_fz;
        const double inv_s = P.inv_s;
        const double p0 = P.org[2] + 0.5 * P.s;
        const double kU = (zs - p0) * inv_s, kL = (zs - P.dz - p0) * inv_s;
        const double tol = (1e-12 * ((fabs(ax) + fabs(ay)) * fabs(t.inv_fz) + fabs(T[2]) + P.zabs)) * inv_s +
                           1e-12 * (fabs(kU) + fabs(kL) + P.nz);
        if (tol < 0.25) {
            // clamped: beyond the lattice only the side matters
            const double hiU = fmin(fmax(kU, -4.0), P.nz + 4.0), hiL = fmin(fmax(kL, -4.0), P.nz + 4.0);
            const int aU = (int)ceil(hiU - tol), aL = (int)floor(hiL + tol);
            const bool ambU = (double)aU <= hiU + tol, ambL = (double)aL >= hiL - tol;
            const int k0 = max(aL + 1, 0), k1 = min(aU - 1, P.nz - 1);
            if (k0 <= k1) flip_range(bits, P, c, k0, k1);
            // the k on a bound and the k whose ray is moved: the reference's own test
            const int special[4] = {ambU ? aU : -1, ambL ? aL : -1, P.kadj[0], P.kadj[1]};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int k = special[m];
                if (k < 0 || k >= P.nz) continue;
                bool seen = false;
                for (int n = 0; n < m; ++n) seen |= special[n] == k;
                if (seen) continue;
                if (exact_hit(P, T, i, j, k) != (k >= k0 && k <= k1)) flip_range(bits, P, c, k, k);
            }
            return;
        }
    }
    const unsigned long long slot = atomicAdd(&cnt->npair, 1ull);
    if (slot < (unsigned long long)P.cap) list[slot] = make_int2(tri, (int)c);  // else: a second run with room for all
}

// A triangle's columns: the lattice range of its xy extent widened by the
// distance within which rounding can matter.  A point d outside an edge has
// a barycentric coordinate at least d / (2 L) outside [0, 1] (no height of
// the triangle exceeds 2 L), so beyond 4 L E no test passes.  `pairs` counts
// the columns of cull_margin's wider extent: the tests this replaces.
struct TriExtent {
    double x0, x1, y0, y1;
    int i0, i1, j0, j1;
    int kind;  // 0: never counts, 1: columns i0..i1, j0..j1, 2: global list
    unsigned pairs;
};

// Lattice indices whose column coordinate may lie in [a, b] (one more on
// either side: the coordinates' rounding).
__device__ __forceinline__ bool index_range(double a, double b, double org, double inv_s, int n, int& k0, int& k1) {
    // clamp in FP64 before converting: margins can be far outside int range
    const double f0 = fmax(floor((a - org) * inv_s) - 1.0, 0.0), f1 = fmin(ceil((b - org) * inv_s) + 1.0, n - 1.0);
    if (!(f0 <= f1)) return false;
    k0 = (int)f0;
    k1 = (int)f1;
    return true;
}

__device__ __forceinline__ TriExtent tri_extent(const VoxParams& P, const double* T) {
    TriExtent e{};
    e.i1 = e.j1 = -1;
    const double m = cull_margin(T, P.zspan);
    e.kind = m < 0.0 ? 0 : (m > 1e29 ? 2 : 1);
    if (e.kind != 1) return e;
    const double xl = fmin(fmin(T[0], T[3]), T[6]), xh = fmax(fmax(T[0], T[3]), T[6]);
    const double yl = fmin(fmin(T[1], T[4]), T[7]), yh = fmax(fmax(T[1], T[4]), T[7]);
    if (!index_range(xl - m, xh + m, P.org[0], P.inv_s, P.nx, e.i0, e.i1) ||
        !index_range(yl - m, yh + m, P.org[1], P.inv_s, P.ny, e.j0, e.j1)) {
        e.i0 = e.j0 = 0;
        e.i1 = e.j1 = -1;
        return e;
    }
    unsigned ni = 0, nj = 0;
    for (int i = e.i0; i <= e.i1; ++i) {
        const double x = column_x(P, i);
        ni += x >= xl - m && x <= xh + m;
    }
    for (int j = e.j0; j <= e.j1; ++j) {
        const double y = column_y(P, j);
        nj += y >= yl - m && y <= yh + m;
    }
    e.pairs = ni * nj;
    // A facet normal so flat in z that the reference rejects the plane crossing
    // of every ray (its denominator, the ray's length times the normal's z, is
    // below 1e-16; a ray's ends move by 0.02 each at most): counted, no columns.
    // Vertical walls whose vertices are rounded out of the vertical: column_pair
    // decides none of their pairs.
    if ((fabs(P.dz) + 0.1 + 1e-12 * P.zabs) * fabs(T[11]) < 1e-16 && isfinite(T[9]) && isfinite(T[10])) {
        e.i0 = e.j0 = 0;
        e.i1 = e.j1 = -1;
        return e;
    }
    const double uX = T[3] - T[0], uY = T[4] - T[1], uZ = T[5] - T[2];
    const double vX = T[6] - T[0], vY = T[7] - T[1], vZ = T[8] - T[2];
    const double nX = uY * vZ - uZ * vY, nY = uZ * vX - uX * vZ, nZ = uX * vY - uY * vX;
    const double L2 = fmax(uX * uX + uY * uY + uZ * uZ, vX * vX + vY * vY + vZ * vZ);
    const double t = 4.0 * (double)sqrtf((float)L2) * barycentric_bound(P, L2, nX * nX + nY * nY + nZ * nZ, nZ);
    const double w = t < m ? t : m;  // (a NaN or infinite bound keeps m)
    e.x0 = xl - w; e.x1 = xh + w;
    e.y0 = yl - w; e.y1 = yh + w;
    if (!index_range(e.x0, e.x1, P.org[0], P.inv_s, P.nx, e.i0, e.i1) ||
        !index_range(e.y0, e.y1, P.org[1], P.inv_s, P.ny, e.j0, e.j1)) {
        e.i0 = e.j0 = 0;
        e.i1 = e.j1 = -1;
    }
    return e;
}

__device__ __forceinline__ void add_pairs(unsigned long long pairs, VoxCounters* __restrict__ cnt) {
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_down_sync(0xffffffffu, pairs, o);
    if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(&cnt->pairs, pairs);
}

// One thread a triangle: classification and, for extents of up to
// kWideColumns columns (a mesh about as fine as the lattice), its columns;
// wider ones go to the wide list.
constexpr int kWideColumns = 32;
struct WideTri {
    TriExtent e;
    int32_t tri;
};
__global__ void __launch_bounds__(128, 4) k_tri_columns(const VoxParams P, const double* __restrict__ tri,
                                                     uint32_t* __restrict__ bits, int2* __restrict__ list,
                                                     int32_t* __restrict__ glob, WideTri* __restrict__ wide,
                                                        VoxCounters* __restrict__ cnt) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long pairs = 0;
    if (t < P.ntri) {
        const double* T = tri + 12 * t;
        const TriExtent e = tri_extent(P, T);
        pairs = e.pairs;
        const int64_t n = (int64_t)(e.i1 - e.i0 + 1) * (e.j1 - e.j0 + 1);
        if (e.kind == 2) {
            glob[atomicAdd(&cnt->nglob, 1ull)] = (int32_t)t;
        } else if (n > kWideColumns) {
            const unsigned long long w = atomicAdd(&cnt->nwide, 1ull);
            wide[w].e = e;
            wide[w].tri = (int32_t)t;
        } else if (n > 0) {
            TriConst k;
            bool have = false;
            for (int j = e.j0; j <= e.j1; ++j) {
                const double yy = column_y(P, j);
                if (yy < e.y0 || yy > e.y1) continue;
                for (int i = e.i0; i <= e.i1; ++i) {
                    const double xx = column_x(P, i);
                    if (xx < e.x0 || xx > e.x1) continue;
                    if (!have) { k = tri_const(P, T); have = true; }
                    column_pair(P, k, T, (int32_t)t, i, j, xx, yy, bits, list, cnt);
                }
            }
        }
    }
    add_pairs(pairs, cnt);
}

// The wide list: one thread a column, a grid row a triangle (one thread
// walked the 576 columns of a cap's facet in 1 ms, one after another).
__global__ void __launch_bounds__(128) k_wide_columns(const VoxParams P, const double* __restrict__ tri,
                                                      uint32_t* __restrict__ bits, int2* __restrict__ list,
                                                      const WideTri* __restrict__ wide,
                                                      VoxCounters* __restrict__ cnt) {
    const unsigned long long nwide = cnt->nwide;
    for (unsigned long long w = blockIdx.y; w < nwide; w += gridDim.y) {
        const TriExtent e = wide[w].e;
        const int nc = e.i1 - e.i0 + 1;
        const int64_t n = (int64_t)nc * (e.j1 - e.j0 + 1);
        int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (c >= n) continue;
        const int32_t t = wide[w].tri;
        const double* T = tri + 12 * (int64_t)t;
        const TriConst k = tri_const(P, T);
        for (; c < n; c += (int64_t)gridDim.x * blockDim.x) {
            const int i = e.i0 + (int)(c % nc), j = e.j0 + (int)(c / nc);
            const double xx = column_x(P, i), yy = column_y(P, j);
            if (xx < e.x0 || xx > e.x1 || yy < e.y0 || yy > e.y1) continue;
            column_pair(P, k, T, t, i, j, xx, yy, bits, list, cnt);
        }
    }
}

// The pairs no bound decided: one warp a pair, the reference's test for
// every k (32 consecutive k a pass: their results are one word of the field).
__global__ void __launch_bounds__(128) k_exact_pairs(const VoxParams P, const double* __restrict__ tri,
                                                     uint32_t* __restrict__ bits, const int2* __restrict__ list,
                                                     const VoxCounters* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    if (cnt->npair > (unsigned long long)P.cap) return;  // the list is not whole: all of it in the second run
    const unsigned long long n = cnt->npair;
    const int nw = (P.nz + 31) / 32;
    const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x / 32);
    for (unsigned long long e = (unsigned long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; e < n * nw;
         e += warps) {
        const int2 p = list[e / nw];
        const int kw = (int)(e % nw), k = kw * 32 + lane;
        const double* T = tri + 12 * (int64_t)p.x;
        const bool hit = k < P.nz && exact_hit(P, T, p.y % P.nx, p.y / P.nx, k);
        const uint32_t h = __ballot_sync(0xffffffffu, hit);
        if (lane == 0 && h) {
            uint32_t* w = bits + (int64_t)kw * P.ncol + p.y;
            const uint32_t d = h ^ (h << 1);
            if (d) atomicXor(w, d);
            if ((h >> 31) && kw + 1 < nw) atomicXor(w + P.ncol, 1u);
        }
    }
}

// The field's running XOR into the mask: thread (column, word of 32 k), the
// parity below the word from the population counts of the words below it;
// the triangles of the global list are tested here point by point.
__global__ void __launch_bounds__(128) k_mask(const VoxParams P, const double* __restrict__ tri,
                                              const uint32_t* __restrict__ bits, const int32_t* __restrict__ glob,
                                              uint8_t* __restrict__ mask, VoxCounters* __restrict__ cnt) {
    if (cnt->npair > (unsigned long long)P.cap) return;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned fluid = 0;
    uint32_t below = 0;  // XOR of the words below kw
    int w = 0;
    for (int kw = blockIdx.y; c < P.ncol && kw < (P.nz + 31) / 32; kw += gridDim.y) {
        for (; w < kw; ++w) below ^= bits[(int64_t)w * P.ncol + c];
        uint32_t v = bits[(int64_t)kw * P.ncol + c];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) v ^= v << d;
        if (__popc(below) & 1) v = ~v;
        const int kn = min(32, P.nz - kw * 32);
        const unsigned long long ng = cnt->nglob;
        if (ng) {
            const int i = (int)(c % P.nx), j = (int)(c / P.nx);
            for (int b = 0; b < kn; ++b) {
                const Ray r = point_ray(P.bb, P.org, P.s, i, j, kw * 32 + b);
                uint32_t h = 0;
                for (unsigned long long q = 0; q < ng; ++q) h ^= (uint32_t)ray_hits(r, tri + 12 * (int64_t)glob[q]);
                v ^= h << b;
            }
        }
        if (kn < 32) v &= (1u << kn) - 1u;
        fluid += __popc(v);
        uint8_t* m = mask + (int64_t)kw * 32 * P.ncol + c;
        for (int b = 0; b < kn; ++b) m[b * P.ncol] = (uint8_t)((v >> b) & 1u);
    }
    fluid = __reduce_add_sync(0xffffffffu, fluid);
    if ((threadIdx.x & 31) == 0 && fluid) atomicAdd(&cnt->fluid, (unsigned long long)fluid);
}

#define VOX_CHECK(call)                                                        \
    do {                                                                       \
        cudaError_t _e = (call);                                               \
        if (_e != cudaSuccess) {                                               \
            if (err) *err = std::string(#call) + ": " + cudaGetErrorString(_e); \
            return _e;                                                         \
        }                                                                      \
    } while (0)

}  // namespace

cudaError_t voxelize_device(const double* tri, int64_t ntri, const double bbox[6], const double origin[3],
                            double spacing, const int dims[3], uint8_t* mask, VoxResult* res, cudaStream_t st,
                            std::string* err) {
    VoxParams P{};
    for (int q = 0; q < 6; ++q) P.bb[q] = bbox[q];
    for (int q = 0; q < 3; ++q) P.org[q] = origin[q];
    P.s = spacing;
    P.inv_s = 1.0 / spacing;
    P.nx = dims[0]; P.ny = dims[1]; P.nz = dims[2];
    P.ncol = (int64_t)P.nx * P.ny;
    P.ntri = ntri;
    if (P.ncol > 0x7fffffffLL || ntri > 0x7fffffffLL) {
        if (err) *err = "lattice too large for the voxelizer grid";
        return cudaErrorInvalidValue;
    }
    P.zspan = (bbox[5] - bbox[4]) + 1.0 + spacing;
    // bounds of the coordinates a test meets
    double far = 0.0;
    for (int q = 0; q < 6; ++q) far = std::fmax(far, std::fabs(bbox[q]));
    for (int q = 0; q < 3; ++q)
        far = std::fmax(far, std::fmax(std::fabs(origin[q]), std::fabs(origin[q] + dims[q] * spacing)));
    P.dz = (bbox[5] - bbox[4]) + 0.1 - 0.5 * spacing;
    P.zabs = far + std::fabs(bbox[5] - bbox[4]) + spacing + 1.0;
    P.span = 4.0 * P.zabs;
    // the k whose ray start or end lies on the bounding box (point_ray moves
    // it): at most one each on an ordinary lattice
    P.kadj[0] = P.kadj[1] = -1;
    P.exact_only = !(P.dz > 1e-6 * P.zabs) || !std::isfinite(P.span);
    double last = -INFINITY;
    int nstart = 0, nend = 0;
    for (int k = 0; k < P.nz; ++k) {
        const double z = origin[2] + k * spacing;
        const double pz = z + spacing / 2, ez = z + (bbox[5] - bbox[4]) + 0.1;
        if (pz == bbox[4]) { P.kadj[0] = k; ++nstart; }
        if (ez == bbox[5]) { P.kadj[1] = k; ++nend; }
        if (!(pz > last)) P.exact_only = 1;
        last = pz;
    }
    if (nstart > 1 || nend > 1) P.exact_only = 1;

    const int nw = (int)ceil_div(P.nz, 32);
    const int64_t tri_alloc = ntri > 0 ? ntri : 1;
    VoxCounters got{};
    // one run with room for `cap` undecided pairs; triangles, mask, counters,
    // bit field, pair, global and wide lists in one allocation
    auto run = [&](int64_t cap) -> cudaError_t {
        P.cap = cap;
        const int64_t npts = P.ncol * P.nz;
        size_t at = 0;
        auto place = [&](size_t bytes) {
            const size_t o = at;
            at = (at + bytes + 255) / 256 * 256;
            return o;
        };
        const size_t o_cnt = place(sizeof(VoxCounters)), b_bits = sizeof(uint32_t) * (size_t)nw * P.ncol;
        const size_t o_bits = place(b_bits), o_list = place(sizeof(int2) * (size_t)cap);
        const size_t o_glob = place(sizeof(int32_t) * tri_alloc), o_wide = place(sizeof(WideTri) * tri_alloc);
        const size_t o_tri = place(sizeof(double) * 12 * tri_alloc), o_mask = place((size_t)npts);
        unsigned char* base = nullptr;
        VOX_CHECK(cudaMallocAsync(&base, at, st));
        VoxCounters* cnt = reinterpret_cast<VoxCounters*>(base + o_cnt);
        uint32_t* bits = reinterpret_cast<uint32_t*>(base + o_bits);
        int2* list = reinterpret_cast<int2*>(base + o_list);
        int32_t* glob = reinterpret_cast<int32_t*>(base + o_glob);
        WideTri* wide = reinterpret_cast<WideTri*>(base + o_wide);
        double* d_tri = reinterpret_cast<double*>(base + o_tri);
        uint8_t* d_mask = base + o_mask;
        auto body = [&]() -> cudaError_t {
            VOX_CHECK(cudaMemsetAsync(base, 0, o_bits + b_bits, st));
            if (ntri > 0) {
                VOX_CHECK(cudaMemcpyAsync(d_tri, tri, sizeof(double) * 12 * ntri, cudaMemcpyHostToDevice, st));
                k_tri_columns<<<(unsigned)ceil_div(ntri, 128), 128, 0, st>>>(P, d_tri, bits, list, glob, wide, cnt);
                k_wide_columns<<<dim3(8, 304), 128, 0, st>>>(P, d_tri, bits, list, wide, cnt);
                k_exact_pairs<<<608, 128, 0, st>>>(P, d_tri, bits, list, cnt);
                VOX_CHECK(cudaGetLastError());
            }
            k_mask<<<dim3((unsigned)ceil_div(P.ncol, 128), (unsigned)std::min(nw, 4096)), 128, 0, st>>>(
                P, d_tri, bits, glob, d_mask, cnt);
            VOX_CHECK(cudaGetLastError());
            // the caller's pages are touched while the kernels run: a copy
            // into pages the process has never written ran at 1.1 GB/s
            for (int64_t k = 0; k < npts; k += 4096) reinterpret_cast<volatile uint8_t*>(mask)[k] = 0;
            VOX_CHECK(cudaMemcpyAsync(&got, cnt, sizeof(got), cudaMemcpyDeviceToHost, st));
            VOX_CHECK(cudaMemcpyAsync(mask, d_mask, (size_t)npts, cudaMemcpyDeviceToHost, st));
            VOX_CHECK(cudaStreamSynchronize(st));
            return cudaSuccess;
        };
        const cudaError_t e = body();
        cudaFreeAsync(base, st);
        return e;
    };
    cudaError_t e = run(std::max<int64_t>(4 * tri_alloc, 65536));
    if (e == cudaSuccess && got.npair > (unsigned long long)P.cap) e = run((int64_t)got.npair);
    if (e != cudaSuccess) return e;
    res->fluid = (int64_t)got.fluid;
    res->tests = (int64_t)(got.pairs + got.nglob * (unsigned long long)P.ncol) * P.nz;
    return cudaSuccess;
}

}  // namespace lbm
