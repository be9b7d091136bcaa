// Geometry set-up on the device: node classes, boundary-node list,
// next-to-wall nodes, bulk segments and wall normals.
//
// Replaces the reference's pointer-graph construction:
//   findBoundaryPoints          ComplexGeometry.cpp:1259-1300
//   classifyBoundaryPoints      ComplexGeometry.cpp:1369-1429 (plane rules instead of PV coordinates)
//   SubDomain::CreateNodes      Subdomain.cpp:91-169 (Boundary vs Node by list membership)
//   Connectivity                Subdomain.cpp:173-197 (-> per-link "missing" bit masks)
//   IdentifyNextToWallLattices  Subdomain.cpp:201-218
//   calculateBoundaryNormals    Subdomain.cpp:224-370
// The reference links one heap object per node with shared_ptr neighbours
// and finds list membership by linear search (Utility.cpp:18-33, O(A*B));
// here a node is one class byte in a dense box and the boundary/next-to-wall
// nodes form one compact, index-sorted list built by a scan.
//
// Compiled with --fmad=false: a triangle's normal, area and centroid are rounded
// as the reference rounds them.  The sums over the triangles are not: they use
// fused multiply-adds, one reciprocal for four distances and parts (k_normals).
#include <algorithm>

#include "lbm_internal.cuh"
#include "setup.cuh"

namespace lbm {
namespace {

template <int Q>
__global__ void k_boundary(const uint8_t* __restrict__ mask, int nx, int ny, int nz, uint8_t* __restrict__ cls) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t npts = (int64_t)nx * ny * nz;
    if (n >= npts) return;
    if (!mask[n]) { cls[n] = CLS_SOLID; return; }
    const int i = (int)(n % nx), j = (int)((n / nx) % ny), k = (int)(n / ((int64_t)nx * ny));
    bool b = false;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        int a = i + Lat<Q>::cx(q), bb = j + Lat<Q>::cy(q), c = k + Lat<Q>::cz(q);
        if (a < 0 || a >= nx || bb < 0 || bb >= ny || c < 0 || c >= nz) { b = true; break; }
        if (!mask[((int64_t)c * ny + bb) * nx + a]) { b = true; break; }
    }
    cls[n] = b ? CLS_WALL : CLS_FLUID;
}

// Extreme fluid layer per axis: ext[0..2] = min index, ext[3..5] = max index.
__global__ void k_extent(const uint8_t* __restrict__ mask, int nx, int ny, int nz, int* __restrict__ ext) {
    // warps reduce before their atomics (6 words for the whole lattice)
    const int64_t npts = (int64_t)nx * ny * nz;
    int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-1, -1, -1};
    for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < npts; n += (int64_t)gridDim.x * blockDim.x) {
        if (!mask[n]) continue;
        const int c[3] = {(int)(n % nx), (int)((n / nx) % ny), (int)(n / ((int64_t)nx * ny))};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = min(lo[d], c[d]);
            hi[d] = max(hi[d], c[d]);
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int l = __reduce_min_sync(0xffffffffu, lo[d]), h = __reduce_max_sync(0xffffffffu, hi[d]);
        if ((threadIdx.x & 31) == 0 && h >= 0) {
            atomicMin(ext + d, l);
            atomicMax(ext + 3 + d, h);
        }
    }
}

struct Rules {
    int n;
    int axis[LBM_MAX_BC];
    int plane[LBM_MAX_BC];
    int region[LBM_MAX_BC];
    double coord[LBM_MAX_BC], tol[LBM_MAX_BC], lo[LBM_MAX_BC][2], hi[LBM_MAX_BC][2];
    double org[3];
    double s;
};

// Plane rules match a lattice index; region rules match coordinates the way
// classifyBoundaryPoints does (ComplexGeometry.cpp:1380-1407; the reference
// compares in long double, here in FP64).  First match wins.
// The class byte records 3 + r (capped at 127 for r >= 124); bcidx holds r.
__global__ void k_classify(uint8_t* __restrict__ cls, int16_t* __restrict__ bcidx, int nx, int ny, int64_t npts,
                           Rules R) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts || cls[n] != CLS_WALL) return;
    const int idx[3] = {(int)(n % nx), (int)((n / nx) % ny), (int)(n / ((int64_t)nx * ny))};
    for (int r = 0; r < R.n; ++r) {
        const int a = R.axis[r];
        bool hit;
        if (!R.region[r]) {
            hit = idx[a] == R.plane[r];
        } else {
            const double x[3] = {R.org[0] + idx[0] * R.s, R.org[1] + idx[1] * R.s, R.org[2] + idx[2] * R.s};
            const int t1 = a == 0 ? 1 : 0, t2 = a == 2 ? 1 : 2;
            hit = fabs(x[a] - R.coord[r]) <= R.tol[r] && R.lo[r][0] < x[t1] && x[t1] < R.hi[r][0] &&
                  R.lo[r][1] < x[t2] && x[t2] < R.hi[r][1];
        }
        if (hit) {
            cls[n] = (uint8_t)(CLS_BC0 + (r < 124 ? r : 124));
            bcidx[n] = (int16_t)r;
            return;
        }
    }
}

template <int Q>
__global__ void k_next_to_wall(uint8_t* __restrict__ cls, int nx, int ny, int nz) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t npts = (int64_t)nx * ny * nz;
    if (n >= npts || cls[n] != CLS_FLUID) return;
    // an interior fluid node has all Q neighbours inside the box
    const int64_t nxy = (int64_t)nx * ny;
    bool nw = false;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        int64_t m = n + Lat<Q>::cx(q) + Lat<Q>::cy(q) * (int64_t)nx + Lat<Q>::cz(q) * nxy;
        if ((cls[m] & CLS_MASK) == CLS_WALL) nw = true;
    }
    if (nw) cls[n] = CLS_FLUID | CLS_NW_BIT;
}

// Boundary-list membership, split in two: next-to-wall nodes (nwflag) and
// the other boundary-list nodes (wall and boundary-condition nodes, oflag).
__global__ void k_flag_special(const uint8_t* __restrict__ cls, int64_t npts, int64_t* __restrict__ oflag,
                               int64_t* __restrict__ nwflag) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts) return;
    const uint8_t c = cls[n];
    const bool nw = (c & CLS_NW_BIT) != 0;
    oflag[n] = (!nw && (c & CLS_MASK) >= CLS_WALL) ? 1 : 0;
    nwflag[n] = nw ? 1 : 0;
}

// Boundary-list position: next-to-wall nodes first, in point order, so that
// a next-to-wall node's list entry s is also its wall-shear-stress index;
// then the other boundary-list nodes in point order.
__global__ void k_special_pos(int64_t* __restrict__ flag, int64_t* __restrict__ pos,
                              const int64_t* __restrict__ nwflag, const int64_t* __restrict__ nwpos, int64_t nnw,
                              int64_t npts) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts) return;
    if (nwflag[n]) {
        flag[n] = 1;
        pos[n] = nwpos[n];
    } else if (flag[n]) {
        pos[n] = nnw + pos[n];
    }
}

__global__ void k_scatter(const int64_t* __restrict__ flag, const int64_t* __restrict__ pos, int64_t npts,
                          int64_t* __restrict__ out) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts || !flag[n]) return;
    out[pos[n]] = n;
}

template <int Q>
__global__ void k_special_info(const int64_t* __restrict__ sp_pt, int64_t nsp, const uint8_t* __restrict__ cls,
                               const int64_t* __restrict__ nwpos, int nx, int ny, int nz,
                               const int16_t* __restrict__ bcidx, uint32_t* __restrict__ miss,
                               uint8_t* __restrict__ spc, int32_t* __restrict__ spnw, int32_t* __restrict__ spbc,
                               double* __restrict__ prof, ProfileSpec ps) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsp) return;
    const int64_t n = sp_pt[s];
    const int i = (int)(n % nx), j = (int)((n / nx) % ny), k = (int)(n / ((int64_t)nx * ny));
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        int a = i + Lat<Q>::cx(q), b = j + Lat<Q>::cy(q), c = k + Lat<Q>::cz(q);
        bool missing = (a < 0 || a >= nx || b < 0 || b >= ny || c < 0 || c >= nz) ||
                       cls[((int64_t)c * ny + b) * nx + a] == CLS_SOLID;
        if (missing) m |= 1u << q;
    }
    miss[s] = m;
    const uint8_t c = cls[n];
    spc[s] = c & CLS_MASK;
    spnw[s] = (c & CLS_NW_BIT) ? (int32_t)nwpos[n] : -1;
    const bool is_bc = (c & CLS_MASK) >= CLS_BC0;
    const int b = is_bc ? (int)bcidx[n] : -1;
    spbc[s] = b;
    double p = 0.0;
    if (is_bc && b < ps.n) {
        if (ps.profile[b] == 0) {
            p = 1.0;
        } else {
            // same expression as the reference harness / oracle profile factor
            const double xyz[3] = {ps.org[0] + i * ps.s, ps.org[1] + j * ps.s, ps.org[2] + k * ps.s};
            const int a = ps.axis[b];
            const int t1 = a == 0 ? 1 : 0, t2 = a == 2 ? 1 : 2;
            double d1 = xyz[t1] - ps.c1[b], d2 = xyz[t2] - ps.c2[b];
            double v = 1.0 - (d1 * d1 + d2 * d2) / (ps.R[b] * ps.R[b]);
            p = v > 0.0 ? v : 0.0;
        }
    }
    prof[s] = p;
}

__global__ void k_active_flags(const uint8_t* __restrict__ cls, int64_t npts, int64_t* __restrict__ flag) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts) return;
    flag[n] = cls[n] != CLS_SOLID ? 1 : 0;
}

// Per active node: index maps.
__global__ void k_active_index(const int64_t* __restrict__ flag, const int64_t* __restrict__ pos, int64_t npts,
                               int32_t* __restrict__ act_idx, int64_t* __restrict__ act_pt) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts) return;
    const bool f = flag[n] != 0;
    act_idx[n] = f ? (int32_t)pos[n] : -1;
    if (f) act_pt[pos[n]] = n;
}

// Per active node: the step kernel's packed word
// (segment | special << 31 | missing mask << 32 | class << 59 | next-to-wall << 63).
template <int Q>
__global__ void k_active_word(const int64_t* __restrict__ act_pt, int64_t nact, const int64_t* __restrict__ spflag,
                              const int64_t* __restrict__ sppos, const uint8_t* __restrict__ cls, int nx, int ny,
                              int nz, const int32_t* __restrict__ seg_of_act, uint64_t* __restrict__ act_word,
                              int32_t* __restrict__ sp_of_act) {
    const int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= nact) return;
    const int64_t n = act_pt[a];
    const int i = (int)(n % nx), j = (int)((n / nx) % ny), k = (int)(n / ((int64_t)nx * ny));
    uint64_t miss = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        int x = i + Lat<Q>::cx(q), y = j + Lat<Q>::cy(q), z = k + Lat<Q>::cz(q);
        bool m = (x < 0 || x >= nx || y < 0 || y >= ny || z < 0 || z >= nz) ||
                 cls[((int64_t)z * ny + y) * nx + x] == CLS_SOLID;
        if (m) miss |= 1ull << q;
    }
    const uint8_t c = cls[n];
    const bool sp = spflag[n] != 0;
    act_word[a] = (uint64_t)(uint32_t)seg_of_act[a] | ((uint64_t)sp << 31) | (miss << 32) |
                  ((uint64_t)((c & CLS_MASK) < CLS_BC0 ? (c & CLS_MASK) : CLS_BC0) << 59) |
                  ((uint64_t)((c & CLS_NW_BIT) ? 1 : 0) << 63);
    sp_of_act[a] = sp ? (int32_t)sppos[n] : -1;
}

// Per triangle: unit normal times area, and centroid (Subdomain.cpp:244-267).
constexpr int kTriWeight = 6;
__global__ void k_tri_weights(const double* __restrict__ tri, int64_t ntri, double* __restrict__ tw) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    const double* T = tri + 12 * t;
    double ux = T[3] - T[0], uy = T[4] - T[1], uz = T[5] - T[2];
    double vx = T[6] - T[0], vy = T[7] - T[1], vz = T[8] - T[2];
    double nx = uy * vz - uz * vy;
    double ny = uz * vx - ux * vz;
    double nz = ux * vy - uy * vx;
    double norm = sqrt(nx * nx + ny * ny + nz * nz);
    if (norm > 0) { nx /= norm; ny /= norm; nz /= norm; }
    double area = 0.5 * norm;
    double* o = tw + kTriWeight * t;
    o[0] = nx * area; o[1] = ny * area; o[2] = nz * area;
    o[3] = (T[0] + T[3] + T[6]) / 3.0;
    o[4] = (T[1] + T[4] + T[7]) / 3.0;
    o[5] = (T[2] + T[5] + T[8]) / 3.0;
}

// 1 / p for p whose exponent is well inside the range: the hardware's estimate
// (20 bits), then r (1 + e + e^2) with e = 1 - p r, what is left being e^3.
__device__ __forceinline__ double reciprocal(double p) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(p));
    const double e = __fma_rn(-p, r, 1.0);
    return __fma_rn(r, __fma_rn(e, e, e), r);
}

// Weighted normals: the sum over all triangles of normal area / distance^2 at
// each point.  Bound by the FP64 pipe (two operations a cycle and SM), so the
// loop is FP64 multiply-adds and one reciprocal for four triangles' squared
// distances: 1/d_0 = d_1 (d_2 d_3) / (d_0 d_1 d_2 d_3) and so on, 12 operations
// a (point, triangle) pair where a division each made it about 30.  The few
// roundings more a term are random and the sums shorter: against the same sum
// with pairwise rounding the normals' error went from 1.8e-15 to 5e-16.  A product beyond the
// mid-range of exponents (a point on a centroid) takes the divisions.
// Triangles are split over grid.y so that the blocks fill the SMs evenly;
// k_normals_sum adds the parts in order.  30k points x
// 13.9k triangles: 21.5 -> 9.4 ms.
constexpr int kNormThreads = 128;
constexpr int kNormTile = 256;

__global__ void __launch_bounds__(kNormThreads) k_normals(const double* __restrict__ tw, int64_t ntri, int64_t per,
                                                         const int64_t* __restrict__ pts, int64_t npts, int nx,
                                                         int ny, double ox, double oy, double oz, double s,
                                                         double* __restrict__ out) {
    __shared__ __align__(16) double tile[kNormTile * kTriWeight];
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double x = 0, y = 0, z = 0;
    if (p < npts) {
        const int64_t n = pts[p];
        const int i = (int)(n % nx), j = (int)((n / nx) % ny), k = (int)(n / ((int64_t)nx * ny));
        x = ox + i * s; y = oy + j * s; z = oz + k * s;
    }
    double n0 = 0.0, n1 = 0.0, n2 = 0.0;
    const int64_t begin = blockIdx.y * per, end = begin + per < ntri ? begin + per : ntri;
    for (int64_t t0 = begin; t0 < end; t0 += kNormTile) {
        const int cnt = (int)min((int64_t)kNormTile, end - t0), cnt4 = (cnt + 3) / 4 * 4;
        __syncthreads();
        for (int e = threadIdx.x; e < cnt * kTriWeight; e += blockDim.x) tile[e] = tw[kTriWeight * t0 + e];
        // the last four are filled up with weightless copies of the last triangle
        if ((int)threadIdx.x < kTriWeight * (cnt4 - cnt)) {
            const int f = threadIdx.x % kTriWeight;
            tile[cnt * kTriWeight + threadIdx.x] = f < 3 ? 0.0 : tw[kTriWeight * (t0 + cnt - 1) + f];
        }
        __syncthreads();
        for (int t = 0; t < cnt4; t += 4) {
            const double2* o2 = reinterpret_cast<const double2*>(tile + kTriWeight * t);
            double o[4][kTriWeight], d[4], w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double2 v = o2[3 * u + k];
                    o[u][2 * k] = v.x;
                    o[u][2 * k + 1] = v.y;
                }
                const double dx = x - o[u][3], dy = y - o[u][4], dz = z - o[u][5];
                d[u] = __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
            }
            const double d01 = d[0] * d[1], d23 = d[2] * d[3], prod = d01 * d23;
            // exponent of the product in [-700, 700]
            if ((uint32_t)__double2hiint(prod) - (323u << 20) < (1400u << 20)) {
                const double r = reciprocal(prod), r01 = r * d23, r23 = r * d01;
                w[0] = r01 * d[1];
                w[1] = r01 * d[0];
                w[2] = r23 * d[3];
                w[3] = r23 * d[2];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    n0 = __fma_rn(o[u][0], w[u], n0);
                    n1 = __fma_rn(o[u][1], w[u], n1);
                    n2 = __fma_rn(o[u][2], w[u], n2);
                }
            } else {
                for (int u = 0; u < 4 && t + u < cnt; ++u) {
                    n0 += tile[kTriWeight * (t + u)] / d[u];
                    n1 += tile[kTriWeight * (t + u) + 1] / d[u];
                    n2 += tile[kTriWeight * (t + u) + 2] / d[u];
                }
            }
        }
    }
    if (p < npts) {
        double* dst = out + 3 * npts * blockIdx.y;
        dst[p] = n0;
        dst[npts + p] = n1;
        dst[2 * npts + p] = n2;
    }
}

// The parts' sum and its direction, into out [3][npts].
__global__ void k_normals_sum(const double* __restrict__ part, int parts, int64_t npts, double* out) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npts) return;
    double n[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < parts; ++k)
        for (int d = 0; d < 3; ++d) n[d] += part[(3 * (int64_t)k + d) * npts + p];
    const double norm = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    for (int d = 0; d < 3; ++d) out[d * npts + p] = norm > 0 ? n[d] / norm : n[d];
}

__global__ void k_scatter_normals(const double* __restrict__ part, const int64_t* __restrict__ idx, int64_t m, int64_t nn,
                                  double* __restrict__ n) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    for (int d = 0; d < 3; ++d) n[d * nn + idx[k]] = part[d * m + k];
}

__global__ void k_normals_float(const double* __restrict__ n, int64_t nn, int64_t stride, float* __restrict__ out) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= stride) return;
    for (int d = 0; d < 3; ++d) out[d * stride + k] = k < nn ? (float)n[d * nn + k] : 0.f;
}

inline unsigned blocks(int64_t n, int t = 256) { return (unsigned)ceil_div(n > 0 ? n : 1, t); }

}  // namespace

#define SETUP_CHECK(call)                                                       \
    do {                                                                        \
        cudaError_t _e = (call);                                                \
        if (_e != cudaSuccess) {                                                \
            err = std::string(#call) + ": " + cudaGetErrorString(_e);          \
            return _e;                                                          \
        }                                                                       \
    } while (0)

cudaError_t build_geometry(int Q, const uint8_t* d_mask, int nx, int ny, int nz, const lbm_bc_spec* bc, int nbc,
                           const double origin[3], double spacing, GeometryLists& out, int32_t** seg_rows,
                           int64_t* nseg, int32_t** seg_of, cudaStream_t st, std::string& err) {
    const int64_t npts = (int64_t)nx * ny * nz;
    out.npts = npts;
    // padded to whole 32-point segments: the bulk kernel reads the class
    // byte of every lane of a segment
    const int64_t npad = ceil_div(npts, 32) * 32;
    SETUP_CHECK(cudaMallocAsync(&out.cls, npad, st));
    SETUP_CHECK(cudaMemsetAsync(out.cls, 0, npad, st));
    if (Q == 19) k_boundary<19><<<blocks(npts), 256, 0, st>>>(d_mask, nx, ny, nz, out.cls);
    else k_boundary<27><<<blocks(npts), 256, 0, st>>>(d_mask, nx, ny, nz, out.cls);
    SETUP_CHECK(cudaGetLastError());

    // plane rules; plane -1 = extreme fluid layer on the face
    Rules R{};
    R.n = nbc;
    bool need_ext = false;
    for (int b = 0; b < nbc; ++b) need_ext |= bc[b].plane < 0 && !bc[b].region;
    int ext[6] = {0, 0, 0, -1, -1, -1};
    if (need_ext) {
        int* d_ext = nullptr;
        int init[6] = {0x7fffffff, 0x7fffffff, 0x7fffffff, -1, -1, -1};
        SETUP_CHECK(cudaMallocAsync(&d_ext, sizeof(init), st));
        SETUP_CHECK(cudaMemcpyAsync(d_ext, init, sizeof(init), cudaMemcpyHostToDevice, st));
        k_extent<<<std::min(blocks(npts), 608u), 256, 0, st>>>(d_mask, nx, ny, nz, d_ext);
        SETUP_CHECK(cudaMemcpyAsync(ext, d_ext, sizeof(ext), cudaMemcpyDeviceToHost, st));
        SETUP_CHECK(cudaStreamSynchronize(st));
        cudaFreeAsync(d_ext, st);
    }
    R.org[0] = origin[0]; R.org[1] = origin[1]; R.org[2] = origin[2];
    R.s = spacing;
    for (int b = 0; b < nbc; ++b) {
        const int face = bc[b].face;
        R.axis[b] = face / 2;
        R.plane[b] = bc[b].plane >= 0 ? bc[b].plane : (face % 2 == 0 ? ext[face / 2] : ext[3 + face / 2]);
        R.region[b] = bc[b].region;
        R.coord[b] = bc[b].coord;
        R.tol[b] = bc[b].tol;
        for (int t = 0; t < 2; ++t) { R.lo[b][t] = bc[b].lo[t]; R.hi[b][t] = bc[b].hi[t]; }
        out.plane[b] = R.plane[b];
    }
    SETUP_CHECK(cudaMallocAsync(&out.bcidx, sizeof(int16_t) * npad, st));
    k_classify<<<blocks(npts), 256, 0, st>>>(out.cls, out.bcidx, nx, ny, npts, R);
    SETUP_CHECK(cudaGetLastError());
    if (Q == 19) k_next_to_wall<19><<<blocks(npts), 256, 0, st>>>(out.cls, nx, ny, nz);
    else k_next_to_wall<27><<<blocks(npts), 256, 0, st>>>(out.cls, nx, ny, nz);
    SETUP_CHECK(cudaGetLastError());

    // compact lists
    int64_t *flag = nullptr, *pos = nullptr, *nwflag = nullptr, *nwpos = nullptr;
    SETUP_CHECK(cudaMallocAsync(&flag, sizeof(int64_t) * npts, st));
    SETUP_CHECK(cudaMallocAsync(&pos, sizeof(int64_t) * npts, st));
    SETUP_CHECK(cudaMallocAsync(&nwflag, sizeof(int64_t) * npts, st));
    SETUP_CHECK(cudaMallocAsync(&nwpos, sizeof(int64_t) * npts, st));
    k_flag_special<<<blocks(npts), 256, 0, st>>>(out.cls, npts, flag, nwflag);
    int64_t nother = 0;
    SETUP_CHECK(exclusive_scan_i64(flag, pos, npts, &nother, st));
    SETUP_CHECK(exclusive_scan_i64(nwflag, nwpos, npts, &out.nnw, st));
    out.nsp = out.nnw + nother;
    k_special_pos<<<blocks(npts), 256, 0, st>>>(flag, pos, nwflag, nwpos, out.nnw, npts);
    SETUP_CHECK(cudaGetLastError());
    SETUP_CHECK(cudaMallocAsync(&out.sp_pt, sizeof(int64_t) * (out.nsp + 1), st));
    SETUP_CHECK(cudaMallocAsync(&out.nw_pt, sizeof(int64_t) * (out.nnw + 1), st));
    k_scatter<<<blocks(npts), 256, 0, st>>>(flag, pos, npts, out.sp_pt);
    k_scatter<<<blocks(npts), 256, 0, st>>>(nwflag, nwpos, npts, out.nw_pt);
    SETUP_CHECK(cudaGetLastError());
    SETUP_CHECK(cudaMallocAsync(&out.sp_miss, sizeof(uint32_t) * (out.nsp + 1), st));
    SETUP_CHECK(cudaMallocAsync(&out.sp_cls, out.nsp + 1, st));
    SETUP_CHECK(cudaMallocAsync(&out.sp_nw, sizeof(int32_t) * (out.nsp + 1), st));
    SETUP_CHECK(cudaMallocAsync(&out.sp_bc, sizeof(int32_t) * (out.nsp + 1), st));
    SETUP_CHECK(cudaMallocAsync(&out.sp_prof, sizeof(double) * (out.nsp + 1), st));
    ProfileSpec ps{};
    ps.n = nbc;
    ps.s = spacing;
    for (int d = 0; d < 3; ++d) ps.org[d] = origin[d];
    for (int b = 0; b < nbc; ++b) {
        ps.profile[b] = bc[b].profile;
        ps.axis[b] = bc[b].face / 2;
        ps.c1[b] = bc[b].c1; ps.c2[b] = bc[b].c2; ps.R[b] = bc[b].R;
    }
    if (out.nsp > 0) {
        if (Q == 19)
            k_special_info<19><<<blocks(out.nsp), 256, 0, st>>>(out.sp_pt, out.nsp, out.cls, nwpos, nx, ny, nz,
                                                               out.bcidx, out.sp_miss, out.sp_cls, out.sp_nw,
                                                               out.sp_bc, out.sp_prof, ps);
        else
            k_special_info<27><<<blocks(out.nsp), 256, 0, st>>>(out.sp_pt, out.nsp, out.cls, nwpos, nx, ny, nz,
                                                               out.bcidx, out.sp_miss, out.sp_cls, out.sp_nw,
                                                               out.sp_bc, out.sp_prof, ps);
        SETUP_CHECK(cudaGetLastError());
    }

    // active index and the packed per-node words of the step kernel
    int64_t *aflag = nullptr, *apos = nullptr;
    SETUP_CHECK(cudaMallocAsync(&aflag, sizeof(int64_t) * npts, st));
    SETUP_CHECK(cudaMallocAsync(&apos, sizeof(int64_t) * npts, st));
    k_active_flags<<<blocks(npts), 256, 0, st>>>(out.cls, npts, aflag);
    SETUP_CHECK(exclusive_scan_i64(aflag, apos, npts, &out.nact, st));
    SETUP_CHECK(cudaMallocAsync(&out.act_idx, sizeof(int32_t) * npts, st));
    SETUP_CHECK(cudaMallocAsync(&out.act_pt, sizeof(int64_t) * (out.nact + 1), st));
    SETUP_CHECK(cudaMallocAsync(&out.act_word, sizeof(uint64_t) * (out.nact + 1), st));
    // padded: the tiled step kernel copies whole 16-byte groups
    SETUP_CHECK(cudaMallocAsync(&out.sp_of_act, sizeof(int32_t) * (out.nact + 4), st));
    k_active_index<<<blocks(npts), 256, 0, st>>>(aflag, apos, npts, out.act_idx, out.act_pt);
    SETUP_CHECK(cudaGetLastError());
    SETUP_CHECK(cudaMallocAsync(seg_of, sizeof(int32_t) * (out.nact + 1), st));
    SETUP_CHECK(build_segments(Q, out, nx, ny, nz, seg_rows, nseg, *seg_of, st));
    if (Q == 19)
        k_active_word<19><<<blocks(out.nact), 256, 0, st>>>(out.act_pt, out.nact, flag, pos, out.cls, nx, ny, nz, *seg_of,
                                                           out.act_word, out.sp_of_act);
    else
        k_active_word<27><<<blocks(out.nact), 256, 0, st>>>(out.act_pt, out.nact, flag, pos, out.cls, nx, ny, nz, *seg_of,
                                                           out.act_word, out.sp_of_act);
    SETUP_CHECK(cudaGetLastError());
    cudaFreeAsync(aflag, st);
    cudaFreeAsync(apos, st);
    cudaFreeAsync(flag, st);
    cudaFreeAsync(pos, st);
    cudaFreeAsync(nwflag, st);
    cudaFreeAsync(nwpos, st);
    SETUP_CHECK(cudaStreamSynchronize(st));
    return cudaSuccess;
}

// Nearest next-to-wall node of each query point (the lattice carries WSS,
// OSI and TAWSS on those nodes).  With g the point in lattice units and c =
// round(g), the cube of half-width R around c holds every lattice point
// closer than R + 0.5; the cube grows (R = 1, 2, 4, ...) until the best
// node found lies within that bound, so the result is the exact nearest
// (ties to the lower next-to-wall index), or -1 beyond rmax.
__global__ void k_nearest_nw(const double* __restrict__ xyz, int64_t nv, const int32_t* __restrict__ act_idx,
                             const int32_t* __restrict__ sp_of_act, int64_t nnw, int nx, int ny, int nz, double ox,
                             double oy, double oz, double sp, int rmax, int64_t* __restrict__ out_idx,
                             double* __restrict__ out_dist) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    const double g[3] = {(xyz[3 * v] - ox) / sp, (xyz[3 * v + 1] - oy) / sp, (xyz[3 * v + 2] - oz) / sp};
    const int dims[3] = {nx, ny, nz};
    int c[3];
    for (int d = 0; d < 3; ++d) {
        double r = rint(g[d]);
        r = r < 0.0 ? 0.0 : (r > dims[d] - 1 ? (double)(dims[d] - 1) : r);
        c[d] = (int)r;
    }
    int64_t best = -1;
    double best_d2 = 0.0;
    for (int R = 1; R <= rmax; R *= 2) {
        const int lo[3] = {max(c[0] - R, 0), max(c[1] - R, 0), max(c[2] - R, 0)};
        const int hi[3] = {min(c[0] + R, nx - 1), min(c[1] + R, ny - 1), min(c[2] + R, nz - 1)};
        for (int k = lo[2]; k <= hi[2]; ++k)
            for (int j = lo[1]; j <= hi[1]; ++j)
                for (int i = lo[0]; i <= hi[0]; ++i) {
                    const int32_t a = act_idx[((int64_t)k * ny + j) * nx + i];
                    if (a < 0) continue;
                    const int32_t e = sp_of_act[a];
                    if (e < 0 || e >= nnw) continue;
                    const double dx = i - g[0], dy = j - g[1], dz = k - g[2];
                    const double d2 = dx * dx + dy * dy + dz * dz;
                    if (best < 0 || d2 < best_d2 || (d2 == best_d2 && e < best)) {
                        best = e;
                        best_d2 = d2;
                    }
                }
        if (best >= 0 && sqrt(best_d2) <= R + 0.5) break;
    }
    out_idx[v] = best;
    if (out_dist) out_dist[v] = best >= 0 ? sqrt(best_d2) * sp : -1.0;
}

cudaError_t nearest_next_to_wall(const double* d_xyz, int64_t nv, const GeometryLists& g, int nx, int ny, int nz,
                                 const double origin[3], double spacing, int rmax, int64_t* d_idx, double* d_dist,
                                 cudaStream_t st) {
    if (nv <= 0) return cudaSuccess;
    k_nearest_nw<<<blocks(nv, 128), 128, 0, st>>>(d_xyz, nv, g.act_idx, g.sp_of_act, g.nnw, nx, ny, nz, origin[0],
                                                 origin[1], origin[2], spacing, rmax, d_idx, d_dist);
    return cudaGetLastError();
}

// Wall distance of every missing link of the boundary list, for the
// interpolated bounce-back: for entry s and arriving population q whose
// source x - c_q (= x + c_i, i = opp q) is not active, the fraction t in
// [0, 1] along the link x -> x + c_i at which it first meets a triangle
// (segment-triangle intersection after Moller and Trumbore, 1997, in FP64),
// stored as q[qi * nsp + s]; 0.5 (half-way) where no link is missing or no
// triangle crosses it.  Triangles are tested in file order; the smallest t
// wins.  tri: ntri rows of x1 y1 z1 x2 y2 z2 x3 y3 z3 nx ny nz.
__device__ __forceinline__ bool seg_tri(const double* P0, const double* d, const double* T, double& t) {
    const double e1[3] = {T[3] - T[0], T[4] - T[1], T[5] - T[2]};
    const double e2[3] = {T[6] - T[0], T[7] - T[1], T[8] - T[2]};
    const double pv[3] = {d[1] * e2[2] - d[2] * e2[1], d[2] * e2[0] - d[0] * e2[2], d[0] * e2[1] - d[1] * e2[0]};
    const double det = e1[0] * pv[0] + e1[1] * pv[1] + e1[2] * pv[2];
    if (fabs(det) < 1e-300) return false;
    const double inv = 1.0 / det;
    const double tv[3] = {P0[0] - T[0], P0[1] - T[1], P0[2] - T[2]};
    const double u = (tv[0] * pv[0] + tv[1] * pv[1] + tv[2] * pv[2]) * inv;
    if (u < 0.0 || u > 1.0) return false;
    const double qv[3] = {tv[1] * e1[2] - tv[2] * e1[1], tv[2] * e1[0] - tv[0] * e1[2], tv[0] * e1[1] - tv[1] * e1[0]};
    const double v = (d[0] * qv[0] + d[1] * qv[1] + d[2] * qv[2]) * inv;
    if (v < 0.0 || u + v > 1.0) return false;
    t = (e2[0] * qv[0] + e2[1] * qv[1] + e2[2] * qv[2]) * inv;
    return t >= 0.0 && t <= 1.0;
}

template <int Q>
__global__ void k_wall_q(const int64_t* __restrict__ sp_pt, const uint32_t* __restrict__ sp_miss, int64_t nsp,
                         int nx, int ny, double ox, double oy, double oz, double sp, const double* __restrict__ tri,
                         int64_t ntri, float* __restrict__ out) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nsp) return;
    const int64_t n = sp_pt[e];
    const int i = (int)(n % nx), j = (int)((n / nx) % ny), k = (int)(n / ((int64_t)nx * ny));
    const double P0[3] = {ox + i * sp, oy + j * sp, oz + k * sp};
    const uint32_t miss = sp_miss[e];
    for (int q = 0; q < Q; ++q) {
        float qw = 0.5f;
        const int ci = Lat<Q>::opp(q);
        if ((miss >> ci) & 1u) {
            const double d[3] = {Lat<Q>::cx(ci) * sp, Lat<Q>::cy(ci) * sp, Lat<Q>::cz(ci) * sp};
            const double lo[3] = {fmin(P0[0], P0[0] + d[0]), fmin(P0[1], P0[1] + d[1]), fmin(P0[2], P0[2] + d[2])};
            const double hi[3] = {fmax(P0[0], P0[0] + d[0]), fmax(P0[1], P0[1] + d[1]), fmax(P0[2], P0[2] + d[2])};
            double best = 2.0;
            for (int64_t r = 0; r < ntri; ++r) {
                const double* T = tri + 12 * r;
                // bounding-box rejection (exact: a hit lies in both boxes)
                if (fmax(T[0], fmax(T[3], T[6])) < lo[0] || fmin(T[0], fmin(T[3], T[6])) > hi[0] ||
                    fmax(T[1], fmax(T[4], T[7])) < lo[1] || fmin(T[1], fmin(T[4], T[7])) > hi[1] ||
                    fmax(T[2], fmax(T[5], T[8])) < lo[2] || fmin(T[2], fmin(T[5], T[8])) > hi[2])
                    continue;
                double t;
                if (seg_tri(P0, d, T, t) && t < best) best = t;
            }
            if (best <= 1.0) qw = (float)best;
        }
        out[(int64_t)q * nsp + e] = qw;
    }
}

cudaError_t wall_distances(int Q, const double* d_tri, int64_t ntri, const GeometryLists& g, int nx, int ny,
                           const double origin[3], double spacing, float* d_q, cudaStream_t st) {
    if (g.nsp <= 0) return cudaSuccess;
    if (Q == 19)
        k_wall_q<19><<<blocks(g.nsp, 128), 128, 0, st>>>(g.sp_pt, g.sp_miss, g.nsp, nx, ny, origin[0], origin[1],
                                                        origin[2], spacing, d_tri, ntri, d_q);
    else
        k_wall_q<27><<<blocks(g.nsp, 128), 128, 0, st>>>(g.sp_pt, g.sp_miss, g.nsp, nx, ny, origin[0], origin[1],
                                                        origin[2], spacing, d_tri, ntri, d_q);
    return cudaGetLastError();
}

cudaError_t surface_normals(const double* d_tri, int64_t ntri, const int64_t* d_pts, int64_t npts, int nx, int ny,
                            const double origin[3], double spacing, double* d_out, cudaStream_t st) {
    if (npts <= 0) return cudaSuccess;
    double* tw = nullptr;
    cudaError_t e = cudaMallocAsync(&tw, sizeof(double) * kTriWeight * (ntri > 0 ? ntri : 1), st);
    if (e != cudaSuccess) return e;
    if (ntri > 0) k_tri_weights<<<blocks(ntri), 256, 0, st>>>(d_tri, ntri, tw);
    // about 8 blocks an SM, at least a tile of triangles each
    const int64_t nb = ceil_div(npts, kNormThreads);
    int64_t parts = std::min(ceil_div(8 * sm_count(), nb), ceil_div(ntri > 0 ? ntri : 1, kNormTile));
    const int64_t per = ceil_div(ceil_div(ntri > 0 ? ntri : 1, parts), 4) * 4;
    parts = ceil_div(ntri > 0 ? ntri : 1, per);
    double* sums = nullptr;
    e = cudaMallocAsync(&sums, sizeof(double) * 3 * npts * parts, st);
    if (e == cudaSuccess) {
        k_normals<<<dim3((unsigned)nb, (unsigned)parts), kNormThreads, 0, st>>>(
            tw, ntri, per, d_pts, npts, nx, ny, origin[0], origin[1], origin[2], spacing, sums);
        k_normals_sum<<<blocks(npts), 256, 0, st>>>(sums, (int)parts, npts, d_out);
        e = cudaGetLastError();
        cudaFreeAsync(sums, st);
    }
    cudaFreeAsync(tw, st);
    return e;
}

cudaError_t scatter_normals(const double* part, const int64_t* idx, int64_t m, int64_t nn, double* n, cudaStream_t st) {
    if (m > 0) k_scatter_normals<<<blocks(m), 256, 0, st>>>(part, idx, m, nn, n);
    return cudaGetLastError();
}

cudaError_t normals_to_float(const double* n, int64_t nn, int64_t stride, float* out, cudaStream_t st) {
    if (nn > 0) k_normals_float<<<blocks(stride), 256, 0, st>>>(n, nn, stride, out);
    return cudaGetLastError();
}

}  // namespace lbm
