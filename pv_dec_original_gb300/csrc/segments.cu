// Pull segments and the tiled step kernel's plan, built on the device.
//
// With populations stored by active index a, the source of population q at
// node a is the active index of point x_a - c_q: a + d_q(a) where that point
// is active.  A segment is a maximal stretch of consecutive active nodes
// whose valid d_q agree for every q (in practice an x-run of a row): node a
// begins a new one when some valid d_q(a) differs from the d_q of a node of
// the current segment.  The reference links one heap object per node
// (Subdomain.cpp:173-197).
//
// That greedy rule reads sequentially; here it is split so that everything
// but a few nodes is decided in parallel, one warp per 32 nodes:
//   p_q(a)  the last node before a where q is valid (ballots within the 32,
//           a maximum scan over the 32s);
//   L(a)    the largest p_q(a) with d_q(p_q(a)) != d_q(a), or -1: a begins a
//           segment exactly if L(a) >= the current segment's first node.  (The
//           valid d_q within a segment agree, so the last one stands for all.)
// L(a) = a - 1 always begins one, whatever came before; a group of 32 with
// such a node hands on a known segment start.  Groups that have candidates
// (L >= 0) but no such node are walked in order, from the start that the
// groups before them hand on.
// The serial loops over points on the host this replaces (segments and the
// tiled kernel's plan) took 110 of the 130-140 ms of a set-up of 218k nodes
// (Grace, one core); these kernels 0.1 ms, bound by their launches and scans.
#include "lbm_internal.cuh"
#include "setup.cuh"

namespace lbm {
namespace {

constexpr int kWarps = 8;  // groups of 32 nodes per block

// Source of population q at active node a (point n at i, j, k): its active index, or -1.
template <int Q>
__device__ __forceinline__ int32_t source_of(const int32_t* __restrict__ act_idx, int q, int64_t n, int i, int j, int k,
                                             int nx, int ny, int nz) {
    const int x = i - Lat<Q>::cx(q), y = j - Lat<Q>::cy(q), z = k - Lat<Q>::cz(q);
    if (x < 0 || x >= nx || y < 0 || y >= ny || z < 0 || z >= nz) return -1;
    return __ldg(act_idx + (n - Lat<Q>::cx(q) - Lat<Q>::cy(q) * (int64_t)nx - Lat<Q>::cz(q) * (int64_t)nx * ny));
}

struct SegGrid {
    const int32_t* act_idx;
    const int64_t* act_pt;
    int64_t nact, ngroups;
    int nx, ny, nz;
};

// One warp's group: lane's node, its coordinates.
struct Lane {
    int64_t g, a, n;
    int i, j, k;
    bool in;
};
__device__ __forceinline__ Lane lane_of(const SegGrid& G) {
    Lane l;
    l.g = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    l.a = l.g * 32 + (threadIdx.x & 31);
    l.in = l.g < G.ngroups && l.a < G.nact;
    l.n = l.in ? G.act_pt[l.a] : 0;
    l.i = (int)(l.n % G.nx);
    const int64_t r = l.n / G.nx;
    l.j = (int)(r % G.ny);
    l.k = (int)(r / G.ny);
    return l;
}

// last[q][group]: the group's last node where q is valid, or -1.
template <int Q>
__global__ void __launch_bounds__(32 * kWarps) k_seg_last(SegGrid G, int32_t* __restrict__ last) {
    const Lane l = lane_of(G);
    if (l.g >= G.ngroups) return;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const bool v = l.in && source_of<Q>(G.act_idx, q, l.n, l.i, l.j, l.k, G.nx, G.ny, G.nz) >= 0;
        const unsigned b = __ballot_sync(0xffffffffu, v);
        if (lane == 0) last[q * G.ngroups + l.g] = b ? (int32_t)(l.g * 32 + 31 - __clz(b)) : -1;
    }
}

// Exclusive maximum scan of rows of n values (one block a row); -1 before the first.
__global__ void __launch_bounds__(1024) k_max_scan(const int32_t* __restrict__ in, int32_t* __restrict__ out, int64_t n) {
    __shared__ int32_t warp_max[32];
    const int32_t* src = in + (int64_t)blockIdx.x * n;
    int32_t* dst = out + (int64_t)blockIdx.x * n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t carry = -1;
    for (int64_t base = 0; base < n; base += 1024) {
        const int64_t e = base + threadIdx.x;
        const int32_t own = e < n ? src[e] : -1;
        int32_t m = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int32_t o = __shfl_up_sync(0xffffffffu, m, d);
            if (lane >= d) m = max(m, o);
        }
        if (lane == 31) warp_max[warp] = m;
        __syncthreads();
        int32_t before = carry, all = carry;
        for (int w = 0; w < 32; ++w) {
            const int32_t o = warp_max[w];
            if (w < warp) before = max(before, o);
            all = max(all, o);
        }
        int32_t ex = __shfl_up_sync(0xffffffffu, m, 1);
        ex = lane == 0 ? before : max(before, ex);
        if (e < n) dst[e] = ex;
        carry = all;
        __syncthreads();
    }
}

// L(a) of every node.
template <int Q>
__global__ void __launch_bounds__(32 * kWarps) k_seg_conflict(SegGrid G, const int32_t* __restrict__ prev,
                                                             int32_t* __restrict__ L) {
    const Lane l = lane_of(G);
    if (l.g >= G.ngroups) return;
    const int lane = threadIdx.x & 31;
    const int64_t base = l.g * 32;
    int32_t best = -1;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int32_t s = l.in ? source_of<Q>(G.act_idx, q, l.n, l.i, l.j, l.k, G.nx, G.ny, G.nz) : -1;
        const bool v = s >= 0;
        const int32_t d = v ? s - (int32_t)l.a : 0;
        const unsigned b = __ballot_sync(0xffffffffu, v), lower = b & ((1u << lane) - 1u);
        int32_t dp = __shfl_sync(0xffffffffu, d, lower ? 31 - __clz(lower) : 0);
        int32_t p = (int32_t)base + (lower ? 31 - __clz(lower) : 0);
        if (v && !lower) {
            // the group's first valid node: its predecessor lies in an earlier group
            p = prev[q * G.ngroups + l.g];
            if (p >= 0) {
                const int64_t n = G.act_pt[p];
                dp = G.act_idx[n - Lat<Q>::cx(q) - Lat<Q>::cy(q) * (int64_t)G.nx -
                               Lat<Q>::cz(q) * (int64_t)G.nx * G.ny] - p;
            }
        }
        if (v && p >= 0 && dp != d) best = max(best, p);
    }
    if (l.in) L[l.a] = best;
}

// Segment starts of a group from the segment start `s` handed on, as a lane
// mask; s becomes the start handed on.  Lanes below `from` are skipped.
__device__ __forceinline__ unsigned walk(int32_t Lv, int64_t base, int from, int32_t& s) {
    unsigned cand = __ballot_sync(0xffffffffu, Lv >= 0) & ~((1u << from) - 1u), starts = 0;
    while (cand) {
        const int b = __ffs(cand) - 1;
        cand &= cand - 1;
        if (__shfl_sync(0xffffffffu, Lv, b) >= s) {
            starts |= 1u << b;
            s = (int32_t)base + b;
        }
    }
    return starts;
}

// Per group: known[g] = the start it hands on if that is known without its
// predecessors (node 0, or a node with L = a - 1), else -1; open[g] = 1 if
// it has candidates but no such node.
__global__ void __launch_bounds__(32 * kWarps) k_seg_known(SegGrid G, const int32_t* __restrict__ L,
                                                          int32_t* __restrict__ known, int64_t* __restrict__ open) {
    const int64_t g = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (g >= G.ngroups) return;
    const int lane = threadIdx.x & 31;
    const int64_t base = g * 32, a = base + lane;
    const int32_t Lv = a < G.nact ? L[a] : -1;
    const unsigned sure = __ballot_sync(0xffffffffu, a < G.nact && (a == 0 || Lv == (int32_t)a - 1));
    const unsigned cand = __ballot_sync(0xffffffffu, Lv >= 0);
    int32_t s = -1;
    if (sure) {
        const int c = __ffs(sure) - 1;
        s = (int32_t)base + c;
        if (c < 31) walk(Lv, base, c + 1, s);
    }
    if (lane == 0) {
        known[g] = s;
        open[g] = !sure && cand ? 1 : 0;
    }
}

__global__ void k_seg_list(const int64_t* __restrict__ open, const int64_t* __restrict__ pos, int64_t n,
                           int32_t* __restrict__ list) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < n && open[g]) list[pos[g]] = (int32_t)g;
}

// The open groups, one warp per run of them between groups with a known
// start: walked in order, known[g] = the last start found (or left -1).
__global__ void __launch_bounds__(32 * kWarps) k_seg_open(SegGrid G, const int32_t* __restrict__ L,
                                                         const int32_t* __restrict__ before,
                                                         const int32_t* __restrict__ list, int64_t nopen,
                                                         int32_t* __restrict__ known) {
    const int64_t w = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (w >= nopen) return;
    const int lane = threadIdx.x & 31;
    // a run begins where a start is known between this open group and the one before it
    auto head = [&](int64_t e) { return e == 0 || before[list[e]] >= ((int64_t)list[e - 1] + 1) * 32; };
    if (!head(w)) return;
    int32_t s = before[list[w]];
    for (int64_t e = w; e < nopen && (e == w || !head(e)); ++e) {
        const int64_t g = list[e], a = g * 32 + lane;
        const int32_t s0 = s;
        walk(a < G.nact ? L[a] : -1, g * 32, 0, s);
        if (lane == 0 && s != s0) known[g] = s;
    }
}

// Segment starts of every group, and their number.
__global__ void __launch_bounds__(32 * kWarps) k_seg_starts(SegGrid G, const int32_t* __restrict__ L,
                                                           const int32_t* __restrict__ before,
                                                           uint32_t* __restrict__ starts, int64_t* __restrict__ count) {
    const int64_t g = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (g >= G.ngroups) return;
    const int lane = threadIdx.x & 31;
    const int64_t a = g * 32 + lane;
    int32_t s = before[g];
    unsigned m = walk(a < G.nact ? L[a] : -1, g * 32, 0, s);
    if (g == 0) m |= 1u;  // (node 0 has no predecessor: never a candidate)
    if (lane == 0) {
        starts[g] = m;
        count[g] = __popc(m);
    }
}

// Per node its segment, per segment its Q offsets (0 where no node has that
// source: the rows start zeroed; all nodes of a segment write the same).
template <int Q>
__global__ void __launch_bounds__(32 * kWarps) k_seg_rows(SegGrid G, const uint32_t* __restrict__ starts,
                                                         const int64_t* __restrict__ first,
                                                         int32_t* __restrict__ seg_of, int32_t* __restrict__ rows) {
    const Lane l = lane_of(G);
    if (!l.in) return;
    const int lane = threadIdx.x & 31;
    const int32_t seg = (int32_t)(first[l.g] + __popc(starts[l.g] & (0xffffffffu >> (31 - lane))) - 1);
    seg_of[l.a] = seg;
    int32_t* row = rows + (int64_t)seg * kDeltaRow<Q>;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int32_t s = source_of<Q>(G.act_idx, q, l.n, l.i, l.j, l.k, G.nx, G.ny, G.nz);
        if (s >= 0) row[q] = s - (int32_t)l.a;
    }
}

#define SEG_CHECK(call)                       \
    do {                                      \
        const cudaError_t _e = (call);        \
        if (_e != cudaSuccess) return _e;     \
    } while (0)

template <int Q>
cudaError_t segments_q(SegGrid G, int32_t** rows_out, int64_t* nseg, int32_t* seg_of, cudaStream_t st) {
    const int64_t ng = G.ngroups;
    const unsigned nb = (unsigned)ceil_div(ng, kWarps);
    // scratch: last / prev [Q][ng], L [32 ng], known / before [ng], open / pos [ng] (int64), list, starts [ng]
    const size_t i4 = sizeof(int32_t), bytes = i4 * (size_t)ng * (2 * Q + 32 + 4) + 2 * sizeof(int64_t) * (size_t)ng;
    unsigned char* base = nullptr;
    SEG_CHECK(cudaMallocAsync(&base, bytes, st));
    int64_t* open = reinterpret_cast<int64_t*>(base);
    int64_t* pos = open + ng;
    int32_t* last = reinterpret_cast<int32_t*>(pos + ng);
    int32_t* prev = last + Q * ng;
    int32_t* L = prev + Q * ng;
    int32_t* known = L + 32 * ng;
    int32_t* before = known + ng;
    int32_t* list = before + ng;
    uint32_t* starts = reinterpret_cast<uint32_t*>(list + ng);
    auto body = [&]() -> cudaError_t {
        k_seg_last<Q><<<nb, 32 * kWarps, 0, st>>>(G, last);
        k_max_scan<<<Q, 1024, 0, st>>>(last, prev, ng);
        k_seg_conflict<Q><<<nb, 32 * kWarps, 0, st>>>(G, prev, L);
        k_seg_known<<<nb, 32 * kWarps, 0, st>>>(G, L, known, open);
        k_max_scan<<<1, 1024, 0, st>>>(known, before, ng);
        int64_t nopen = 0;
        SEG_CHECK(exclusive_scan_i64(open, pos, ng, &nopen, st));
        if (nopen > 0) {
            k_seg_list<<<(unsigned)ceil_div(ng, 256), 256, 0, st>>>(open, pos, ng, list);
            k_seg_open<<<(unsigned)ceil_div(nopen, kWarps), 32 * kWarps, 0, st>>>(G, L, before, list, nopen, known);
            k_max_scan<<<1, 1024, 0, st>>>(known, before, ng);
        }
        k_seg_starts<<<nb, 32 * kWarps, 0, st>>>(G, L, before, starts, open);
        SEG_CHECK(cudaGetLastError());
        SEG_CHECK(exclusive_scan_i64(open, pos, ng, nseg, st));
        SEG_CHECK(cudaMalloc(rows_out, i4 * ((size_t)*nseg * kDeltaRow<Q> + 1)));
        SEG_CHECK(cudaMemsetAsync(*rows_out, 0, i4 * (size_t)*nseg * kDeltaRow<Q>, st));
        k_seg_rows<Q><<<nb, 32 * kWarps, 0, st>>>(G, starts, pos, seg_of, *rows_out);
        return cudaGetLastError();
    };
    const cudaError_t e = body();
    cudaFreeAsync(base, st);
    return e;
}

// Plan of a tile (one block, kTileNodes threads): windows of the valid pull
// sources per plane, widened to 16 bytes (A elements), the tile's segments and
// next-to-wall entries.  most[0..2]: the largest window, segment count and
// entry count; most[3]: a window that leaves its plane.
template <int Q>
__global__ void __launch_bounds__(kTileNodes) k_tile_plan(SegGrid G, const int32_t* __restrict__ seg_of,
                                                          const int32_t* __restrict__ sp_of_act, int64_t nnw,
                                                          int64_t stride, int A, int32_t* __restrict__ plan,
                                                          int* __restrict__ most) {
    __shared__ int lo[Q + 1], hi[Q + 1];
    const int64_t t = blockIdx.x, a0 = t * kTileNodes, a = a0 + threadIdx.x;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x <= Q) {
        lo[threadIdx.x] = 0x7fffffff;
        hi[threadIdx.x] = -1;
    }
    __syncthreads();
    const bool in = a < G.nact;
    const int64_t n = in ? G.act_pt[a] : 0;
    const int i = (int)(n % G.nx), j = (int)((n / G.nx) % G.ny), k = (int)(n / ((int64_t)G.nx * G.ny));
#pragma unroll
    for (int q = 0; q <= Q; ++q) {
        int32_t s = -1;
        if (in) {
            if (q < Q) s = source_of<Q>(G.act_idx, q < Q ? q : 0, n, i, j, k, G.nx, G.ny, G.nz);
            else s = sp_of_act[a] < nnw ? sp_of_act[a] : -1;
        }
        const int l = __reduce_min_sync(0xffffffffu, s >= 0 ? s : 0x7fffffff), h = __reduce_max_sync(0xffffffffu, s);
        if (lane == 0 && h >= 0) {
            atomicMin(lo + q, l);
            atomicMax(hi + q, h);
        }
    }
    __syncthreads();
    int32_t* pl = plan + t * (2 * Q + kTilePlanExtra);
    if (threadIdx.x < Q) {
        const int q = threadIdx.x;
        int l0 = 0, len = 0;
        if (hi[q] >= 0) {
            l0 = lo[q] / A * A;
            const int h1 = (hi[q] + 1 + A - 1) / A * A;
            len = h1 - l0;
            if (h1 > stride) most[3] = 1;
            atomicMax(most, len);
        }
        pl[q] = l0;
        pl[Q + q] = len;
    } else if (threadIdx.x == 32) {
        const int64_t a1 = (a0 + kTileNodes < G.nact ? a0 + kTileNodes : G.nact) - 1;
        const int count = seg_of[a1] - seg_of[a0] + 1;
        pl[2 * Q] = seg_of[a0];
        pl[2 * Q + 1] = count;
        atomicMax(most + 1, count);
    } else if (threadIdx.x == 64) {
        int e0 = 0, ne = 0;
        if (hi[Q] >= 0) {
            e0 = lo[Q] / 4 * 4;
            ne = (hi[Q] + 1 + 3) / 4 * 4 - e0;
            atomicMax(most + 2, ne);
        }
        pl[2 * Q + 2] = e0;
        pl[2 * Q + 3] = ne;
    }
}

__global__ void k_tile_cap(int32_t* __restrict__ plan, int64_t ntiles, int width, int at, int cap) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ntiles && plan[t * width + at] > cap) plan[t * width + at] = cap;  // the rest read their rows from global memory
}

}  // namespace

cudaError_t build_segments(int Q, const GeometryLists& g, int nx, int ny, int nz, int32_t** rows, int64_t* nseg,
                           int32_t* seg_of, cudaStream_t st) {
    *nseg = 0;
    if (g.nact <= 0) return cudaMalloc(rows, sizeof(int32_t));
    const SegGrid G{g.act_idx, g.act_pt, g.nact, ceil_div(g.nact, 32), nx, ny, nz};
    return Q == 19 ? segments_q<19>(G, rows, nseg, seg_of, st) : segments_q<27>(G, rows, nseg, seg_of, st);
}

cudaError_t build_tile_plan(int Q, const GeometryLists& g, int nx, int ny, int nz, const int32_t* seg_of,
                            int64_t stride, int elem_size, int32_t* plan, int most[4], cudaStream_t st) {
    const SegGrid G{g.act_idx, g.act_pt, g.nact, 0, nx, ny, nz};
    const unsigned nt = (unsigned)ceil_div(g.nact, kTileNodes);
    int* d_most = nullptr;
    SEG_CHECK(cudaMallocAsync(&d_most, 4 * sizeof(int), st));
    cudaError_t e = cudaMemsetAsync(d_most, 0, 4 * sizeof(int), st);
    if (e == cudaSuccess) {
        if (Q == 19)
            k_tile_plan<19><<<nt, kTileNodes, 0, st>>>(G, seg_of, g.sp_of_act, g.nnw, stride, 16 / elem_size, plan, d_most);
        else
            k_tile_plan<27><<<nt, kTileNodes, 0, st>>>(G, seg_of, g.sp_of_act, g.nnw, stride, 16 / elem_size, plan, d_most);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(most, d_most, 4 * sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFreeAsync(d_most, st);
    return e;
}

cudaError_t cap_tile_segments(int Q, int32_t* plan, int64_t ntiles, int cap, cudaStream_t st) {
    k_tile_cap<<<(unsigned)ceil_div(ntiles, 256), 256, 0, st>>>(plan, ntiles, 2 * Q + kTilePlanExtra, 2 * Q + 1, cap);
    return cudaGetLastError();
}

}  // namespace lbm
