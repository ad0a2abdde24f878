// Network upload, contact grid, tunnelling-contact search, Hoshen-Kopelman
// labelling, junction compression, elements, percolation (device).
#include <algorithm>
#include <cmath>
#include <mutex>

#include "ctx.cuh"
#include "trace.cuh"
#include "uf.cuh"

namespace cicy {

namespace {

constexpr double kZero = 1.0e-10;  // MathMatrix.h:18

// ---------------------------------------------------------------------------
// Contact grid (Contact_grid.cpp:104-295).  Region coordinates and overlap flags
// use the exact upstream operation sequence (FP64, no contraction).
struct PointRegions {
    long long t[4];
    int n;
};

__device__ __forceinline__ PointRegions regions_of(double px, double py, double pz, const GridGeom g) {
    // Calculate_region_coordinates (Contact_grid.cpp:163-184)
    int a = (int)((px - g.min[0]) / g.l[0]);
    if (a < 0) a = 0; else if (a >= g.n[0]) a = g.n[0] - 1;
    int b = (int)((py - g.min[1]) / g.l[1]);
    if (b < 0) b = 0; else if (b >= g.n[1]) b = g.n[1] - 1;
    int c = (int)((pz - g.min[2]) / g.l[2]);
    if (c < 0) c = 0; else if (c >= g.n[2]) c = g.n[2] - 1;
    // Calculate_overlapping_flags (Contact_grid.cpp:186-212)
    double x1 = (double)a * g.l[0] + g.min[0];
    double x2 = x1 + g.l[0];
    double y1 = (double)b * g.l[1] + g.min[1];
    double y2 = y1 + g.l[1];
    double z1 = (double)c * g.l[2] + g.min[2];
    double z2 = z1 + g.l[2];
    const double ov = g.overlap;
    int f0 = 0, f1 = 0, f2 = 0;
    if ((a > 0) && (px >= x1) && (px <= x1 + ov)) f0 = -1;
    else if ((a < g.n[0] - 1) && (px >= x2 - ov) && (px <= x2)) f0 = 1;
    if ((b > 0) && (py >= y1) && (py <= y1 + ov)) f1 = -1;
    else if ((b < g.n[1] - 1) && (py >= y2 - ov) && (py <= y2)) f1 = 1;
    if ((c > 0) && (pz >= z1) && (pz <= z1 + ov)) f2 = -1;
    else if ((c < g.n[2] - 1) && (pz >= z2 - ov) && (pz <= z2)) f2 = 1;
    // Assign_point_to_regions_cnts + Calculate_t (Contact_grid.cpp:214-295)
    const long long sx = g.n[0], sxy = (long long)g.n[0] * g.n[1];
    PointRegions r;
    r.n = 0;
    r.t[r.n++] = a + b * sx + c * sxy;
    if (f0) r.t[r.n++] = (a + f0) + b * sx + c * sxy;
    if (f1) r.t[r.n++] = a + (b + f1) * sx + c * sxy;
    if (f2) r.t[r.n++] = a + b * sx + (c + f2) * sxy;
    return r;
}

__device__ __forceinline__ int trav_rank(const int32_t* __restrict__ off, int n, int q) {
    int lo = 0, hi = n;  // find last i with off[i] <= q
    while (hi - lo > 1) {
        int m = (lo + hi) >> 1;
        if (off[m] <= q) lo = m; else hi = m;
    }
    return lo;
}

// Points in traversal order q = (rank in cnts_inside, position in structure):
// the order Fill_sectioned_domain_cnts pushes them (Contact_grid.cpp:114-160).  The count pass
// keeps each point's regions and its arrival number in them, so the scatter pass neither divides
// nor counts again (25k-CNT network: 72 + 99 us when both passes did both, 80 + 21 us so).
__global__ void k_grid_count(int n_trav, const int32_t* __restrict__ trav_off, int n_inside, const int32_t* __restrict__ inside,
                             const int32_t* __restrict__ cstart, const double* __restrict__ x, const double* __restrict__ y,
                             const double* __restrict__ z, GridGeom g, int32_t* __restrict__ trav_pt, int32_t* __restrict__ cnt,
                             int4* __restrict__ regs, ushort4* __restrict__ ranks) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n_trav; q += gridDim.x * blockDim.x) {
        int r = trav_rank(trav_off, n_inside, q);
        int P = cstart[inside[r]] + (q - trav_off[r]);
        trav_pt[q] = P;
        PointRegions pr = regions_of(x[P], y[P], z[P], g);
        int t[4];
        unsigned short k[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            t[i] = i < pr.n ? (int)pr.t[i] : -1;
            // a region of more than kSegSortMax points is an error the sort reports: numbers past 16 bits only have to stay inside it
            k[i] = i < pr.n ? (unsigned short)min(atomicAdd(&cnt[t[i]], 1), 65535) : 0;
        }
        regs[q] = make_int4(t[0], t[1], t[2], t[3]);
        ranks[q] = make_ushort4(k[0], k[1], k[2], k[3]);
    }
}

__global__ void k_grid_scatter(int n_trav, const int4* __restrict__ regs, const ushort4* __restrict__ ranks,
                               const int32_t* __restrict__ region_ptr, uint32_t* __restrict__ slot_q) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n_trav; q += gridDim.x * blockDim.x) {
        const int4 t = regs[q];
        const ushort4 k = ranks[q];
        slot_q[region_ptr[t.x] + k.x] = (uint32_t)q;
        if (t.y >= 0) slot_q[region_ptr[t.y] + k.y] = (uint32_t)q;
        if (t.z >= 0) slot_q[region_ptr[t.z] + k.z] = (uint32_t)q;
        if (t.w >= 0) slot_q[region_ptr[t.w] + k.w] = (uint32_t)q;
    }
}

// ---------------------------------------------------------------------------
// Tunnelling-contact search: every j<k pair of every region, as
// Hoshen_Kopelman::Label_cnts_in_window (Hoshen_Kopelman.cpp:255-369) scans
// them.  A block stages the points of a contiguous run of slots in shared
// memory; each thread owns slots j and walks k = j+1 .. end of their region.
//
// One pair in about 200 is a contact, and the test upstream makes is FP64 with a square root.
// The walk therefore only rules pairs out, in FP32 on positions relative to the window (16 B per
// staged point, one conflict-free load a pair): a pair is dropped when its FP32 distance is above
// the largest cutoff by more than the rounding of both positions can be.  The others are queued
// in shared memory and tested exactly as upstream does, all threads taking queued pairs, so the
// square roots and the gathers of exact points are not paid by whole warps for one lane's pair
// (25k-CNT network: 310 us with the FP64 test on every pair, 195 us so).
constexpr int kPairThreads = 256;
constexpr int kPairTile = 512;      // slots owned by one block
constexpr int kPairStage = 1024;    // slots staged in shared memory (tile + region tail): 16 KB
constexpr int kPairQueue = 1024;    // pairs queued before the block tests them

struct PairGeom {
    double min[3];
    float far;    // positions further than this from the window's corner go to the exact test
    float cut2;   // pairs above this squared FP32 distance are no contact
    double vdw, tunnel;
};

struct RawContacts {
    int cap;
    int32_t* count;   // contacts found
    int32_t* per_cnt; // contacts of each smaller CNT
    int32_t *a, *b, *pa, *pb, *pos;
    double* d;
    uint64_t* key;
    size_t lay(Carver v) {
        d = v.take<double>(cap); key = v.take<uint64_t>(cap);
        for (int32_t** q : {&a, &b, &pa, &pb, &pos}) *q = v.take<int32_t>(cap);
        return v.at;
    }
};

// Staged point: position relative to the window (NaN: test exactly) and CNT.
__device__ __forceinline__ float4 load_slot(int s, const PairGeom& g, const uint32_t* __restrict__ slot_sorted,
                                            const int32_t* __restrict__ trav_pt, const double* __restrict__ x, const double* __restrict__ y,
                                            const double* __restrict__ z, const int32_t* __restrict__ flag) {
    const int P = trav_pt[slot_sorted[s]];
    float4 v;
    v.x = (float)(x[P] - g.min[0]);
    v.y = (float)(y[P] - g.min[1]);
    v.z = (float)(z[P] - g.min[2]);
    if (!(fabsf(v.x) <= g.far && fabsf(v.y) <= g.far && fabsf(v.z) <= g.far)) v.x = __int_as_float(0x7fffffff);
    v.w = __int_as_float(flag[P]);
    return v;
}

__global__ void __launch_bounds__(kPairThreads) k_pairs(int n_slots, PairGeom g, const int32_t* __restrict__ region_ptr,
                                                        const int32_t* __restrict__ slot_region,
                                                        const uint32_t* __restrict__ slot_sorted,
                                                        const int32_t* __restrict__ trav_pt, const double* __restrict__ x,
                                                        const double* __restrict__ y, const double* __restrict__ z,
                                                        const int32_t* __restrict__ flag, const double* __restrict__ radii,
                                                        const int* __restrict__ status, RawContacts raw) {
    __shared__ float4 st[kPairStage];
    __shared__ int2 queue[kPairQueue];
    __shared__ int n_queue;
    if (*status != 0) return;  // a region too long to be ordered: its slots are not set
    const int s0 = blockIdx.x * kPairTile;
    const int s_last = min(s0 + kPairTile, n_slots) - 1;
    const int stage_end = min(region_ptr[slot_region[s_last] + 1], s0 + kPairStage);
    for (int s = s0 + threadIdx.x; s < stage_end; s += kPairThreads) st[s - s0] = load_slot(s, g, slot_sorted, trav_pt, x, y, z, flag);
    if (threadIdx.x == 0) n_queue = 0;
    __syncthreads();
    // the exact test of slots (s, k) of one region
    auto test = [&](int s, int k) {
        const int P1 = trav_pt[slot_sorted[s]], P2 = trav_pt[slot_sorted[k]];
        const int c1 = flag[P1], c2 = flag[P2];
        // Point_3D::distance_to (Geometry_3D.cpp:64-70), then the junction distance
        double dx = x[P1] - x[P2], dy = y[P1] - y[P2], dz = z[P1] - z[P2];
        double dist_cnts = sqrt(dx * dx + dy * dy + dz * dz);
        double dj = dist_cnts - radii[c1] - radii[c2];
        if (dj < g.vdw) dj = g.vdw;
        if (!(dj <= g.tunnel)) return;
        const bool lo1 = c1 < c2;
        const int a = lo1 ? c1 : c2;
        const int pos = atomicAdd(raw.count, 1);
        if (pos >= raw.cap) return;
        raw.a[pos] = a;
        raw.b[pos] = lo1 ? c2 : c1;
        raw.pa[pos] = lo1 ? P1 : P2;
        raw.pb[pos] = lo1 ? P2 : P1;
        raw.d[pos] = dj;
        const int t = slot_region[s], r0 = region_ptr[t];
        raw.key[pos] = ((uint64_t)t << 26) | ((uint64_t)(s - r0) << 13) | (uint64_t)(k - r0);
        raw.pos[pos] = atomicAdd(&raw.per_cnt[a], 1);
    };
    for (int s = s0 + threadIdx.x; s <= s_last; s += kPairThreads) {
        const int r1 = region_ptr[slot_region[s] + 1];
        const float4 p1 = st[s - s0];
        for (int k = s + 1; k < r1; k++) {
            const float4 p2 = (k < stage_end) ? st[k - s0] : load_slot(k, g, slot_sorted, trav_pt, x, y, z, flag);
            const float dx = p1.x - p2.x, dy = p1.y - p2.y, dz = p1.z - p2.z;
            if (__float_as_int(p1.w) == __float_as_int(p2.w) || dx * dx + dy * dy + dz * dz > g.cut2) continue;
            const int q = atomicAdd(&n_queue, 1);
            if (q < kPairQueue) queue[q] = make_int2(s, k);
            else test(s, k);
        }
    }
    __syncthreads();
    const int nq = min(n_queue, kPairQueue);
    for (int q = threadIdx.x; q < nq; q += kPairThreads) test(queue[q].x, queue[q].y);
}

// ---------------------------------------------------------------------------
// Contacts of each CNT a with larger CNTs b, from the unordered list of contact visits: ordered by
// (b, point of a), point_contacts (for each (Pa, CNTb) the strictly smallest junction distance,
// first in scan order on ties, Hoshen_Kopelman.cpp:353-364), the union of a and b, and
// Compress_cnt_cnt_contact_segments (:443-554) on each (a, b).  A CNT has a few to a few hundred
// visits, so a warp orders and reduces them at once (a CTA above kConWarpCap, in global memory
// above kConCtaCap); a counting sort by CNT and these two launches replace a radix sort of all
// visits and eleven launches with three host reads between them.
constexpr int kConWarps = 8, kConWarpCap = 128;
constexpr int kConCtaThreads = 256, kConCtaCap = 2048;

__global__ void k_cnt_init(int n, int32_t* __restrict__ parent, unsigned long long* __restrict__ minkey, int32_t* __restrict__ per_cnt,
                           int32_t* __restrict__ face_bits, int32_t* __restrict__ has_junc) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        per_cnt[i] = 0;
        if (i == n) break;
        parent[i] = i;
        minkey[i] = ~0ull;
        face_bits[i] = 0;
        has_junc[i] = 0;
    }
}

__global__ void k_raw_place(int n, RawContacts raw, const int32_t* __restrict__ ofs, int32_t* __restrict__ perm) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) perm[ofs[raw.a[i]] + raw.pos[i]] = i;
}

struct ContactOut {  // per visit segment of each CNT: its contacts, its junctions
    int32_t *b, *pa, *pb;
    double* d;
    int32_t *jp1, *jp2, *jn2;
    double* jd;
    int64_t* counts;            // contacts (low half), junctions (high half)
    unsigned long long* kmin;   // first visit in scan order
    int32_t* parent;
    int min_points;
    // sorting scratch of the segments too
    int32_t *perm, *idx;
    uint64_t* key;
    size_t lay(Carver v, size_t n) {
        d = v.take<double>(n); jd = v.take<double>(n); key = v.take<uint64_t>(n);
        for (int32_t** q : {&b, &pa, &pb, &jp1, &jp2, &jn2, &perm, &idx}) *q = v.take<int32_t>(n);
        return v.at;
    }
};

template <int T>
__device__ __forceinline__ void con_sync() {
    if constexpr (T == 32) __syncwarp();
    else __syncthreads();
}

template <int T>
__device__ __forceinline__ int con_scan(int v, int tid, int* ws, int& total) {
    const int lane = tid & 31;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    if constexpr (T == 32) {
        total = __shfl_sync(0xffffffffu, incl, 31);
        return incl - v;
    } else {
        if (lane == 31) ws[tid >> 5] = incl;
        __syncthreads();
        int below = 0, all = 0;
        for (int k = 0; k < T / 32; k++) {
            if (k < (tid >> 5)) below += ws[k];
            all += ws[k];
        }
        __syncthreads();
        total = all;
        return below + incl - v;
    }
}

// One (a, b) group of contacts [k, e): its junctions (written at jo when kWrite); returns their number.
template <bool kWrite>
__device__ __forceinline__ int compress_group(int k, int e, const ContactOut& O, int jo) {
    const int cj = O.b[k];
    long long Pi0 = O.pa[k], Pj0 = O.pb[k];
    double dmin = O.d[k];
    long long Pi_j = Pi0, Pj_j = Pj0;
    int out = 0;
    auto emit = [&]() {
        if (kWrite) {
            O.jp1[jo + out] = (int32_t)Pi_j;
            O.jp2[jo + out] = (int32_t)Pj_j;
            O.jn2[jo + out] = cj;
            O.jd[jo + out] = dmin;
        }
        out++;
    };
    for (k++; k < e && O.b[k] == cj; k++) {
        long long Pi1 = O.pa[k], Pj1 = O.pb[k];
        double d = O.d[k];
        long long dj = Pj1 - Pj0;
        if (dj < 0) dj = -dj;
        if (Pi1 - Pi0 >= O.min_points || dj >= O.min_points) {
            emit();
            dmin = d; Pi_j = Pi1; Pj_j = Pj1;
        } else if (d < dmin) {
            dmin = d; Pi_j = Pi1; Pj_j = Pj1;
        }
        Pi0 = Pi1;
        Pj0 = Pj1;
    }
    emit();
    return out;
}

template <int T>
__device__ __forceinline__ void contacts_of(int a, int o, int L, const RawContacts& raw, const ContactOut& O, uint64_t* K, int32_t* I, int tid, int* ws) {
    unsigned long long km = ~0ull;
    for (int t = tid; t < L; t += T) {
        const int i = O.perm[o + t];
        K[t] = ((uint64_t)(uint32_t)raw.b[i] << 32) | (uint32_t)raw.pa[i];
        I[t] = i;
        km = min(km, (unsigned long long)raw.key[i]);
    }
    con_sync<T>();
    // bitonic sort of (K, I), smaller key first in every comparison (positions past L act as +infinity)
    auto order = [&](int u, int v) {
        if (v >= L) return;
        const uint64_t ku = K[u], kv = K[v];
        if (ku > kv) {
            K[u] = kv;
            K[v] = ku;
            const int32_t t = I[u];
            I[u] = I[v];
            I[v] = t;
        }
    };
    int P = 1;
    while (P < L) P <<= 1;
    for (int half = 1, lg = 0; 2 * half <= P; half <<= 1, lg++) {
        for (int q = tid; q < P / 2; q += T) {
            const int base = (q >> lg) << (lg + 1), r = q & (half - 1);
            order(base + r, base + 2 * half - 1 - r);
        }
        con_sync<T>();
        for (int stride = half >> 1; stride > 0; stride >>= 1) {
            for (int q = tid; q < P / 2; q += T) {
                const int u = ((q & ~(stride - 1)) << 1) | (q & (stride - 1));
                order(u, u + stride);
            }
            con_sync<T>();
        }
    }
    int nu = 0, tot;
    for (int i0 = 0; i0 < L; i0 += T) {
        const int i = i0 + tid;
        const bool head = i < L && (i == 0 || K[i] != K[i - 1]);
        const int u = o + nu + con_scan<T>(head ? 1 : 0, tid, ws, tot);
        if (head) {
            int best = I[i];
            double bd = raw.d[best];
            uint64_t bk = raw.key[best];
            for (int j = i + 1; j < L && K[j] == K[i]; j++) {
                const int v = I[j];
                const double d = raw.d[v];
                const uint64_t k = raw.key[v];
                if (d < bd || (d == bd && k < bk)) { best = v; bd = d; bk = k; }
            }
            O.b[u] = raw.b[best];
            O.pa[u] = raw.pa[best];
            O.pb[u] = raw.pb[best];
            O.d[u] = bd;
        }
        nu += tot;
    }
    con_sync<T>();
    int nj = 0;
    for (int i0 = 0; i0 < nu; i0 += T) {
        const int i = i0 + tid;
        const bool head = i < nu && (i == 0 || O.b[o + i] != O.b[o + i - 1]);
        const int c = head ? compress_group<false>(o + i, o + nu, O, 0) : 0;
        const int jo = o + nj + con_scan<T>(c, tid, ws, tot);
        if (head) {
            compress_group<true>(o + i, o + nu, O, jo);
            uf_unite(O.parent, a, O.b[o + i]);
        }
        nj += tot;
    }
    for (int w = 16; w > 0; w >>= 1) km = min(km, __shfl_xor_sync(0xffffffffu, km, w));
    if constexpr (T == 32) {
        if (tid == 0) O.kmin[a] = km;
    } else {
        if ((tid & 31) == 0) atomicMin(&O.kmin[a], km);
    }
    if (tid == 0) O.counts[a] = (int64_t)nu | ((int64_t)nj << 32);
    con_sync<T>();
}

__global__ void __launch_bounds__(kConWarps * 32) k_contacts(int n, const int32_t* __restrict__ ofs, RawContacts raw, ContactOut O,
                                                             int32_t* __restrict__ list, int32_t* n_list) {
    __shared__ uint64_t sk[kConWarps][kConWarpCap];
    __shared__ int32_t si[kConWarps][kConWarpCap];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int a = blockIdx.x * kConWarps + warp; a < n; a += gridDim.x * kConWarps) {
        const int o = ofs[a], L = ofs[a + 1] - o;
        if (L == 0 || L > kConWarpCap) {
            if (lane == 0) {
                O.kmin[a] = ~0ull;
                O.counts[a] = 0;
                if (L) list[atomicAdd(n_list, 1)] = a;
            }
            continue;
        }
        contacts_of<32>(a, o, L, raw, O, sk[warp], si[warp], lane, nullptr);
    }
}

__global__ void __launch_bounds__(kConCtaThreads) k_contacts_cta(const int32_t* __restrict__ ofs, RawContacts raw, ContactOut O,
                                                                 const int32_t* __restrict__ list, const int32_t* n_list) {
    __shared__ uint64_t sk[kConCtaCap];
    __shared__ int32_t si[kConCtaCap];
    __shared__ int ws[kConCtaThreads / 32];
    const int nl = *n_list;
    for (int q = blockIdx.x; q < nl; q += gridDim.x) {
        const int a = list[q], o = ofs[a], L = ofs[a + 1] - o;
        const bool fits = L <= kConCtaCap;
        contacts_of<kConCtaThreads>(a, o, L, raw, O, fits ? sk : O.key + o, fits ? si : O.idx + o, threadIdx.x, ws);
    }
}

// Segments to the compact lists, four threads per CNT; the junctions' points are marked as elements.
constexpr int kEmitLanes = 4;
__global__ void k_contact_emit(int n, const int32_t* __restrict__ ofs, const int64_t* __restrict__ base, ContactOut O, int32_t* __restrict__ ua,
                               int32_t* __restrict__ ub, int32_t* __restrict__ upa, int32_t* __restrict__ upb, double* __restrict__ ud,
                               int32_t* __restrict__ jp1, int32_t* __restrict__ jn1, int32_t* __restrict__ jp2, int32_t* __restrict__ jn2,
                               double* __restrict__ jd, int32_t* __restrict__ mark, int32_t* __restrict__ has_junc) {
    const int lane = threadIdx.x % kEmitLanes;
    for (int a = (blockIdx.x * blockDim.x + threadIdx.x) / kEmitLanes; a < n; a += gridDim.x * blockDim.x / kEmitLanes) {
        const int64_t c = O.counts[a];
        const int o = ofs[a], nu = (int)(uint32_t)c, nj = (int)(c >> 32), uo = (int)(uint32_t)base[a], jo = (int)(base[a] >> 32);
        for (int t = lane; t < nu; t += kEmitLanes) {
            ua[uo + t] = a;
            ub[uo + t] = O.b[o + t];
            upa[uo + t] = O.pa[o + t];
            upb[uo + t] = O.pb[o + t];
            ud[uo + t] = O.d[o + t];
        }
        for (int t = lane; t < nj; t += kEmitLanes) {
            const int P1 = O.jp1[o + t], P2 = O.jp2[o + t], b = O.jn2[o + t];
            jp1[jo + t] = P1;
            jn1[jo + t] = a;
            jp2[jo + t] = P2;
            jn2[jo + t] = b;
            jd[jo + t] = O.jd[o + t];
            mark[P1] = 1;
            mark[P2] = 1;
            has_junc[a] = 1;
            has_junc[b] = 1;
        }
    }
}

// ---------------------------------------------------------------------------
// Labels.  Roots into a separate array so no thread ever reads a half-flattened parent[]; each
// cluster's first contact in scan order (one atomic per warp when its CNTs share a root: in a
// percolating network nearly all do, and one atomic per contact visit took 95-630 us).
__global__ void k_uf_flatten(int n, const int32_t* __restrict__ parent, const unsigned long long* __restrict__ kmin, int32_t* __restrict__ root,
                             unsigned long long* minkey) {
    const int step = gridDim.x * blockDim.x;
    for (int i0 = blockIdx.x * blockDim.x; i0 < n; i0 += step) {
        const int i = i0 + threadIdx.x;
        int r = -1;
        unsigned long long k = ~0ull;
        if (i < n) {
            r = uf_root(parent, i);
            root[i] = r;
            k = kmin[i];
        }
        const bool has = k != ~0ull;
        const unsigned m = __ballot_sync(0xffffffffu, has);
        if (!m) continue;
        const int r0 = __shfl_sync(0xffffffffu, r, __ffs(m) - 1);
        if (__all_sync(0xffffffffu, !has || r == r0)) {
            for (int w = 16; w > 0; w >>= 1) k = min(k, __shfl_xor_sync(0xffffffffu, k, w));
            if ((threadIdx.x & 31) == 0) atomicMin(&minkey[r0], k);
        } else if (has) {
            atomicMin(&minkey[r], k);
        }
    }
}

// The upstream label of a cluster is the rank of its first contact in scan
// order (HK76 creates labels in scan order and Merge_labels keeps the smaller
// root, Hoshen_Kopelman.cpp:2908-2989; Cleanup_labels renumbers roots in
// ascending order, :374-425).
__global__ void k_root_flags(int n, const int32_t* __restrict__ root, const unsigned long long* __restrict__ minkey,
                             int32_t* __restrict__ flag) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        flag[i] = (root[i] == i && minkey[i] != ~0ull) ? 1 : 0;
}

__global__ void k_root_keys(int n, const int32_t* __restrict__ flag, const int32_t* __restrict__ scan,
                            const unsigned long long* __restrict__ minkey, uint64_t* __restrict__ keys, uint32_t* __restrict__ vals,
                            int32_t* __restrict__ rank) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (flag[i]) {
            keys[scan[i]] = minkey[i];
            vals[scan[i]] = (uint32_t)i;
            rank[i] = 0;
        }
}

// Ranks of the *count keys (all different): each block compares 256 of them with a tile of 1,024
// and adds the smaller ones.  Quadratic, but a launch of a few microseconds for the thousands of
// labels a network has (a one-CTA radix sort of 64-bit keys took 15-60 us and a host read of the
// count); used up to kRankMax CNTs.
constexpr int kRankMax = 60000;
constexpr int kRankTile = 1024;
__global__ void __launch_bounds__(256) k_root_rank(const int32_t* __restrict__ count, const uint64_t* __restrict__ keys,
                                                   const uint32_t* __restrict__ vals, int32_t* rank) {
    __shared__ uint64_t tile[kRankTile];
    const int L = *count;
    const int nx = (L + 255) / 256, ny = (L + kRankTile - 1) / kRankTile;
    for (long long w = blockIdx.x; w < (long long)nx * ny; w += gridDim.x) {
        const int i = (int)(w % nx) * 256 + threadIdx.x, t0 = (int)(w / nx) * kRankTile, m = min(kRankTile, L - t0);
        for (int t = threadIdx.x; t < m; t += 256) tile[t] = keys[t0 + t];
        __syncthreads();
        if (i < L) {
            const uint64_t k = keys[i];
            int r = 0;
            for (int t = 0; t < m; t++) r += tile[t] < k ? 1 : 0;
            if (ny == 1) rank[vals[i]] = r;
            else atomicAdd(&rank[vals[i]], r);
        }
        __syncthreads();
    }
}

__global__ void k_sorted_rank(int n, const uint32_t* __restrict__ vals, int32_t* __restrict__ rank) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) rank[vals[i]] = i;
}

// Labels, and the end points of CNTs with a junction marked as elements (Complete_cnt_elements,
// Hoshen_Kopelman.cpp:557-572).
__global__ void k_labels(int n, const int32_t* __restrict__ root, const unsigned long long* __restrict__ minkey,
                         const int32_t* __restrict__ rank, const int32_t* __restrict__ has_junc, const int32_t* __restrict__ cstart,
                         const int32_t* __restrict__ clen, int32_t* __restrict__ labels, int32_t* __restrict__ mark) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int r = root[i];
        labels[i] = (minkey[r] != ~0ull) ? rank[r] : -1;
        if (has_junc[i] && clen[i] > 0) {
            mark[cstart[i]] = 1;
            mark[cstart[i] + clen[i] - 1] = 1;
        }
    }
}

// ---------------------------------------------------------------------------
// Percolation (Hoshen_Kopelman.cpp:2366-2589): faces {2,4} x, {3,5} y, {0,1} z.
__global__ void k_faces(const int32_t* __restrict__ bptr, const int32_t* __restrict__ bidx, const int32_t* __restrict__ labels,
                        int32_t* face_bits) {
    for (int f = 0; f < 6; f++)
        for (int i = bptr[f] + blockIdx.x * blockDim.x + threadIdx.x; i < bptr[f + 1]; i += gridDim.x * blockDim.x) {
            const int L = labels[bidx[i]];
            if (L != -1 && !(__ldcg(&face_bits[L]) >> f & 1)) atomicOr(&face_bits[L], 1 << f);
        }
}

__global__ void k_perc(int n, const int32_t* __restrict__ face_bits, int32_t* __restrict__ perc_bits, int32_t* __restrict__ flag) {
    for (int L = blockIdx.x * blockDim.x + threadIdx.x; L < n; L += gridDim.x * blockDim.x) {
        const int b = face_bits[L];
        const int p = ((b & 0x14) == 0x14 ? 1 : 0) | ((b & 0x28) == 0x28 ? 2 : 0) | ((b & 0x03) == 0x03 ? 4 : 0);
        perc_bits[L] = p;
        flag[L] = p != 0;
    }
}

// Directions of the percolated clusters, in label order: the first kHostFams for the host at once.
constexpr int kHostFams = 8;
__global__ void k_families(int n, const int32_t* __restrict__ perc_bits, const int32_t* __restrict__ perc_index, int32_t* __restrict__ out,
                           int32_t* __restrict__ host) {
    for (int L = blockIdx.x * blockDim.x + threadIdx.x; L < n; L += gridDim.x * blockDim.x)
        if (perc_bits[L]) {
            out[perc_index[L]] = perc_bits[L];
            if (perc_index[L] < kHostFams) host[perc_index[L]] = perc_bits[L];
        }
}

// One percolated cluster: members (cnts_inside order, Make_particle_clusters :2331-2363) and its
// junctions (Group_junctions_same_particle, :2686-2710) flagged in one array, scanned at once.
__global__ void k_one_cluster_flags(int n_inside, int nj_max, const int32_t* __restrict__ nj, const int32_t* __restrict__ inside, const int32_t* __restrict__ jn1,
                                    const int32_t* __restrict__ labels, const int32_t* __restrict__ perc_bits, int32_t* __restrict__ flag) {
    const int n = n_inside + *nj;  // the flags up to n_inside + nj_max are cleared past it
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n_inside + nj_max; i += gridDim.x * blockDim.x) {
        const int L = i < n ? labels[i < n_inside ? inside[i] : jn1[i - n_inside]] : -1;
        flag[i] = (L >= 0 && perc_bits[L] != 0) ? 1 : 0;
    }
}

__global__ void k_one_cluster_lists(int n_inside, int nj_max, const int32_t* __restrict__ inside, const int32_t* __restrict__ flag,
                                    const int32_t* __restrict__ scan, int32_t* __restrict__ clu, int32_t* __restrict__ cj,
                                    int32_t* __restrict__ counts) {
    const int before = scan[n_inside];  // members: the flags ahead of the junctions'
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_inside + nj_max; i += gridDim.x * blockDim.x)
        if (flag[i]) {
            if (i < n_inside) clu[scan[i]] = inside[i];
            else cj[scan[i] - before] = i - n_inside;
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        counts[0] = before;
        counts[1] = scan[n_inside + nj_max] - before;
    }
}

// Percolated clusters in cnts_inside order (Make_particle_clusters :2331-2363,
// Determine_family_of_percolated_clusters :2524-2589).
__global__ void k_cluster_members(int n_inside, const int32_t* __restrict__ inside, const int32_t* __restrict__ labels,
                                  const int32_t* __restrict__ perc_bits, const int32_t* __restrict__ perc_index,
                                  int bits_rank, int32_t* __restrict__ flag, uint64_t* __restrict__ key) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_inside; i += gridDim.x * blockDim.x) {
        int L = labels[inside[i]];
        bool in = (L >= 0) && perc_bits[L] != 0;
        flag[i] = in ? 1 : 0;
        key[i] = in ? (((uint64_t)perc_index[L] << bits_rank) | (uint64_t)i) : 0;
    }
}

// Group_junctions_same_particle (Hoshen_Kopelman.cpp:2686-2710).
__global__ void k_junction_members(int nj, const int32_t* __restrict__ jn1, const int32_t* __restrict__ labels,
                                   const int32_t* __restrict__ perc_bits, const int32_t* __restrict__ perc_index, int bits_j,
                                   int32_t* __restrict__ flag, uint64_t* __restrict__ key) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nj; i += gridDim.x * blockDim.x) {
        int L = labels[jn1[i]];
        bool in = (L >= 0) && perc_bits[L] != 0;
        flag[i] = in ? 1 : 0;
        key[i] = in ? (((uint64_t)perc_index[L] << bits_j) | (uint64_t)i) : 0;
    }
}

__global__ void k_compact_kv(int n, const int32_t* __restrict__ flag, const int32_t* __restrict__ scan, const uint64_t* __restrict__ kin,
                             uint64_t* __restrict__ kout, uint32_t* __restrict__ vout) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (flag[i]) {
            kout[scan[i]] = kin[i];
            vout[scan[i]] = (uint32_t)i;
        }
}

// CSR from keys sorted by (group << shift | member): counts per group and the member ids.
__global__ void k_group_count(int n, const uint64_t* __restrict__ keys, int shift, int32_t* __restrict__ cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) atomicAdd(&cnt[keys[i] >> shift], 1);
}

__global__ void k_member_values(int n, const uint64_t* __restrict__ keys, uint64_t mask, const int32_t* __restrict__ map,
                                int32_t* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int m = (int)(keys[i] & mask);
        out[i] = map ? map[m] : m;
    }
}

int grid_for(long long n, int threads = 256) {
    long long b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148LL * 32) b = 148LL * 32;
    return (int)b;
}

}  // namespace

Ctx::~Ctx() {
    for (auto* s : systems) delete s;
    for (auto* s : sys_pool) delete s;
    delete hy;
}

namespace {
struct WordPages {
    static constexpr int kSlots = 32;
    struct Page {
        int64_t* p;
        uint32_t used;
    };
    std::mutex m;
    std::vector<Page> pages;
};
WordPages& word_pages() {
    static WordPages* w = new WordPages;  // not destroyed: a context may outlive static objects
    return *w;
}
}  // namespace

int64_t* host_words_take() {
    WordPages& w = word_pages();
    std::lock_guard<std::mutex> lock(w.m);
    for (auto& g : w.pages)
        for (int k = 0; k < WordPages::kSlots; k++)
            if (!(g.used >> k & 1)) {
                g.used |= 1u << k;
                return g.p + (size_t)k * W_COUNT;
            }
    w.pages.reserve(w.pages.size() + 1);
    int64_t* p = nullptr;
    CICY_CUDA(cudaHostAlloc(&p, sizeof(int64_t) * W_COUNT * WordPages::kSlots, cudaHostAllocMapped | cudaHostAllocPortable));
    w.pages.push_back(WordPages::Page{p, 1u});
    return p;
}

void host_words_return(int64_t* slot) {
    WordPages& w = word_pages();
    std::lock_guard<std::mutex> lock(w.m);
    for (size_t i = 0; i < w.pages.size(); i++) {
        WordPages::Page& g = w.pages[i];
        if (slot < g.p || slot >= g.p + (size_t)W_COUNT * WordPages::kSlots) continue;
        g.used &= ~(1u << ((slot - g.p) / W_COUNT));
        if (!g.used && w.pages.size() > 1) {
            cudaFreeHost(g.p);
            w.pages.erase(w.pages.begin() + i);
        }
        return;
    }
}

int32_t read_i32(Ctx& c, const int32_t* dptr) {
    CICY_CUDA(cudaMemcpyAsync(c.words.host + W_READ, dptr, sizeof(int32_t), cudaMemcpyDeviceToHost, c.stream));
    CICY_CUDA(cudaStreamSynchronize(c.stream));
    return *reinterpret_cast<const int32_t*>(c.words.host + W_READ);
}

void check_status(Ctx& c, const char* where) {
    CICY_CUDA(cudaMemcpyAsync(c.words.host + W_STATUS, c.status.get(), sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    CICY_CUDA(cudaStreamSynchronize(c.stream));
    const int st = *reinterpret_cast<const int*>(c.words.host + W_STATUS);
    if (st == DEV_OK) return;
    CICY_CUDA(cudaMemsetAsync(c.status.get(), 0, sizeof(int), c.stream));
    if (st == DEV_TIMEOUT) throw Fail{CICY_E_TIMEOUT, std::string(where) + ": a bounded device wait gave up"};
    if (st == DEV_CAPACITY) throw Fail{CICY_E_CAPACITY, std::string(where) + ": a grid region holds more than 8192 points"};
    if (st == DEV_ZERO_DIAG) throw Fail{CICY_E_ZERO_DIAGONAL, std::string(where) + ": zero on the stiffness diagonal"};
    throw Fail{CICY_E_INTERNAL, std::string(where) + ": device status " + std::to_string(st)};
}

// ---------------------------------------------------------------------------
void upload_network(Ctx& c, const cicy_network& n) {
    if (n.n_points < 0 || n.n_cnts < 0 || n.n_inside < 0 || !n.structure_ptr || !n.radii)
        throw Fail{CICY_E_INPUT, "cicy_upload_network: missing arrays"};
    if (n.n_points >= (1LL << 31) - 1) throw Fail{CICY_E_CAPACITY, "cicy_upload_network: 2^31 or more points"};
    cudaStream_t s = c.stream;
    c.stage = 0;  // no network until the upload is complete
    c.n_points = (int)n.n_points;
    c.n_cnts = n.n_cnts;
    c.n_inside = n.n_inside;
    c.window = n.window;
    // structure lists -> (start, length) runs of consecutive point ids
    c.h_cstart.assign(n.n_cnts, 0);
    c.h_clen.assign(n.n_cnts, 0);
    for (int i = 0; i < n.n_cnts; i++) {
        int64_t b = n.structure_ptr[i], e = n.structure_ptr[i + 1];
        if (e < b) throw Fail{CICY_E_INPUT, "cicy_upload_network: structure_ptr not ascending"};
        if (e > b) {
            int64_t p0 = n.structure_idx[b];
            if (p0 < 0 || p0 + (e - b) > n.n_points) throw Fail{CICY_E_INPUT, "cicy_upload_network: point id out of range"};
            for (int64_t k = b + 1; k < e; k++)
                if (n.structure_idx[k] != n.structure_idx[k - 1] + 1)
                    throw Fail{CICY_E_INPUT, "cicy_upload_network: CNT " + std::to_string(i) + " is not a run of consecutive point ids"};
            c.h_cstart[i] = (int32_t)p0;
        }
        c.h_clen[i] = (int32_t)(e - b);
    }
    c.r_max = 0;
    for (int i = 0; i < n.n_cnts; i++) c.r_max = std::fmax(c.r_max, n.radii[i]);
    std::vector<int32_t> trav_off(n.n_inside + 1, 0);
    for (int i = 0; i < n.n_inside; i++) {
        int ci = n.cnts_inside[i];
        if (ci < 0 || ci >= n.n_cnts) throw Fail{CICY_E_INPUT, "cicy_upload_network: cnts_inside out of range"};
        trav_off[i + 1] = trav_off[i] + c.h_clen[ci];
    }
    c.n_trav = trav_off[n.n_inside];
    c.h_bcnt_ptr.assign(7, 0);
    c.h_bpts_ptr.assign(7, 0);
    if (n.boundary_cnt_ptr)
        for (int f = 0; f < 7; f++) c.h_bcnt_ptr[f] = (int32_t)n.boundary_cnt_ptr[f];
    if (n.boundary_pts_ptr)
        for (int f = 0; f < 7; f++) c.h_bpts_ptr[f] = (int32_t)n.boundary_pts_ptr[f];
    std::vector<int32_t> bpts(c.h_bpts_ptr[6]);
    for (int i = 0; i < c.h_bpts_ptr[6]; i++) bpts[i] = (int32_t)n.boundary_pts_idx[i];

    const size_t np = std::max<int64_t>(n.n_points, 1), nc = std::max(n.n_cnts, 1);
    c.x.ensure(np); c.y.ensure(np); c.z.ensure(np); c.flag.ensure(np);
    c.radii.ensure(nc); c.cstart.ensure(nc); c.clen.ensure(nc);
    c.inside.ensure(std::max(n.n_inside, 1));
    c.trav_off.ensure(n.n_inside + 1);
    c.bcnt_ptr.ensure(7); c.bpts_ptr.ensure(7);
    c.bcnt_idx.ensure(std::max(c.h_bcnt_ptr[6], 1));
    c.bpts_idx.ensure(std::max(c.h_bpts_ptr[6], 1));
    c.status.ensure(1);
    c.i32_scalar.ensure(8);
    auto up = [&](void* d, const void* h, size_t bytes) {
        if (bytes) CICY_CUDA(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s));
    };
    up(c.x.get(), n.x, sizeof(double) * n.n_points);
    up(c.y.get(), n.y, sizeof(double) * n.n_points);
    up(c.z.get(), n.z, sizeof(double) * n.n_points);
    up(c.flag.get(), n.flag, sizeof(int32_t) * n.n_points);
    up(c.radii.get(), n.radii, sizeof(double) * n.n_cnts);
    up(c.cstart.get(), c.h_cstart.data(), sizeof(int32_t) * n.n_cnts);
    up(c.clen.get(), c.h_clen.data(), sizeof(int32_t) * n.n_cnts);
    up(c.inside.get(), n.cnts_inside, sizeof(int32_t) * n.n_inside);
    up(c.trav_off.get(), trav_off.data(), sizeof(int32_t) * (n.n_inside + 1));
    up(c.bcnt_ptr.get(), c.h_bcnt_ptr.data(), sizeof(int32_t) * 7);
    up(c.bpts_ptr.get(), c.h_bpts_ptr.data(), sizeof(int32_t) * 7);
    up(c.bcnt_idx.get(), n.boundary_cnt_idx, sizeof(int32_t) * c.h_bcnt_ptr[6]);
    up(c.bpts_idx.get(), bpts.data(), sizeof(int32_t) * c.h_bpts_ptr[6]);
    CICY_CUDA(cudaMemsetAsync(c.status.get(), 0, sizeof(int), s));
    CICY_CUDA(cudaStreamSynchronize(s));
    c.stage = 1;
    c.have_backbone = false;
    c.have_volumes = false;
    c.have_hybrid = false;
}

// ---------------------------------------------------------------------------
void run_contact_grid(Ctx& c, const cicy_params& p, bool wait) {
    if (c.stage < 1) throw Fail{CICY_E_STATE, "cicy_contact_grid: no network uploaded"};
    cudaStream_t s = c.stream;
    CICY_TRACE("contact_grid", s);
    const cicy_cuboid& w = c.window;
    // Generate_contact_grid + Adjust_regions_if_needed (Contact_grid.cpp:18-102)
    GridGeom g{};
    g.n[0] = std::max(1, (int)(w.len_x / p.gs_min[0]));
    g.n[1] = std::max(1, (int)(w.len_y / p.gs_min[1]));
    g.n[2] = std::max(1, (int)(w.len_z / p.gs_min[2]));
    g.l[0] = p.gs_min[0]; g.l[1] = p.gs_min[1]; g.l[2] = p.gs_min[2];
    const double max_ov = std::max(p.gs_overlap_cnt, p.gs_overlap_gnp);
    const double lens[3] = {w.len_x, w.len_y, w.len_z};
    for (int a = 0; a < 3; a++)
        if (p.gs_min[a] < 2 * max_ov) {
            g.l[a] = 2.0 * (max_ov + kZero);
            g.n[a] = 1 + (int)(lens[a] / g.l[a]);
        }
    g.min[0] = w.min_x; g.min[1] = w.min_y; g.min[2] = w.min_z;
    g.overlap = p.gs_overlap_cnt;
    g.total = (long long)g.n[0] * g.n[1] * g.n[2];
    if (g.total <= 0) throw Fail{CICY_E_INPUT, "Generate_contact_grid: invalid number of subregions"};
    if (g.total >= (1LL << 31) - 2 || g.total >= (1LL << 38)) throw Fail{CICY_E_CAPACITY, "Generate_contact_grid: too many regions"};
    const int R = (int)g.total;
    c.stage = 1;  // no grid until this one is complete
    c.grid = g;
    c.region_cnt.ensure(R + 1);
    c.region_ptr.ensure(R + 1);
    c.trav_pt.ensure(std::max(c.n_trav, 1));
    Carver v{};
    v.take<int4>(c.n_trav);
    v.take<ushort4>(c.n_trav);
    c.trav_reg.ensure(std::max<size_t>(v.at, 1));
    v = Carver{c.trav_reg.get()};
    int4* const trav_reg = v.take<int4>(c.n_trav);
    ushort4* const trav_rank = v.take<ushort4>(c.n_trav);
    CICY_CUDA(cudaMemsetAsync(c.region_cnt.get(), 0, sizeof(int32_t) * (R + 1), s));
    if (c.n_trav > 0) {
        k_grid_count<<<grid_for(c.n_trav), 256, 0, s>>>(c.n_trav, c.trav_off.get(), c.n_inside, c.inside.get(), c.cstart.get(),
                                                      c.x.get(), c.y.get(), c.z.get(), g, c.trav_pt.get(), c.region_cnt.get(),
                                                      trav_reg, trav_rank);
        c.launches++;
    }
    exclusive_scan_i32(c.region_cnt.get(), c.region_ptr.get(), R + 1, reinterpret_cast<int32_t*>(c.words.dev + W_READ), c.scan_tmp32, s,
                       c.launches);
    CICY_CUDA(cudaStreamSynchronize(s));
    c.n_slots = *reinterpret_cast<const int32_t*>(c.words.host + W_READ);
    const int S = c.n_slots;
    c.slot_q.ensure(std::max(S, 1));
    c.slot_sorted.ensure(std::max(S, 1));
    c.slot_region.ensure(std::max(S, 1));
    c.seg_large.ensure(R + 1);
    if (c.n_trav > 0) {
        k_grid_scatter<<<grid_for(c.n_trav), 256, 0, s>>>(c.n_trav, trav_reg, trav_rank, c.region_ptr.get(), c.slot_q.get());
        c.launches++;
    }
    segmented_sort_u32(c.region_ptr.get(), R, c.slot_q.get(), c.slot_sorted.get(), c.slot_region.get(), c.seg_large.get(),
                       c.i32_scalar.get() + 1, c.status.get(), s, c.launches);
    CICY_LAUNCH_CHECK();
    if (wait) check_status(c, "Generate_contact_grid");
    c.stage = 2;
}

// ---------------------------------------------------------------------------
void run_clusters(Ctx& c, const cicy_params& p) {
    if (c.stage < 2) throw Fail{CICY_E_STATE, "cicy_clusters: run cicy_contact_grid first"};
    cudaStream_t s = c.stream;
    CICY_TRACE("clusters", s);
    TraceSeq tr(s);
    const int S = c.n_slots, nc = c.n_cnts, NC = std::max(nc, 1), NP = std::max(c.n_points, 1);
    const int bp = bits_for((uint64_t)NP), bc = bits_for((uint64_t)NC);
    if (bp + 2 * bc > 64) throw Fail{CICY_E_CAPACITY, "too many points/CNTs for the 64-bit contact key"};
    // device words of this stage, copied to the host together
    enum { C_RAW = 0, C_LONG = 1, C_LABELS = 2, C_PERC = 3, C_FAM = 4, C_ONE = C_FAM + kHostFams, C_UJ = C_ONE + 2, C_WORDS = C_UJ + 2 };
    static_assert(C_UJ % 2 == 0 && C_WORDS * sizeof(int32_t) <= (W_COUNT - W_CLU) * sizeof(int64_t), "host words");
    c.clu_words.ensure(C_WORDS);
    int32_t* dw = c.clu_words.get();
    const int32_t* hw = reinterpret_cast<const int32_t*>(c.words.host + W_CLU);
    c.parent.ensure(NC); c.minkey.ensure(NC); c.uf_root.ensure(NC); c.labels.ensure(NC); c.root_rank.ensure(NC);
    c.face_bits.ensure(NC); c.perc_bits.ensure(NC); c.perc_index.ensure(NC + 1); c.perc_fam.ensure(NC); c.has_junc.ensure(NC);
    int32_t *con_cnt, *con_ofs, *con_long;
    int64_t *con_uj, *con_base;
    unsigned long long* kmin;
    auto lay = [&](Carver v) {
        for (int64_t** q : {&con_uj, &con_base}) *q = v.take<int64_t>(NC);
        kmin = v.take<unsigned long long>(NC);
        for (int32_t** q : {&con_cnt, &con_ofs, &con_long}) *q = v.take<int32_t>(NC + 1);
        return v.at;
    };
    c.con_of_cnt.ensure(lay(Carver{}));
    lay(Carver{c.con_of_cnt.get()});
    c.mark.ensure(NP + 1); c.mark_scan.ensure(NP + 1);
    // ---- pair tests ----
    PairGeom pg{};
    pg.min[0] = c.window.min_x; pg.min[1] = c.window.min_y; pg.min[2] = c.window.min_z;
    const double extent = std::max({c.window.len_x, c.window.len_y, c.window.len_z});
    pg.far = (float)(4.0 * extent);
    // cutoff of the largest CNTs, plus what rounding two positions below 4 extents to 24 bits can take off their distance
    const double cut = std::max(p.tunneling_dist + 2.0 * c.r_max, 0.0), margin = 1e-6 * (extent + cut);
    pg.cut2 = (float)((cut + margin) * (cut + margin) * (1.0 + 1e-6));
    pg.vdw = p.van_der_waals_dist;
    pg.tunnel = p.tunneling_dist;
    int cap = std::max(1 << 16, S / 4);
    RawContacts raw{};
    raw.count = dw + C_RAW;
    raw.per_cnt = con_cnt;
    for (int attempt = 0; attempt < 2; attempt++) {
        raw.cap = cap;
        c.con_raw.ensure(raw.lay(Carver{}));
        raw.lay(Carver{c.con_raw.get()});
        CICY_CUDA(cudaMemsetAsync(dw, 0, sizeof(int32_t) * C_WORDS, s));
        k_cnt_init<<<grid_for(nc + 1), 256, 0, s>>>(nc, c.parent.get(), c.minkey.get(), con_cnt, c.face_bits.get(), c.has_junc.get());
        if (S > 0) {
            k_pairs<<<ceil_div(S, kPairTile), kPairThreads, 0, s>>>(S, pg, c.region_ptr.get(), c.slot_region.get(), c.slot_sorted.get(),
                                                                    c.trav_pt.get(), c.x.get(), c.y.get(), c.z.get(), c.flag.get(),
                                                                    c.radii.get(), c.status.get(), raw);
            c.launches++;
        }
        c.launches++;
        exclusive_scan_i32(con_cnt, con_ofs, nc + 1, nullptr, c.scan_tmp32, s, c.launches);
        CICY_LAUNCH_CHECK();
        CICY_CUDA(cudaMemcpyAsync(c.words.host + W_CLU, dw, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        c.stage = 1;  // a grid that failed is not used again
        check_status(c, "Generate_contact_grid");  // also waits for the count
        c.stage = 2;
        c.n_raw = hw[C_RAW];
        if (c.n_raw <= cap) break;
        cap = c.n_raw + c.n_raw / 8 + 1024;
        if (attempt == 1) throw Fail{CICY_E_INTERNAL, "contact buffer overflow"};
    }
    const int NR = c.n_raw, NR1 = std::max(NR, 1);
    tr.mark("clusters.pairs");
    // ---- point_contacts, junctions, unions (every list is at most as long as the visits) ----
    ContactOut co{};
    co.counts = con_uj;
    co.kmin = kmin;
    co.parent = c.parent.get();
    co.min_points = p.min_points;
    c.con_seg.ensure(co.lay(Carver{}, NR1));
    co.lay(Carver{c.con_seg.get()}, NR1);
    c.uc_a.ensure(NR1); c.uc_b.ensure(NR1); c.uc_pa.ensure(NR1); c.uc_pb.ensure(NR1); c.uc_d.ensure(NR1);
    c.j_p1.ensure(NR1); c.j_n1.ensure(NR1); c.j_p2.ensure(NR1); c.j_n2.ensure(NR1); c.j_d.ensure(NR1);
    CICY_CUDA(cudaMemsetAsync(c.mark.get(), 0, sizeof(int32_t) * (NP + 1), s));
    k_raw_place<<<grid_for(NR), 256, 0, s>>>(NR, raw, con_ofs, co.perm);
    k_contacts<<<grid_for(32LL * nc, kConWarps * 32), kConWarps * 32, 0, s>>>(nc, con_ofs, raw, co, con_long, dw + C_LONG);
    k_contacts_cta<<<148 * 4, kConCtaThreads, 0, s>>>(con_ofs, raw, co, con_long, dw + C_LONG);
    exclusive_scan_i64(con_uj, con_base, nc, reinterpret_cast<int64_t*>(dw + C_UJ), c.scan_tmp64, s, c.launches);
    k_contact_emit<<<grid_for((long long)nc * kEmitLanes), 256, 0, s>>>(
        nc, con_ofs, con_base, co, c.uc_a.get(), c.uc_b.get(), c.uc_pa.get(), c.uc_pb.get(), c.uc_d.get(), c.j_p1.get(),
        c.j_n1.get(), c.j_p2.get(), c.j_n2.get(), c.j_d.get(), c.mark.get(), c.has_junc.get());
    c.launches += 4;
    tr.mark("clusters.contacts");
    // ---- labels ----
    c.sort_k.ensure(NC + 1);
    c.sort_v.ensure(NC + 1);
    c.flags.ensure((size_t)std::max((long long)NC, (long long)c.n_inside + NR) + 1);
    c.flags_scan.ensure((size_t)std::max((long long)NC, (long long)c.n_inside + NR) + 1);
    k_uf_flatten<<<grid_for(nc), 256, 0, s>>>(nc, c.parent.get(), kmin, c.uf_root.get(), c.minkey.get());
    k_root_flags<<<grid_for(nc), 256, 0, s>>>(nc, c.uf_root.get(), c.minkey.get(), c.flags.get());
    exclusive_scan_i32(c.flags.get(), c.flags_scan.get(), nc, dw + C_LABELS, c.scan_tmp32, s, c.launches);
    k_root_keys<<<grid_for(nc), 256, 0, s>>>(nc, c.flags.get(), c.flags_scan.get(), c.minkey.get(), c.sort_k.get(), c.sort_v.get(),
                                             c.root_rank.get());
    if (nc <= kRankMax) {
        k_root_rank<<<148 * 4, 256, 0, s>>>(dw + C_LABELS, c.sort_k.get(), c.sort_v.get(), c.root_rank.get());
    } else {
        const int nl = read_i32(c, dw + C_LABELS);
        radix_sort_pairs(c.sort_k.get(), c.sort_v.get(), nl, bits_for((uint64_t)c.grid.total) + 26, c.rs, s, c.launches);
        k_sorted_rank<<<grid_for(nl), 256, 0, s>>>(nl, c.sort_v.get(), c.root_rank.get());
    }
    k_labels<<<grid_for(nc), 256, 0, s>>>(nc, c.uf_root.get(), c.minkey.get(), c.root_rank.get(), c.has_junc.get(), c.cstart.get(), c.clen.get(),
                                          c.labels.get(), c.mark.get());
    c.launches += 5;
    tr.mark("clusters.labels");
    // ---- elements: marked points in order (junction points and the ends of CNTs with junctions) ----
    c.elem_idx.ensure((size_t)std::max(1LL, std::min((long long)c.n_points, 2LL * NR + 2LL * nc)));
    exclusive_scan_flags_i32(c.mark.get(), c.mark_scan.get(), c.n_points + 1, nullptr, c.elem_idx.get(), c.scan_tmp32, s, c.launches);
    tr.mark("clusters.elements");
    // ---- percolation and families; lists of one percolated cluster ----
    c.clu_idx.ensure(std::max(c.n_inside, 1));
    c.cj_idx.ensure(NR1);
    if (c.h_bcnt_ptr[6] > 0) {
        k_faces<<<grid_for(c.h_bcnt_ptr[6]), 256, 0, s>>>(c.bcnt_ptr.get(), c.bcnt_idx.get(), c.labels.get(), c.face_bits.get());
        c.launches++;
    }
    k_perc<<<grid_for(nc), 256, 0, s>>>(nc, c.face_bits.get(), c.perc_bits.get(), c.flags.get());
    exclusive_scan_i32(c.flags.get(), c.perc_index.get(), nc, dw + C_PERC, c.scan_tmp32, s, c.launches);
    k_families<<<grid_for(nc), 256, 0, s>>>(nc, c.perc_bits.get(), c.perc_index.get(), c.perc_fam.get(), dw + C_FAM);
    k_one_cluster_flags<<<grid_for((long long)c.n_inside + NR), 256, 0, s>>>(c.n_inside, NR, dw + C_UJ + 1, c.inside.get(), c.j_n1.get(),
                                                                             c.labels.get(), c.perc_bits.get(), c.flags.get());
    exclusive_scan_i32(c.flags.get(), c.flags_scan.get(), c.n_inside + NR + 1, nullptr, c.scan_tmp32, s, c.launches);
    k_one_cluster_lists<<<grid_for((long long)c.n_inside + NR), 256, 0, s>>>(c.n_inside, NR, c.inside.get(), c.flags.get(), c.flags_scan.get(),
                                                                             c.clu_idx.get(), c.cj_idx.get(), dw + C_ONE);
    c.launches += 4;
    CICY_CUDA(cudaMemcpyAsync(c.words.host + W_CLU, dw, sizeof(int32_t) * C_WORDS, cudaMemcpyDeviceToHost, s));
    CICY_CUDA(cudaStreamSynchronize(s));
    c.n_uc = hw[C_UJ];
    c.n_junc = hw[C_UJ + 1];
    c.n_labels = hw[C_LABELS];
    c.n_perc = hw[C_PERC];
    const int NJ = c.n_junc;
    // families in percolated order (Family_map, Hoshen_Kopelman.cpp:2591-2622)
    c.h_family.resize(c.n_perc);
    static const int fam_of_bits[8] = {-1, 0, 1, 3, 2, 4, 5, 6};
    std::vector<int32_t> bits(hw + C_FAM, hw + C_FAM + std::min(c.n_perc, kHostFams));
    if (c.n_perc > kHostFams) {
        bits.resize(c.n_perc);
        CICY_CUDA(cudaMemcpyAsync(bits.data(), c.perc_fam.get(), sizeof(int32_t) * c.n_perc, cudaMemcpyDeviceToHost, s));
        CICY_CUDA(cudaStreamSynchronize(s));
    }
    for (int k = 0; k < c.n_perc; k++) c.h_family[k] = fam_of_bits[bits[k]];
    tr.mark("clusters.percolation");
    // percolated clusters (CNTs in cnts_inside order) and their junctions
    const int NP_ = std::max(c.n_perc, 1);
    c.clu_ptr.ensure(NP_ + 1); c.cj_ptr.ensure(NP_ + 1);
    c.h_clu_ptr.assign(c.n_perc + 1, 0);
    c.h_cj_ptr.assign(c.n_perc + 1, 0);
    if (c.n_perc == 1) {
        c.h_clu_ptr[1] = hw[C_ONE];
        c.h_cj_ptr[1] = hw[C_ONE + 1];
    } else if (c.n_perc > 1) {
        // several clusters: the lists ordered by cluster with a radix sort
        const int br = bits_for((uint64_t)std::max(c.n_inside, 1));
        const int longest = std::max(c.n_inside, NJ) + 1;
        c.work_i32a.ensure(c.n_perc + 1);
        c.sort_k.ensure(longest);
        c.sort_v.ensure(longest);
        DBuf<uint64_t> stage_keys;
        stage_keys.ensure(longest);
        k_cluster_members<<<grid_for(c.n_inside), 256, 0, s>>>(c.n_inside, c.inside.get(), c.labels.get(), c.perc_bits.get(),
                                                             c.perc_index.get(), br, c.flags.get(), stage_keys.get());
        exclusive_scan_i32(c.flags.get(), c.flags_scan.get(), c.n_inside, c.i32_scalar.get(), c.scan_tmp32, s, c.launches);
        k_compact_kv<<<grid_for(c.n_inside), 256, 0, s>>>(c.n_inside, c.flags.get(), c.flags_scan.get(), stage_keys.get(), c.sort_k.get(), c.sort_v.get());
        c.launches += 2;
        int nm = read_i32(c, c.i32_scalar.get());
        radix_sort_pairs(c.sort_k.get(), c.sort_v.get(), nm, br + bits_for((uint64_t)c.n_perc), c.rs, s, c.launches);
        CICY_CUDA(cudaMemsetAsync(c.work_i32a.get(), 0, sizeof(int32_t) * (c.n_perc + 1), s));
        k_group_count<<<grid_for(nm), 256, 0, s>>>(nm, c.sort_k.get(), br, c.work_i32a.get());
        exclusive_scan_i32(c.work_i32a.get(), c.clu_ptr.get(), c.n_perc + 1, nullptr, c.scan_tmp32, s, c.launches);
        k_member_values<<<grid_for(nm), 256, 0, s>>>(nm, c.sort_k.get(), (1ull << br) - 1, c.inside.get(), c.clu_idx.get());
        c.launches += 2;
        CICY_CUDA(cudaMemcpyAsync(c.h_clu_ptr.data(), c.clu_ptr.get(), sizeof(int32_t) * (c.n_perc + 1), cudaMemcpyDeviceToHost, s));
        // junctions
        const int bj = bits_for((uint64_t)std::max(NJ, 1));
        int njm = 0;
        if (NJ > 0) {
            k_junction_members<<<grid_for(NJ), 256, 0, s>>>(NJ, c.j_n1.get(), c.labels.get(), c.perc_bits.get(), c.perc_index.get(),
                                                          bj, c.flags.get(), stage_keys.get());
            exclusive_scan_i32(c.flags.get(), c.flags_scan.get(), NJ, c.i32_scalar.get(), c.scan_tmp32, s, c.launches);
            k_compact_kv<<<grid_for(NJ), 256, 0, s>>>(NJ, c.flags.get(), c.flags_scan.get(), stage_keys.get(), c.sort_k.get(), c.sort_v.get());
            c.launches += 2;
            njm = read_i32(c, c.i32_scalar.get());
            radix_sort_pairs(c.sort_k.get(), c.sort_v.get(), njm, bj + bits_for((uint64_t)c.n_perc), c.rs, s, c.launches);
        }
        CICY_CUDA(cudaMemsetAsync(c.work_i32a.get(), 0, sizeof(int32_t) * (c.n_perc + 1), s));
        if (njm > 0) {
            k_group_count<<<grid_for(njm), 256, 0, s>>>(njm, c.sort_k.get(), bj, c.work_i32a.get());
            k_member_values<<<grid_for(njm), 256, 0, s>>>(njm, c.sort_k.get(), (1ull << bj) - 1, nullptr, c.cj_idx.get());
            c.launches += 2;
        }
        exclusive_scan_i32(c.work_i32a.get(), c.cj_ptr.get(), c.n_perc + 1, nullptr, c.scan_tmp32, s, c.launches);
        CICY_CUDA(cudaMemcpyAsync(c.h_cj_ptr.data(), c.cj_ptr.get(), sizeof(int32_t) * (c.n_perc + 1), cudaMemcpyDeviceToHost, s));
        CICY_CUDA(cudaStreamSynchronize(s));
        stage_keys.release();
    }
    CICY_LAUNCH_CHECK();
    tr.mark("clusters.members");
    c.stage = 3;
    c.have_backbone = false;
    c.have_volumes = false;
    c.have_hybrid = false;
}

}  // namespace cicy
