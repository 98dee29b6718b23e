// The SES arrangement of a sphere set built on the device, in f64:
// active spheres in Morton order (geom/arrangement.rs:476-489), the cell
// grids (geom/cells.rs:27-84), containment (:497-514), neighbour rows
// (:522-545), the exposed intersection circles of each pair with their
// blockers and the exposed triple points (:674-752; as host/arrangement.cpp
// restates them), statuses, the rows of exposed spheres and the grids of
// circle centres and vertices (field/point.rs:235-270).
//
// Every value is the host build's bit for bit: the same f64 operations in
// the same order (no FMA contraction, IEEE division and square root), sets
// ordered by the same unique keys (stable radix sorts keep input order on
// equal keys, as the host's stable counting sort and pair sort do).  One
// decision uses a transcendental function: whether an angular gap between
// buried runs of a circle exceeds 1e-12 rad (atan2 of two crossing
// vectors).  The device's atan2 and the host's differ by a few ulps; a gap
// whose device value lies within 1e-13 rad of that threshold, or of the
// wrap at 0 / 2 pi, cannot be decided the same way with certainty, and the
// device then declines the whole build (the host builds it).  So does a
// circle with more candidate blockers than a warp keeps.  A sphere field
// (SAS or vdW) has the spheres, their grid and containment alone.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>

#include "common.cuh"
#include "kernels.hpp"
#include "sas.hpp"
#include "scan.cuh"

namespace smb {
namespace {

constexpr double S_EPS = 1e-9;           // arrangement.rs:26
constexpr double S_ANG_EPS = 1e-12;      // arrangement.rs:29
constexpr double S_PERIOD = 4.0;         // arrangement.rs:277
constexpr double S_PSEUDO_EPS = 1e-12;   // arrangement.rs:279
constexpr double S_TWO_PI = 6.283185307179586;
constexpr double S_ANG_MARGIN = 1e-13;   // device/host atan2 disagreement bound on a gap
// A gap between two runs clear of 0 and of the whole circle by this much in
// the diamond parameter is an angle clear of them by as much (the angle grows
// by 1 to 2 per unit of the parameter), so it is exposed without atan2.
constexpr double S_CLEAR_GAP = 1e-6;
constexpr int MAX_SPANS = 64;            // candidate blockers a warp keeps per circle
constexpr int RED_BLOCKS = 592;          // partial reductions
constexpr int C_WARPS = 4;               // warps a block in the circle passes

enum : uint32_t { DECLINE_ANGLE = 1, DECLINE_SPANS = 2 };

struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 operator+(D3 a, D3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3 operator-(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3 operator*(D3 a, double s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ D3 operator/(D3 a, double s) { return {a.x / s, a.y / s, a.z / s}; }
__device__ __forceinline__ double dotp(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 crossp(D3 a, D3 o) {
    return {a.y * o.z - a.z * o.y, a.z * o.x - a.x * o.z, a.x * o.y - a.y * o.x};
}
__device__ __forceinline__ double normp(D3 a) { return sqrt(dotp(a, a)); }
__device__ __forceinline__ double distp(D3 a, D3 b) { return normp(a - b); }
__device__ __forceinline__ D3 xyz(double4 v) { return {v.x, v.y, v.z}; }

__host__ __device__ __forceinline__ unsigned long long to_u64d(double v) {  // Rust's saturating cast
    if (!(v > 0.0)) return 0;
    return v >= 18446744073709551616.0 ? ~0ull : (unsigned long long)v;
}

__device__ __forceinline__ unsigned long long interleave(uint32_t v) {  // cells.rs:135-143
    unsigned long long x = (unsigned long long)v & 0x1fffff;
    x = (x | (x << 32)) & 0x001f00000000ffffULL;
    x = (x | (x << 16)) & 0x001f0000ff0000ffULL;
    x = (x | (x << 8)) & 0x100f00f00f00f00fULL;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ULL;
    x = (x | (x << 2)) & 0x1249249249249249ULL;
    return x;
}

// Bounding box (and, for spheres, the largest expanded radius and the
// count of spheres with r > 0) per block.
struct Box {
    double lo[3], hi[3], mx;
    unsigned long long cnt;
};

__device__ void box_reduce(Box b, Box* out) {
    __shared__ Box sh[256];
    sh[threadIdx.x] = b;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (int(threadIdx.x) < o) {
            Box& a = sh[threadIdx.x];
            const Box& c = sh[threadIdx.x + o];
            for (int k = 0; k < 3; k++) a.lo[k] = fmin(a.lo[k], c.lo[k]), a.hi[k] = fmax(a.hi[k], c.hi[k]);
            a.mx = fmax(a.mx, c.mx);
            a.cnt += c.cnt;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = sh[0];
}

__device__ __forceinline__ Box box_empty() {
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    return Box{{inf, inf, inf}, {-inf, -inf, -inf}, 0.0, 0};
}

// Active spheres (r > 0): centres' box, max(r + probe), count.
__global__ void k_box_active(const double* xyzr, size_t n, double probe, Box* out) {
    Box b = box_empty();
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const double* s = xyzr + 4 * i;
        if (!(s[3] > 0.0)) continue;
        for (int k = 0; k < 3; k++) b.lo[k] = fmin(b.lo[k], s[k]), b.hi[k] = fmax(b.hi[k], s[k]);
        b.mx = fmax(b.mx, s[3] + probe);
        b.cnt++;
    }
    box_reduce(b, out);
}

// Two sets of points at p + stride * i (blockIdx.y picks the set): box; mx =
// the largest word `wmax` of each point.
struct PointSet {
    const double* p;
    size_t stride, n;
    int wmax;
};
__global__ void k_box_points(PointSet s0, PointSet s1, Box* out) {
    const PointSet& P = blockIdx.y ? s1 : s0;
    Box b = box_empty();
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < P.n; i += size_t(gridDim.x) * blockDim.x) {
        const double* q = P.p + P.stride * i;
        for (int k = 0; k < 3; k++) b.lo[k] = fmin(b.lo[k], q[k]), b.hi[k] = fmax(b.hi[k], q[k]);
        if (P.wmax >= 0) b.mx = fmax(b.mx, q[P.wmax]);
        b.cnt++;
    }
    box_reduce(b, out + size_t(blockIdx.y) * gridDim.x);
}

// out[block] = the union of the block's n partial boxes.
__global__ void k_box_final(const Box* part, uint32_t n, Box* out) {
    Box b = box_empty();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const Box& c = part[size_t(blockIdx.x) * n + i];
        for (int k = 0; k < 3; k++) b.lo[k] = fmin(b.lo[k], c.lo[k]), b.hi[k] = fmax(b.hi[k], c.hi[k]);
        b.mx = fmax(b.mx, c.mx);
        b.cnt += c.cnt;
    }
    box_reduce(b, out);
}

// Morton keys of the active spheres' cells, ties by input index (the sort
// is stable); inactive spheres sort last.
__global__ void k_morton(const double* xyzr, size_t n, double lx, double ly, double lz, double cell,
                         unsigned long long inactive, unsigned long long* keys, uint32_t* vals) {
    const size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const double* s = xyzr + 4 * i;
    vals[i] = uint32_t(i);
    if (!(s[3] > 0.0)) {
        keys[i] = inactive;
        return;
    }
    const double px = (s[0] - lx) / cell, py = (s[1] - ly) / cell, pz = (s[2] - lz) / cell;
    const uint32_t qx = uint32_t(min(to_u64d(px), 0x1fffffull)), qy = uint32_t(min(to_u64d(py), 0x1fffffull)),
                   qz = uint32_t(min(to_u64d(pz), 0x1fffffull));
    keys[i] = interleave(qx) | (interleave(qy) << 1) | (interleave(qz) << 2);
}

__global__ void k_take_spheres(const double* xyzr, const uint32_t* order, size_t n, double probe, double4* sph,
                               double* rvdw, uint32_t* orig) {
    const size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (k >= n) return;
    const uint32_t i = order[k];
    const double* s = xyzr + 4 * size_t(i);
    sph[k] = make_double4(s[0], s[1], s[2], s[3] + probe);
    rvdw[k] = s[3];
    orig[k] = i;
}

// Grid::coord (geom/cells.rs:91-104).
__device__ __forceinline__ uint32_t grid_coord(double p, double o, double cell, uint32_t dim) {
    const double c = floor((p - o) / cell);
    if (!(c > 0.0)) return 0;
    const unsigned long long v = to_u64d(c);
    return v >= dim - 1 ? dim - 1 : uint32_t(v);
}

__global__ void k_cell_keys(const double* p, size_t stride, size_t n, double ox, double oy, double oz, double cell,
                            uint32_t dx, uint32_t dy, uint32_t dz, uint32_t* keys, uint32_t* vals) {
    const size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const double* q = p + stride * i;
    keys[i] = (grid_coord(q[2], oz, cell, dz) * dy + grid_coord(q[1], oy, cell, dy)) * dx + grid_coord(q[0], ox, cell, dx);
    vals[i] = uint32_t(i);
}

// starts[c] = first position of cell c among the sorted keys (cells + 1).
__global__ void k_cell_starts(const uint32_t* sorted, size_t n, size_t cells, uint32_t* starts) {
    const size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (c > cells) return;
    size_t lo = 0, hi = n;
    while (lo < hi) {
        const size_t mid = (lo + hi) >> 1;
        if (sorted[mid] < c) lo = mid + 1;
        else hi = mid;
    }
    starts[c] = uint32_t(lo);
}

// Containment (arrangement.rs:497-514), a warp per sphere.
__global__ void __launch_bounds__(256) k_contained(const double4* sph, const uint32_t* orig, size_t n, DGrid g,
                                                   double max_expanded, uint32_t* contained) {
    const size_t i = (blockIdx.x * size_t(blockDim.x) + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= n) return;
    const double4 si = sph[i];
    const D3 ci = xyz(si);
    const double Ri = si.w;
    bool found = false;
    warp_for_near(g, si.x, si.y, si.z, Ri + max_expanded, lane, [&](uint32_t j) {
        if (found || j == i) return;
        const double4 sj = sph[j];
        const double d = distp(ci, xyz(sj));
        if (d + Ri <= sj.w + S_EPS && (sj.w - Ri > S_EPS || d > S_EPS || orig[j] < orig[i])) found = true;
    });
    found = __any_sync(0xffffffffu, found);
    if (lane == 0) contained[i] = found ? 1u : 0u;
}

// Neighbour rows (arrangement.rs:522-545), a warp per sphere: count (the
// row's length and how many of it lie above i), then fill.  The fill lists
// the row in scan order in tmp and places each entry by its rank, so rows
// ascend; the entries above i also go to the upper pairs (urow, uj) at uoff.
// One thread per sphere left the chip idle below about 100,000 spheres
// (2,803 spheres: 117 + 185 us for the two passes, 11 blocks).
template <bool FILL>
__global__ void __launch_bounds__(256) k_rows(const double4* sph, const uint32_t* contained, size_t n, DGrid g,
                                              double max_expanded, uint32_t* count, uint32_t* upper,
                                              const uint32_t* off, const uint32_t* uoff, uint32_t* tmp,
                                              uint32_t* items, uint32_t* urow, uint32_t* uj) {
    const size_t i = (blockIdx.x * size_t(blockDim.x) + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= n) return;
    if (contained[i]) {
        if (!FILL && lane == 0) count[i] = 0, upper[i] = 0;
        return;
    }
    const double4 si = sph[i];
    const D3 ci = xyz(si);
    uint32_t c = 0, up = 0;
    uint32_t* t = FILL ? tmp + off[i] : nullptr;
    warp_box_items(g, cell_box(g, si.x, si.y, si.z, si.w + max_expanded), lane, [&](bool valid, uint32_t j) {
        bool keep = false;
        if (valid && j != i && !contained[j]) {
            const double4 sj = sph[j];
            const D3 dc = ci - xyz(sj);
            keep = sqrt_lt(dotp(dc, dc), si.w + sj.w - S_EPS);  // |ci - cj| < Ri + Rj - eps
        }
        const uint32_t m = __ballot_sync(0xffffffffu, keep);
        if (FILL && keep) t[c + __popc(m & ((1u << lane) - 1u))] = j;
        c += __popc(m);
        up += __popc(__ballot_sync(0xffffffffu, keep && j > i));
    });
    if constexpr (!FILL) {
        if (lane == 0) count[i] = c, upper[i] = up;
    } else {
        __syncwarp();
        uint32_t* row = items + off[i];
        const uint32_t lower = c - up;
        for (uint32_t a = lane; a < c; a += 32) {
            const uint32_t v = t[a];
            uint32_t r = 0;
            for (uint32_t q = 0; q < c; q++) r += t[q] < v;
            row[r] = v;
            if (v > i) {
                const uint32_t u = uoff[i] + (r - lower);
                urow[u] = uint32_t(i), uj[u] = v;
            }
        }
    }
}

// The circle of an (i, j) pair (arrangement.rs:674-700) and its cut by a
// third sphere (:251-274).
struct Circle {
    D3 m, u, e1, e2;
    double rho;
};

__device__ __forceinline__ int cut(const Circle& c, D3 s, double R, double en[2], double lv[2]) {
    const D3 g = c.m - s;
    const double a = 2.0 * c.rho * dotp(c.e1, g);
    const double b = 2.0 * c.rho * dotp(c.e2, g);
    const double rhs = R * R - dotp(g, g) - c.rho * c.rho;
    const double amp = sqrt(a * a + b * b);
    if (amp <= rhs) return 1;
    if (amp <= -rhs || amp == 0.0) return 0;
    const double cp = a / amp, sp = b / amp, ca = rhs / amp;
    const double sa = sqrt(fmax(1.0 - ca * ca, 0.0));
    en[0] = cp * ca - sp * sa, en[1] = sp * ca + cp * sa;
    lv[0] = cp * ca + sp * sa, lv[1] = sp * ca - cp * sa;
    return 2;
}

// fl(sqrt(d2)) <= T, T >= 0, decided from the squares where they are clear
// (sqrt_ge's margin).
__device__ __forceinline__ bool sqrt_le(double d2, double T) {
    const double t2 = T * T;
    if (t2 > 1e-280) {
        if (d2 <= t2 * (1.0 - 0x1p-49)) return true;
        if (d2 >= t2 * (1.0 + 0x1p-49)) return false;
    }
    return sqrt(d2) <= T;
}

// cut's return value alone, without its root and divisions.
__device__ __forceinline__ int cut_kind(const Circle& c, D3 s, double R) {
    const D3 g = c.m - s;
    const double a = 2.0 * c.rho * dotp(c.e1, g);
    const double b = 2.0 * c.rho * dotp(c.e2, g);
    const double rhs = R * R - dotp(g, g) - c.rho * c.rho;
    const double amp2 = a * a + b * b;
    if (rhs >= 0.0 && sqrt_le(amp2, rhs)) return 1;
    if (amp2 == 0.0 || (rhs <= 0.0 && sqrt_le(amp2, -rhs))) return 0;
    return 2;
}

__device__ __forceinline__ double diamond(double x, double y) {  // arrangement.rs:282-297
    if (y >= 0.0) return x >= 0.0 ? y / (x + y) : 1.0 - x / (y - x);
    return x < 0.0 ? 2.0 - y / (-x - y) : 3.0 + x / (x - y);
}

__device__ __forceinline__ long long order_bits(double v) {  // f64::total_cmp as an integer key
    const long long b = __double_as_longlong(v);
    return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}

__device__ __forceinline__ double wrap_tau(double a) {  // f64::rem_euclid(TAU)
    const double r = fmod(a, S_TWO_PI);
    return r < 0.0 ? r + S_TWO_PI : r;
}

// A circle's blocked spans, in a warp's shared memory: start and end
// parameters and the blocking sphere (its cut points are recomputed where
// needed); ord: the spans by (start, -end, sphere); re, first, last: runs.
struct Spans {
    double start[MAX_SPANS], end[MAX_SPANS], re[MAX_SPANS];
    uint32_t sphere[MAX_SPANS];
    uint8_t ord[MAX_SPANS], first[MAX_SPANS], last[MAX_SPANS];
};

// any_exposed (arrangement.rs:340-405): 1 exposed, 0 buried, -1 declined.
// The warp ranks the n spans (their keys differ, spheres being distinct) and
// forms the runs: a span opens one where its start is beyond the largest end
// before it, which is the open run's end (runs are disjoint and ascend).
// Runs keep the span that opened them (its start and entry point) and the
// first span that reached their end (its exit point); one lane closes the
// circle and looks at the gaps.
__device__ int any_exposed(Spans& S, int n, const Circle& C, const double4* sph, int lane) {
    if (n == 0) return 1;
    for (int a = lane; a < n; a += 32) {
        const long long sa = order_bits(S.start[a]), ea = order_bits(S.end[a]);
        int r = 0;
        for (int b = 0; b < n; b++) {
            const long long sb = order_bits(S.start[b]), eb = order_bits(S.end[b]);
            r += sb != sa ? sb < sa : (eb != ea ? eb > ea : S.sphere[b] < S.sphere[a]);
        }
        S.ord[r] = uint8_t(a);
    }
    __syncwarp();
    int m = 0, last = 0;  // runs so far; the span that gave the largest end so far
    double re = -1.0;     // and that end (starts are at least 0)
    for (int b = 0; b < n; b += 32) {
        const int a = b + lane;
        const int s = a < n ? S.ord[a] : 0;
        const double ss = a < n ? S.start[s] : 0.0;
        double mx = a < n ? S.end[s] : -1.0;  // inclusive prefix maximum, the first of equal ones
        int arg = s;
        if (lane == 0 && re >= mx) mx = re, arg = last;
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, mx, o);
            const int ya = __shfl_up_sync(0xffffffffu, arg, o);
            if (lane >= o && y >= mx) mx = y, arg = ya;
        }
        double before = __shfl_up_sync(0xffffffffu, mx, 1);
        if (lane == 0) before = re;
        const bool head = a < n && !(ss <= before);
        const uint32_t heads = __ballot_sync(0xffffffffu, head);
        const int r = m + __popc(heads & ((2u << lane) - 1u)) - 1;  // the span's run
        if (head) S.first[r] = uint8_t(s);
        // The run's last span so far holds its end.
        if (a < n && (lane == 31 || a + 1 == n || ((heads >> (lane + 1)) & 1u))) S.re[r] = mx, S.last[r] = uint8_t(arg);
        m += __popc(heads);
        re = __shfl_sync(0xffffffffu, mx, 31), last = __shfl_sync(0xffffffffu, arg, 31);
    }
    __syncwarp();
    int ex = 0;
    if (lane == 0) {
        int b0 = 0;  // runs[b0 .. m)
        while (m - b0 > 1) {
            const double fs = S.start[S.first[b0]], fe = S.re[b0];
            const int l = m - 1;
            if (S.re[l] - S_PERIOD < fs) break;
            if (fe + S_PERIOD > S.re[l]) S.re[l] = fe + S_PERIOD, S.last[l] = S.last[b0];
            b0++;
        }
        const int cnt = m - b0;
        for (int k = 0; k < cnt && ex == 0; k++) {
            const int cur = b0 + k, nxt = b0 + (k + 1) % cnt;
            const double ns = S.start[S.first[nxt]];
            const double next_start = k + 1 < cnt ? ns : ns + S_PERIOD;
            const double gap = next_start - S.re[cur];
            if (gap > S_CLEAR_GAP && gap < S_PERIOD - S_CLEAR_GAP) {
                ex = 1;
            } else if (gap > S_PSEUDO_EPS) {
                double en[2], lv[2], en2[2], lv2[2];
                const double4 sc = sph[S.sphere[S.last[cur]]], sn = sph[S.sphere[S.first[nxt]]];
                cut(C, xyz(sc), sc.w, en, lv);
                cut(C, xyz(sn), sn.w, en2, lv2);
                const double a0 = wrap_tau(atan2(lv[1], lv[0]));
                const double a1 = atan2(en2[1], en2[0]);
                const double w = wrap_tau(a1 - a0);
                if (w < S_ANG_EPS + S_ANG_MARGIN || w > S_TWO_PI - S_ANG_MARGIN) ex = -1;
                else if (w > S_ANG_EPS) ex = 1;
            }
        }
    }
    return __shfl_sync(0xffffffffu, ex, 0);
}

// A pair's counts in one word: circle exposed (0 or 1), blockers (at most
// MAX_SPANS), triple points (at most two per blocker).
__device__ __forceinline__ uint32_t pair_word(uint32_t blk, uint32_t vtx) { return 1u | blk << 1 | vtx << 9; }
// The same three sums over a tile, apart: 4,096 words sum to less than 2^24.
__device__ __forceinline__ unsigned long long pair_sums(uint32_t w) {
    return (unsigned long long)(w & 1u) << 48 | (unsigned long long)((w >> 1) & 0xFFu) << 24 | (w >> 9);
}

// Scan of the pairs' words: per tile, then over the tiles (three sums each,
// totals in total[0..3)), then per pair with an exposed circle its index in
// the circle list and the offsets of its blockers (cb_off, with the total as
// its tail) and vertices.
__global__ void __launch_bounds__(SCAN_THREADS) k_pair_tiles(const uint32_t* w, uint32_t n,
                                                             unsigned long long* tiles) {
    __shared__ unsigned long long sh[SCAN_THREADS / 32];
    const uint64_t base = uint64_t(blockIdx.x) * SCAN_TILE;
    unsigned long long s = 0, t;
    for (int k = 0; k < SCAN_ITEMS; k++) {
        const uint64_t i = base + uint64_t(k) * SCAN_THREADS + threadIdx.x;
        if (i < n) s += pair_sums(w[i]);
    }
    block_exclusive_scan<SCAN_THREADS>(s, sh, &t);
    if (threadIdx.x == 0) tiles[blockIdx.x] = t;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_pair_sums(const unsigned long long* tiles, uint32_t n_tiles,
                                                            unsigned long long* base, unsigned long long* total) {
    __shared__ unsigned long long sh[SCAN_THREADS / 32];
    unsigned long long carry[3] = {0, 0, 0};
    for (uint32_t b0 = 0; b0 < n_tiles; b0 += SCAN_THREADS) {
        const uint32_t i = b0 + threadIdx.x;
        const unsigned long long v = i < n_tiles ? tiles[i] : 0;
        const unsigned long long part[3] = {v >> 48, (v >> 24) & 0xFFFFFFu, v & 0xFFFFFFu};
        for (int k = 0; k < 3; k++) {
            unsigned long long t;
            const unsigned long long e = block_exclusive_scan<SCAN_THREADS>(part[k], sh, &t);
            if (i < n_tiles) base[3 * size_t(i) + k] = carry[k] + e;
            carry[k] += t;
        }
    }
    if (threadIdx.x < 3) total[threadIdx.x] = carry[threadIdx.x];
}

__global__ void __launch_bounds__(SCAN_THREADS) k_pair_apply(const uint32_t* w, uint32_t n,
                                                             const unsigned long long* base, uint32_t* xlist,
                                                             uint32_t* cb_off, uint32_t* v_off, uint32_t nc,
                                                             uint32_t ncb) {
    __shared__ unsigned long long sh[SCAN_THREADS / 32];
    if (blockIdx.x == 0 && threadIdx.x == 0) cb_off[nc] = ncb;
    const uint64_t at = uint64_t(blockIdx.x) * SCAN_TILE + uint64_t(threadIdx.x) * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    unsigned long long s = 0, t;
    for (int k = 0; k < SCAN_ITEMS; k++) {
        v[k] = at + k < n ? w[at + k] : 0u;
        s += pair_sums(v[k]);
    }
    unsigned long long run = block_exclusive_scan<SCAN_THREADS>(s, sh, &t);
    const unsigned long long* b = base + 3 * size_t(blockIdx.x);
    const uint32_t b0 = uint32_t(b[0]), b1 = uint32_t(b[1]), b2 = uint32_t(b[2]);
    for (int k = 0; k < SCAN_ITEMS; k++) {
        if (v[k]) {
            const uint32_t c = b0 + uint32_t(run >> 48);
            xlist[c] = uint32_t(at + k);
            cb_off[c] = b1 + uint32_t((run >> 24) & 0xFFFFFFu);
            v_off[c] = b2 + uint32_t(run & 0xFFFFFFu);
        }
        run += pair_sums(v[k]);
    }
}

// Circles, blockers and triple points of each upper pair (i, j > i)
// (arrangement.rs:674-752).  A warp takes `batch` pairs: its lanes build one
// circle each, then take each pair together, the row's candidates k first (a
// neighbour of j too: the rows' own test, so no walk of j's row) and, where
// none buries the circle, its spans and triple points.  Count pass: the
// pair's word (0: no exposed circle) and exposed[] of both spheres; fill
// pass, over the exposed circles (xlist): the records at their offsets.
// Bound by f64 instructions: roots and divisions are taken by one lane per
// circle and for the candidates that cut it alone (54,500 pairs: 392 us with
// a thread per pair, 179 with every lane building the circle and cutting, 1,500
// instructions a pair).
template <bool FILL>
__global__ void __launch_bounds__(32 * C_WARPS) k_circles(const double4* sph, const uint32_t* nb_off,
                                                          const uint32_t* nb_items, size_t n_pairs, uint32_t batch,
                                                          const uint32_t* urow, const uint32_t* uj,
                                                          const uint32_t* xlist, uint32_t* word, uint32_t* exposed,
                                                          const uint32_t* cb_off, const uint32_t* v_off, double* circ,
                                                          uint32_t* ij, uint32_t* cb_items, double4* vert,
                                                          uint32_t* vatoms, uint32_t* decline) {
    __shared__ Spans sh[C_WARPS];
    __shared__ Circle sh_c[C_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t id0 = (blockIdx.x * size_t(C_WARPS) + warp) * batch;
    if (id0 >= n_pairs) return;
    const int np = int(min(size_t(batch), n_pairs - id0));
    Spans& S = sh[warp];
    const uint32_t below = (1u << lane) - 1u;
    uint32_t my_u = 0, my_i = 0, my_j = 0;
    bool cuts = false;  // the pair's spheres cut in a circle
    if (lane < np) {
        my_u = FILL ? xlist[id0 + lane] : uint32_t(id0 + lane);
        my_i = urow[my_u], my_j = uj[my_u];
        const double4 si = sph[my_i], sj = sph[my_j];
        const D3 ci = xyz(si), cj = xyz(sj);
        const double Ri = si.w, Rj = sj.w;
        const double d = distp(ci, cj);
        const D3 axis = (cj - ci) / d;
        const double t = (d * d + Ri * Ri - Rj * Rj) / (2.0 * d);
        const double rho2 = Ri * Ri - t * t;
        cuts = !(rho2 <= 0.0);
        const double ax = fabs(axis.x), ay = fabs(axis.y), az = fabs(axis.z);  // orthonormal_basis (geom/vec.rs:112-125)
        const D3 helper = (ax <= ay && ax <= az) ? D3{1, 0, 0} : (ay <= az ? D3{0, 1, 0} : D3{0, 0, 1});
        const D3 hx = crossp(helper, axis);
        const D3 e1 = hx / normp(hx);
        const D3 e2 = crossp(axis, e1);
        sh_c[warp][lane] = Circle{ci + axis * t, axis, e1, e2, sqrt(rho2)};
    }
    const uint32_t todo = __ballot_sync(0xffffffffu, cuts);
    uint32_t my_word = 0;  // count pass: lane's pair
    __syncwarp();
    for (int q = 0; q < np; q++) {
        if (!((todo >> q) & 1u)) continue;
        const uint32_t i = __shfl_sync(0xffffffffu, my_i, q), j = __shfl_sync(0xffffffffu, my_j, q);
        const size_t id = id0 + q;
        const Circle C = sh_c[warp][q];
        const double4 sj = sph[j];
        const D3 cj = xyz(sj);
        const double Rj = sj.w;
        const uint32_t r0 = nb_off[i], r1 = nb_off[i + 1];
        int ns = 0;
        bool buried = false;
        for (uint32_t b = r0; b < r1 && !buried; b += 32) {
            const uint32_t pk = b + lane;
            int kind = 0;
            uint32_t k = 0;
            if (pk < r1) {
                k = nb_items[pk];
                const double4 sk = sph[k];
                const D3 dc = cj - xyz(sk);
                // k in j's row: k_rows' test (k is i's neighbour, so it is not
                // contained; the test is symmetric in j and k).
                if (k != j && sqrt_lt(dotp(dc, dc), Rj + sk.w - S_EPS)) kind = cut_kind(C, xyz(sk), sk.w);
            }
            buried = __any_sync(0xffffffffu, kind == 1);
            const uint32_t m = __ballot_sync(0xffffffffu, kind == 2);
            const int a = ns + __popc(m & below);
            if (kind == 2 && a < MAX_SPANS) S.sphere[a] = k;
            ns += __popc(m);
        }
        if (buried) continue;
        if (ns > MAX_SPANS) {
            if (lane == 0) atomicOr(decline, DECLINE_SPANS);
            continue;
        }
        __syncwarp();
        if (!FILL) {
            for (int a = lane; a < ns; a += 32) {
                const double4 sk = sph[S.sphere[a]];
                double en[2], lv[2];
                cut(C, xyz(sk), sk.w, en, lv);
                const double s0 = diamond(en[0], en[1]);
                double s1 = diamond(lv[0], lv[1]);
                if (s1 <= s0) s1 += S_PERIOD;
                S.start[a] = s0, S.end[a] = s1;
            }
            __syncwarp();
            const int ex = any_exposed(S, ns, C, sph, lane);
            if (ex < 0 && lane == 0) atomicOr(decline, DECLINE_ANGLE);
            if (ex <= 0) {
                __syncwarp();
                continue;
            }
        }
        // Triple points with the blockers k > j: candidate 2 a + w is blocker
        // a's exit (w = 0) or entry point.
        uint32_t nv = 0;
        const uint32_t v0 = FILL ? v_off[id] : 0;
        for (int t0 = 0; t0 < 2 * ns; t0 += 32) {
            const int ti = t0 + lane;
            const uint32_t k = ti < 2 * ns ? S.sphere[ti >> 1] : 0u;
            bool free = false;
            D3 p{0, 0, 0};
            if (ti < 2 * ns && k > j) {
                double en[2], lv[2];
                const double4 sk = sph[k];
                if (cut(C, xyz(sk), sk.w, en, lv) == 2) {
                    const double c0 = (ti & 1) ? en[0] : lv[0], c1 = (ti & 1) ? en[1] : lv[1];
                    p = C.m + (C.e1 * c0 + C.e2 * c1) * C.rho;
                    free = true;
                    for (uint32_t pl = r0; pl < r1 && free; pl++) {
                        const uint32_t l = nb_items[pl];
                        if (l != j && l != k) {
                            // |p - c| >= R - eps, decided from the square where it
                            // is clear (sqrt_ge: the same result as the rounded root).
                            const double4 sl = sph[l];
                            const D3 dp = p - xyz(sl);
                            free = sqrt_ge(dotp(dp, dp), sl.w - S_EPS);
                        }
                    }
                }
            }
            const uint32_t m = __ballot_sync(0xffffffffu, free);
            if (FILL && free) {
                const uint32_t v = v0 + nv + __popc(m & below);
                vert[v] = make_double4(p.x, p.y, p.z, 0.0);
                uint32_t* va = vatoms + 3 * size_t(v);
                va[0] = i, va[1] = j, va[2] = k;
            }
            nv += __popc(m);
        }
        if (!FILL) {
            if (lane == q) my_word = pair_word(uint32_t(ns), nv);
            if (lane == 0) exposed[i] = 1, exposed[j] = 1;
        } else {
            for (int a = lane; a < ns; a += 32) cb_items[cb_off[id] + a] = S.sphere[a];
        }
        __syncwarp();
    }
    if (lane >= np) return;
    if (!FILL) {
        word[my_u] = my_word;
    } else {
        const Circle C = sh_c[warp][lane];
        double* rec = circ + 12 * (id0 + lane);
        rec[0] = C.m.x, rec[1] = C.m.y, rec[2] = C.m.z, rec[3] = C.u.x, rec[4] = C.u.y, rec[5] = C.u.z;
        rec[6] = C.e1.x, rec[7] = C.e1.y, rec[8] = C.e1.z, rec[9] = C.rho, rec[10] = 0.0, rec[11] = 0.0;
        ij[2 * (id0 + lane)] = my_i, ij[2 * (id0 + lane) + 1] = my_j;
    }
}

// Pairs a warp of the circle passes takes: enough warps to fill the chip
// four times over (64 an SM) first, then up to one circle per lane.
uint32_t circle_batch(size_t n_pairs, int sms) {
    return uint32_t(std::min<size_t>(32, std::max<size_t>(1, n_pairs / (size_t(sms) * 64))));
}

// Status (contained 2, exposed 0, buried 1), the row lengths kept (exposed
// spheres only; point.rs:244-245) and the number of contained spheres.  A
// sphere field (nb_off null) has no rows and every sphere not contained
// exposed.
__global__ void __launch_bounds__(256) k_status(const uint32_t* contained, const uint32_t* exposed,
                                                const uint32_t* nb_off, size_t n, uint32_t* status,
                                                uint32_t* keep_len, unsigned long long* n_contained) {
    const size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    const bool in = i < n, cont = in && contained[i];
    if (in) {
        const uint32_t len = nb_off ? nb_off[i + 1] - nb_off[i] : 0;
        const bool ex = !cont && (len == 0 || exposed[i]);
        status[i] = cont ? STATUS_CONTAINED : (ex ? STATUS_EXPOSED : STATUS_BURIED);
        if (keep_len) keep_len[i] = ex ? len : 0;
    }
    const int c = __syncthreads_count(cont);
    if (threadIdx.x == 0 && c) atomicAdd(n_contained, (unsigned long long)c);
}

__global__ void __launch_bounds__(256) k_keep_rows(const uint32_t* nb_off, const uint32_t* nb_items,
                                                   const uint32_t* keep_len, const uint32_t* new_off, size_t n,
                                                   uint32_t* out) {
    const size_t i = (blockIdx.x * size_t(blockDim.x) + threadIdx.x) >> 5;
    if (i >= n) return;
    for (uint32_t a = threadIdx.x & 31, c = keep_len[i]; a < c; a += 32) out[new_off[i] + a] = nb_items[nb_off[i] + a];
}

// Host side.
struct Ctx {
    cudaStream_t s;
    DevArrangement& out;
    std::vector<void*> temp;
    std::string* msg;
    bool ok = true;
    void* alloc(size_t bytes, bool keep) {
        void* p = nullptr;
        if (mem_alloc(&p, std::max<size_t>(bytes, 16)) != cudaSuccess) {
            ok = false;
            if (msg) *msg = "device memory for the arrangement";
            return nullptr;
        }
        if (keep) out.owned.push_back(p), out.bytes += bytes;
        else temp.push_back(p);
        return p;
    }
    ~Ctx() {
        cudaStreamSynchronize(s);  // the temporaries were used on this stream alone
        for (void* p : temp) mem_free_synced(p);
        pinned_free(host);
    }
    // n bytes at the device address src, once everything queued so far has
    // run (page-locked; valid until the next call).
    void* host = nullptr;
    const void* read(const void* src, size_t bytes) {
        if (!host) host = pinned_alloc(READ_BYTES);
        if (!host || cudaMemcpyAsync(host, src, bytes, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            return nullptr;
        return host;
    }
    static constexpr size_t READ_BYTES = 512;
};

unsigned blocks_for(size_t n, unsigned t = 256) { return unsigned(std::max<size_t>(1, (n + t - 1) / t)); }

// What the device reports back: bits of one read.
struct Report {
    Box box[2];                  // active spheres; then circle centres and vertices
    unsigned long long tot[4];   // scan totals
    unsigned long long contained;
    uint32_t decline, pad;
};
static_assert(sizeof(Report) <= Ctx::READ_BYTES, "Report fits the read buffer");

// Grid::build (geom/cells.rs:27-84) over n points at p + stride * i whose
// bounding box is known.
bool build_grid(Ctx& X, const double* p, size_t stride, size_t n, double cell_in, const Box& b, DGrid& G) {
    G = DGrid{};
    G.cell = cell_in;
    if (n == 0) {
        G.dx = G.dy = G.dz = 1;
        uint32_t* st = static_cast<uint32_t*>(X.alloc(8, true));
        if (!st || cudaMemsetAsync(st, 0, 8, X.s) != cudaSuccess) return false;
        G.starts = st;
        G.items = static_cast<uint32_t*>(X.alloc(4, true));
        return G.items != nullptr;
    }
    const double e[3] = {b.hi[0] - b.lo[0], b.hi[1] - b.lo[1], b.hi[2] - b.lo[2]};
    const size_t max_cells = std::max<size_t>(8 * n, size_t(1) << 16);
    double cell = cell_in;
    uint32_t dims[3];
    for (;;) {
        unsigned __int128 total = 1;
        bool ok = true;
        for (int a = 0; a < 3; a++) {
            const uint64_t v = to_u64d(std::floor(e[a] / cell));
            if (v >= UINT32_MAX) ok = false;
            dims[a] = ok ? uint32_t(v + 1) : 1;
            total *= (unsigned __int128)(v + 1);
        }
        if (ok && total <= max_cells) break;
        cell *= 2.0;
    }
    G.ox = b.lo[0], G.oy = b.lo[1], G.oz = b.lo[2], G.cell = cell;
    G.dx = dims[0], G.dy = dims[1], G.dz = dims[2];
    const size_t cells = size_t(dims[0]) * dims[1] * dims[2];
    if (cells >= (size_t(1) << 32) - 1 || n >= (size_t(1) << 31)) return false;
    uint32_t* keys = static_cast<uint32_t*>(X.alloc(n * 4, false));
    uint32_t* keys2 = static_cast<uint32_t*>(X.alloc(n * 4, false));
    uint32_t* vals = static_cast<uint32_t*>(X.alloc(n * 4, false));
    uint32_t* items = static_cast<uint32_t*>(X.alloc(n * 4, true));
    uint32_t* starts = static_cast<uint32_t*>(X.alloc((cells + 1) * 4, true));
    if (!X.ok) return false;
    k_cell_keys<<<blocks_for(n), 256, 0, X.s>>>(p, stride, n, G.ox, G.oy, G.oz, cell, dims[0], dims[1], dims[2], keys,
                                                vals);
    unsigned bits = 1;
    while (bits < 32 && (uint64_t(1) << bits) < cells) bits++;
    size_t tmp = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp, keys, keys2, vals, items, int(n), 0, int(bits), X.s);
    void* t = X.alloc(tmp, false);
    if (!t) return false;
    if (cub::DeviceRadixSort::SortPairs(t, tmp, keys, keys2, vals, items, int(n), 0, int(bits), X.s) != cudaSuccess)
        return false;
    k_cell_starts<<<blocks_for(cells + 1), 256, 0, X.s>>>(keys2, n, cells, starts);
    G.starts = starts;
    G.items = items;
    count_launches(3);
    return cudaGetLastError() == cudaSuccess;
}

}  // namespace

void DevArrangement::release() {
    for (void* p : owned) mem_free(p);
    owned.clear();
    bytes = 0;
}

int build_arrangement_device(smb_device* d, const double* xyzr, size_t ns, double probe, int kind,
                             DevArrangement& out, std::string* msg) {
    out = DevArrangement();
    if (cudaSetDevice(d->index) != cudaSuccess) return 2;
    Ctx X{d->stream, out, {}, msg};
    cudaStream_t s = d->stream;
    auto fail = [&](const char* what) {
        if (msg && msg->empty()) *msg = what;
        out.release();
        return 2;
    };
    const bool spheres = kind != SMB_KIND_SES;
    if (ns >= (size_t(1) << 31)) return fail("too many spheres for the device arrangement");
    double* dx = static_cast<double*>(X.alloc(ns * 32, false));
    Box* part = static_cast<Box*>(X.alloc(sizeof(Box) * 2 * RED_BLOCKS, false));
    Report* rep = static_cast<Report*>(X.alloc(sizeof(Report), false));
    if (!X.ok) return fail("device memory");
    if (ns && cudaMemcpyAsync(dx, xyzr, ns * 32, cudaMemcpyHostToDevice, s) != cudaSuccess) return fail("upload");
    if (cudaMemsetAsync(rep, 0, sizeof(Report), s) != cudaSuccess) return fail("report");
    auto red_blocks = [](size_t n) { return std::min<unsigned>(RED_BLOCKS, blocks_for(n)); };
    // Active spheres, max_expanded, Morton order.
    {
        const unsigned nb = red_blocks(ns);
        k_box_active<<<nb, 256, 0, s>>>(dx, ns, probe, part);
        k_box_final<<<1, 256, 0, s>>>(part, nb, rep->box);
        count_launches(2);
    }
    const Report* R = static_cast<const Report*>(X.read(rep, sizeof(Report)));
    if (!R) return fail("reduction");
    const Box ba = R->box[0];
    const size_t n = size_t(ba.cnt);
    const double max_expanded = ba.mx;
    const double cell = std::fmax(2.0 * max_expanded, 1e-6);
    DArr& A = out.A;
    A.n = uint32_t(n);
    A.max_expanded = max_expanded;
    A.probe = probe;
    out.n = n;
    double4* sph = static_cast<double4*>(X.alloc(n * 32, true));
    double* rvdw = static_cast<double*>(X.alloc(n * 8, true));
    uint32_t* orig = static_cast<uint32_t*>(X.alloc(n * 4, true));
    uint32_t* status = static_cast<uint32_t*>(X.alloc(n * 4, true));
    if (!X.ok) return fail("device memory");
    if (n) {
        // Key bits: the cells of the box on each axis, interleaved (the rest
        // are zero); inactive spheres take the next power of two.
        unsigned axis_bits = 1;
        for (int k = 0; k < 3; k++) {
            const uint64_t q = std::min<uint64_t>(to_u64d((ba.hi[k] - ba.lo[k]) / cell), 0x1fffff);
            while (axis_bits < 21 && (q >> axis_bits)) axis_bits++;
        }
        const unsigned bits = 3 * axis_bits;
        unsigned long long* keys = static_cast<unsigned long long*>(X.alloc(ns * 8, false));
        unsigned long long* keys2 = static_cast<unsigned long long*>(X.alloc(ns * 8, false));
        uint32_t* vals = static_cast<uint32_t*>(X.alloc(ns * 4, false));
        uint32_t* order = static_cast<uint32_t*>(X.alloc(ns * 4, false));
        if (!X.ok) return fail("device memory");
        k_morton<<<blocks_for(ns), 256, 0, s>>>(dx, ns, ba.lo[0], ba.lo[1], ba.lo[2], cell, 1ull << bits, keys, vals);
        const int end = int(bits) + (ns > n ? 1 : 0);
        size_t tmp = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tmp, keys, keys2, vals, order, int(ns), 0, end, s);
        void* t = X.alloc(tmp, false);
        if (!t || cub::DeviceRadixSort::SortPairs(t, tmp, keys, keys2, vals, order, int(ns), 0, end, s) != cudaSuccess)
            return fail("sort");
        k_take_spheres<<<blocks_for(n), 256, 0, s>>>(dx, order, n, probe, sph, rvdw, orig);
        count_launches(2);
    }
    A.sph = sph, A.rvdw = rvdw, A.status = status;
    out.orig = orig;
    for (int k = 0; k < 3; k++) out.lo[k] = n ? ba.lo[k] : 0.0, out.hi[k] = n ? ba.hi[k] : 0.0;
    if (n) {
        const double ex = out.hi[0] - out.lo[0], ey = out.hi[1] - out.lo[1], ez = out.hi[2] - out.lo[2];
        out.extent = std::sqrt(ex * ex + ey * ey + ez * ez) + 4.0 * max_expanded + 4.0 * probe + 1.0;
    }
    if (!build_grid(X, reinterpret_cast<const double*>(sph), 4, n, cell, ba, A.gs)) return fail("sphere grid");
    // Containment.
    uint32_t* contained = static_cast<uint32_t*>(X.alloc(n * 4, false));
    if (!X.ok) return fail("device memory");
    if (n) {
        count_launches(1);
        k_contained<<<blocks_for(n, 8), 256, 0, s>>>(sph, orig, n, A.gs, max_expanded, contained);
    }
    size_t nc = 0, ncb = 0, nv = 0, n_kept = 0;
    double *circ = nullptr;
    double4* vert = nullptr;
    uint32_t *ij = nullptr, *cb_off = nullptr, *cb_items = nullptr, *vatoms = nullptr, *nb_items = nullptr;
    uint32_t* nb_off = static_cast<uint32_t*>(X.alloc((n + 1) * 4, true));
    if (!X.ok) return fail("device memory");
    Box bc{}, bv{};
    if (spheres || !n) {
        // No rows, circles or vertices.
        cb_off = static_cast<uint32_t*>(X.alloc(4, true));
        nb_items = static_cast<uint32_t*>(X.alloc(4, true)), cb_items = static_cast<uint32_t*>(X.alloc(4, true));
        circ = static_cast<double*>(X.alloc(96, true)), vert = static_cast<double4*>(X.alloc(32, true));
        ij = static_cast<uint32_t*>(X.alloc(8, true)), vatoms = static_cast<uint32_t*>(X.alloc(12, true));
        if (!X.ok) return fail("device memory");
        if (cudaMemsetAsync(cb_off, 0, 4, s) != cudaSuccess || cudaMemsetAsync(nb_off, 0, (n + 1) * 4, s) != cudaSuccess)
            return fail("rows");
        if (n) {
            count_launches(1);
            k_status<<<blocks_for(n), 256, 0, s>>>(contained, nullptr, nullptr, n, status, nullptr, &rep->contained);
        }
        R = static_cast<const Report*>(X.read(rep, sizeof(Report)));
        if (!R) return fail("status");
    } else {
        uint32_t* rlen = static_cast<uint32_t*>(X.alloc(n * 4, false));
        uint32_t* ulen = static_cast<uint32_t*>(X.alloc(n * 4, false));
        uint32_t* roff = static_cast<uint32_t*>(X.alloc((n + 1) * 4, false));
        uint32_t* uoff = static_cast<uint32_t*>(X.alloc((n + 1) * 4, false));
        uint32_t* exposed = static_cast<uint32_t*>(X.alloc(n * 4, false));
        unsigned long long* tiles =
            static_cast<unsigned long long*>(X.alloc(size_t(scan_tiles_needed(uint32_t(n + 1))) * 8 + 64, false));
        if (!X.ok) return fail("device memory");
        if (cudaMemsetAsync(exposed, 0, n * 4, s) != cudaSuccess) return fail("rows");
        k_rows<false><<<blocks_for(n, 8), 256, 0, s>>>(sph, contained, n, A.gs, max_expanded, rlen, ulen, nullptr,
                                                       nullptr, nullptr, nullptr, nullptr, nullptr);
        launch_scan(rlen, uint32_t(n), roff, nullptr, tiles, &rep->tot[0], s, true);
        launch_scan(ulen, uint32_t(n), uoff, nullptr, tiles, &rep->tot[1], s, true);
        count_launches(1);
        if (!(R = static_cast<const Report*>(X.read(rep, sizeof(Report))))) return fail("rows");
        const size_t n_entries = size_t(R->tot[0]), n_upper = size_t(R->tot[1]);
        if (n_entries >= (size_t(1) << 32)) return fail("too many neighbour pairs for the device arrangement");
        uint32_t* items = static_cast<uint32_t*>(X.alloc(n_entries * 4, false));
        uint32_t* unsorted = static_cast<uint32_t*>(X.alloc(n_entries * 4, false));
        uint32_t* urow = static_cast<uint32_t*>(X.alloc(n_upper * 4, false));
        uint32_t* uj = static_cast<uint32_t*>(X.alloc(n_upper * 4, false));
        uint32_t* word = static_cast<uint32_t*>(X.alloc(n_upper * 4, false));
        const uint32_t p_tiles = uint32_t((n_upper + SCAN_TILE - 1) / SCAN_TILE);
        unsigned long long* pt = static_cast<unsigned long long*>(X.alloc(size_t(p_tiles) * 32, false));
        if (!X.ok) return fail("device memory");
        k_rows<true><<<blocks_for(n, 8), 256, 0, s>>>(sph, contained, n, A.gs, max_expanded, nullptr, nullptr, roff,
                                                      uoff, unsorted, items, urow, uj);
        count_launches(1);
        if (n_upper) {
            const uint32_t batch = circle_batch(n_upper, d->info.multiprocessors);
            k_circles<false><<<blocks_for(n_upper, C_WARPS * batch), 32 * C_WARPS, 0, s>>>(
                sph, roff, items, n_upper, batch, urow, uj, nullptr, word, exposed, nullptr, nullptr, nullptr, nullptr,
                nullptr, nullptr, nullptr, &rep->decline);
            k_pair_tiles<<<p_tiles, SCAN_THREADS, 0, s>>>(word, uint32_t(n_upper), pt);
            k_pair_sums<<<1, SCAN_THREADS, 0, s>>>(pt, p_tiles, pt + p_tiles, rep->tot);
            count_launches(3);
            if (!(R = static_cast<const Report*>(X.read(rep, sizeof(Report))))) return fail("circles");
            if (R->decline) {
                if (msg)
                    *msg = (R->decline & DECLINE_ANGLE)
                               ? "a circle's exposure is within the device's atan2 error of its threshold"
                               : "a circle has more candidate blockers than the device keeps";
                out.release();
                return 1;
            }
            nc = size_t(R->tot[0]), ncb = size_t(R->tot[1]), nv = size_t(R->tot[2]);
        }
        if (ncb >= (size_t(1) << 32) || nv >= (size_t(1) << 32)) return fail("arrangement too large for the device");
        circ = static_cast<double*>(X.alloc(nc * 96, true));
        ij = static_cast<uint32_t*>(X.alloc(nc * 8, true));
        cb_off = static_cast<uint32_t*>(X.alloc((nc + 1) * 4, true));
        cb_items = static_cast<uint32_t*>(X.alloc(ncb * 4, true));
        vert = static_cast<double4*>(X.alloc(nv * 32, true));
        vatoms = static_cast<uint32_t*>(X.alloc(nv * 12, true));
        uint32_t* keep_len = static_cast<uint32_t*>(X.alloc(n * 4, false));
        uint32_t* xlist = static_cast<uint32_t*>(X.alloc(nc * 4, false));
        uint32_t* v_off = static_cast<uint32_t*>(X.alloc(nc * 4, false));
        if (!X.ok) return fail("device memory");
        if (nc) {
            k_pair_apply<<<p_tiles, SCAN_THREADS, 0, s>>>(word, uint32_t(n_upper), pt + p_tiles, xlist, cb_off, v_off,
                                                          uint32_t(nc), uint32_t(ncb));
            const uint32_t batch = circle_batch(nc, d->info.multiprocessors);
            k_circles<true><<<blocks_for(nc, C_WARPS * batch), 32 * C_WARPS, 0, s>>>(
                sph, roff, items, nc, batch, urow, uj, xlist, word, exposed, cb_off, v_off, circ, ij, cb_items, vert, vatoms,
                &rep->decline);
            count_launches(2);
        } else if (cudaMemsetAsync(cb_off, 0, 4, s) != cudaSuccess) {
            return fail("circles");
        }
        // Statuses, the rows of exposed spheres, the boxes of circle centres
        // (with the largest radius) and vertices.
        k_status<<<blocks_for(n), 256, 0, s>>>(contained, exposed, roff, n, status, keep_len, &rep->contained);
        launch_scan(keep_len, uint32_t(n), nb_off, nullptr, tiles, &rep->tot[3], s, true);
        const unsigned nb = red_blocks(std::max(nc, nv));
        k_box_points<<<dim3(nb, 2), 256, 0, s>>>(PointSet{circ, 12, nc, 9},
                                                 PointSet{reinterpret_cast<const double*>(vert), 4, nv, -1}, part);
        k_box_final<<<2, 256, 0, s>>>(part, nb, rep->box);
        count_launches(3);
        if (!(R = static_cast<const Report*>(X.read(rep, sizeof(Report))))) return fail("status");
        n_kept = size_t(R->tot[3]);
        nb_items = static_cast<uint32_t*>(X.alloc(n_kept * 4, true));
        if (!X.ok) return fail("device memory");
        k_keep_rows<<<blocks_for(n, 8), 256, 0, s>>>(roff, items, keep_len, nb_off, n, nb_items);
        count_launches(1);
        bc = R->box[0], bv = R->box[1];
    }
    out.n_contained = size_t(R->contained);
    A.nb_off = nb_off, A.nb_items = nb_items;
    A.nc = uint32_t(nc), A.nv = uint32_t(nv);
    // Rows sorted in k_rows, blockers listed in row order.
    A.flags = DARR_ROWS_SORTED | (spheres ? DARR_SPHERES : 0u);
    A.circ = circ, A.cb_off = cb_off, A.cb_items = cb_items, A.vert = vert;
    out.circle_ij = ij, out.vertex_atoms = vatoms;
    out.n_circles = nc, out.n_vertices = nv, out.nb_items = n_kept, out.cb_items = ncb;
    out.kind = kind;
    A.rho_max = nc ? bc.mx : 0.0;
    // Grids of circle centres and vertices.
    if (!build_grid(X, circ, 12, nc, cell, bc, A.gc)) return fail("circle grid");
    if (!build_grid(X, reinterpret_cast<const double*>(vert), 4, nv, cell, bv, A.gv)) return fail("vertex grid");
    if (cudaGetLastError() != cudaSuccess) return fail("kernel launch");
    return 0;
}

bool arrangement_to_host(const DevArrangement& D, smbh::Arrangement& H) {
    const DArr& A = D.A;
    const size_t n = D.n, nc = D.n_circles, nv = D.n_vertices;
    H = smbh::Arrangement();
    H.kind = D.kind;
    H.probe = A.probe;
    H.n = n;
    H.n_contained = D.n_contained;
    H.max_expanded = A.max_expanded;
    H.rho_max = A.rho_max;
    H.extent = D.extent;
    std::vector<double> sph(4 * n), circ(12 * nc), vert(4 * nv);
    H.radius.resize(n), H.orig.resize(n), H.status.resize(n), H.nb_off.resize(n + 1), H.nb_items.resize(D.nb_items);
    H.circle_ij.resize(2 * nc), H.cb_off.resize(nc + 1), H.cb_items.resize(D.cb_items), H.vertex_atoms.resize(3 * nv);
    auto get = [](void* dst, const void* src, size_t bytes) {
        return !bytes || cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost) == cudaSuccess;
    };
    bool ok = get(sph.data(), A.sph, n * 32) && get(H.radius.data(), A.rvdw, n * 8) &&
              get(H.orig.data(), D.orig, n * 4) && get(H.status.data(), A.status, n * 4) &&
              get(H.nb_off.data(), A.nb_off, (n + 1) * 4) && get(H.nb_items.data(), A.nb_items, D.nb_items * 4) &&
              get(circ.data(), A.circ, nc * 96) && get(H.circle_ij.data(), D.circle_ij, nc * 8) &&
              get(H.cb_off.data(), A.cb_off, (nc + 1) * 4) && get(H.cb_items.data(), A.cb_items, D.cb_items * 4) &&
              get(vert.data(), A.vert, nv * 32) && get(H.vertex_atoms.data(), D.vertex_atoms, nv * 12);
    if (!ok) return false;
    H.center.resize(3 * n), H.expanded.resize(n);
    for (size_t i = 0; i < n; i++)
        H.center[3 * i] = sph[4 * i], H.center[3 * i + 1] = sph[4 * i + 1], H.center[3 * i + 2] = sph[4 * i + 2],
        H.expanded[i] = sph[4 * i + 3];
    H.circle.resize(10 * nc);
    for (size_t c = 0; c < nc; c++)
        for (int k = 0; k < 10; k++) H.circle[10 * c + k] = circ[12 * c + k];
    H.vertex.resize(3 * nv);
    for (size_t v = 0; v < nv; v++)
        for (int k = 0; k < 3; k++) H.vertex[3 * v + k] = vert[4 * v + k];
    const DGrid* g[3] = {&A.gs, &A.gc, &A.gv};
    smbh::Grid* h[3] = {&H.cells, &H.circle_cells, &H.vertex_cells};
    const size_t cnt[3] = {n, nc, nv};
    for (int k = 0; k < 3; k++) {
        smbh::Grid& G = *h[k];
        G.origin[0] = g[k]->ox, G.origin[1] = g[k]->oy, G.origin[2] = g[k]->oz, G.cell = g[k]->cell;
        G.dims[0] = g[k]->dx, G.dims[1] = g[k]->dy, G.dims[2] = g[k]->dz;
        const size_t cells = size_t(G.dims[0]) * G.dims[1] * G.dims[2];
        G.starts.resize(cells + 1);
        G.items.resize(cnt[k]);
        if (!get(G.starts.data(), g[k]->starts, (cells + 1) * 4) || !get(G.items.data(), g[k]->items, cnt[k] * 4))
            return false;
    }
    return true;
}

}  // namespace smb
