// nf_mutual.cu -- the mutual pencil engine: each pair of particles of a slab
// range is evaluated once and its force added to both.
//
// What bounds the one-sided sweep (nf_box.cu) is the FP32 pipe: 14 paired
// instructions per two interactions (13 with the Newton step of this engine).
// Of these only the three accumulations belong to one particle; separation,
// r^2 and g are the same for the pair seen from the other side.  Evaluating a
// pair once and accumulating it twice costs 16 instructions for four
// interactions: 8 per two.
// Sweep times, one-sided -> mutual (with the list ordered as below): uniform
// 64^3 0.922 -> 0.768 ms, clustered 128^3 8.96 -> 6.87, clustered 256^3 119.1
// -> 88.0 (2.8e12 pairs/s; 89.9 on another GPU), density 100^3 6.46 -> 4.10;
// 3.2e12 pairs/s where pencils hold thousands of sinks.
// On clustered 256^3 the FMA pipe is busy 67 % (one instruction in three
// reads three distinct register pairs and issues at 2/3 rate).  Of a warp's
// time on uniform 160^3, 79 % is the mutual loop, 7 % the centre column
// one-sided, 8 % staging, 6 % the rest; padding of tiles and groups is 11 %.
//
// Which pairs.  A sink pencil (cells (x, y, zc-R .. zc+R)) meets the source
// cells (x+dx, y+dy, zc) as in the one-sided scheme, but only those of half
// the columns: dx > 0, or dx == 0 and dy > 0 (mutual columns).  Columns
// outside the slab range [lo, hi) have no sinks there to receive a reaction:
// they are met one-sided, in both signs of dx.  The pencil's own column
// (dx == dy == 0) is one-sided where cells are sparse; where one of a pair of
// its cells holds DENSE_CELL particles or more, the pair is met mutually (by
// the pencil of the lower cell), and a dense centre cell meets itself in a
// triangle: a tile against the particles after it, mutually, and against
// itself one-sided.
//
// How a warp does it.  Up to 32*S sinks sit in registers (S per lane, in
// pairs: two per FP32 instruction).  64 sources at a time are staged into the
// warp's shared-memory slot.  One-sided: every lane reads each source
// (broadcast).  Mutual: in step t of 32, lane l meets source (l + t) mod 32
// of a group of 32, and the running reaction of that source moves from lane
// l + 1 to lane l by shuffle, so that after 32 steps lane l holds the whole
// reaction of source l on it from the tile's 32*S sinks.  Each source is
// staged twice, 32 slots apart, so that (l + t) needs no wrap.
//
// Where sums go.  Reactions arrive at a particle from many warps in no fixed
// order, so all sums meet in 64-bit fixed point, added with integer atomics:
// associative, so the same work list gives the same bits in whatever order it
// runs.  Another list -- another kernel shape, slab range or GPU size, other
// SICs -- cuts tiles and streams elsewhere: the groups of FP32 partials below
// and the rounding of each piece to the unit differ, and results agree to
// rounding.  The unit is 2^-fbits of the kernel's force unit, with fbits set from
// a strict bound on a sink's sum (largest possible pair force x most sources
// a sink can meet) so that it cannot overflow; see mutual_bits() for the
// condition under which its resolution is below FP32's own noise.  FP32
// partials run over at most 128 terms as in the one-sided engine: a tile's
// sums are folded every 128 sources into a compensated (h, l) pair, a
// source's reaction is a sum over one tile.  A partial that is not finite
// (a NaN or infinite position) marks the particle, whose record is NaN.
//
// Work list.  Built on the device: tiles cut into pieces of bounded cost
// along their chunks (any piece adds its own sums: no combining), ordered by
// sinks per lane and cost, taken by warps from a counter.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "nf_internal.h"
#include "nf_pair.cuh"

namespace nf {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int MAXW = 5;
constexpr int MAXSRC = 25;
constexpr int CHUNK = 64;  // sources staged at a time: two groups of 32
constexpr int GROUP = 32;
constexpr int WPC = ENGINE_WARPS_PER_CTA;
constexpr int FOLD = 2;    // chunks between folds of the FP32 partials
constexpr int DENSE_CELL = 192;
constexpr int NCLASS = 64;  // classes of the work list: sinks per lane x octave of cost

// What a pencil's stream of sources consists of, in stream order: mutual
// columns [0, Ms), the centre cell [Ms, Ms + own), one-sided columns up to M.
struct Stream {
    int Ms, own, M;
    int own_begin;       // first centre-cell sink in the pencil's sink stream
    unsigned present;    // sink cells holding sinks of the tile (bit a)
    unsigned mutual;     // other sink cells of the own column met mutually by this pencil
    unsigned onesided;   // ... met one-sided
    bool triangle;       // the centre cell meets itself in a triangle
    int a, b;            // the tile's centre-cell sinks, as indices in the centre cell
};

struct Seg {
    int b, e;       // stream range
    bool mutual;
    unsigned mask;  // sink cells taking part
    int kind;       // 0 mutual columns, 1 centre cell, 2 one-sided columns
};

constexpr int NSEG = 6;

// Segment i of a tile's pass over its stream; false if it holds no pair.
__host__ __device__ __forceinline__ bool segment(const Stream &s, int R, int i, Seg &g) {
    const unsigned own = 1u << R;
    const bool tri = s.triangle && (s.present & own);
    const int o = s.Ms;
    switch (i) {
    case 0: g = Seg{0, s.Ms, true, ~0u, 0}; break;
    case 1: g = Seg{o, o + (tri ? s.b : s.own), true, s.mutual, 1}; break;
    case 2: g = Seg{o + s.b, o + s.own, true, tri ? (s.mutual | own) : 0u, 1}; break;
    case 3: g = Seg{o + s.a, o + s.b, false, tri ? own : 0u, 1}; break;
    case 4: g = Seg{o, o + s.own, false, s.onesided | (s.triangle ? 0u : own), 1}; break;
    default: g = Seg{o + s.own, s.M, false, ~0u, 2}; break;
    }
    g.mask &= s.present;
    return g.mask != 0 && g.e > g.b;
}

// Cells, and the slabs [lo, hi) that hold the sinks.  onesided: no pair is met
// mutually (a drop-in SIC: a sink's sum then runs over its sources in the same
// order whatever rows and z cells the SIC holds, and differs between SICs only
// by where pieces are cut and by the fixed-point unit: nodes of a z-split agree
// with the one domain to 2e-6 of |a| instead of 7.5e-6).
struct Geometry {
    const int64_t *__restrict__ cs;
    int cpd, R, lo, hi;
    bool onesided;
};

// Class of source column (dx, dy) for a pencil at slab x: 0 mutual, 1 the own
// column, 2 one-sided, 3 not met here (its pencil meets this one).
__host__ __device__ __forceinline__ int column_class(const Geometry &g, int x, int dx, int dy) {
    if (dx == 0 && dy == 0) return 1;
    const int xs = wrapc(x + dx, g.cpd);
    if (g.onesided || xs < g.lo || xs >= g.hi) return 2;
    return dx > 0 || (dx == 0 && dy > 0) ? 0 : 3;
}

// Counts of the pencil's sink cells -> the own column's part of Stream.
__host__ __device__ __forceinline__ void own_column(Stream &s, const int *spre, int R, bool onesided) {
    const int W = 2 * R + 1;
    s.own_begin = spre[R];
    s.own = spre[R + 1] - spre[R];
    s.triangle = !onesided && s.own >= DENSE_CELL;
    s.mutual = s.onesided = 0;
    for (int a = 0; a < W; a++) {
        if (a == R) continue;
        const bool dense = !onesided && max(s.own, spre[a + 1] - spre[a]) >= DENSE_CELL;
        if (!dense) s.onesided |= 1u << a;
        else if (a > R) s.mutual |= 1u << a;
    }
}

// The tile's part of Stream: sinks [s0, s1) of the pencil's sink stream.
__host__ __device__ __forceinline__ void own_tile(Stream &s, const int *spre, int R, int s0, int s1) {
    s.present = 0;
    for (int a = 0; a < 2 * R + 1; a++)
        if (max(s0, spre[a]) < min(s1, spre[a + 1])) s.present |= 1u << a;
    s.a = max(s0, spre[R]) - s.own_begin;
    s.b = min(s1, spre[R + 1]) - s.own_begin;
}

// ------------------------------------------------------------------------
// work list
// ------------------------------------------------------------------------

// SM sub-partition cycles of one chunk of 64 sources, by sinks per lane,
// mutual and one-sided, and of a tile's set-up: what the list is balanced by.
__host__ __device__ __forceinline__ long long chunk_cost(int S, bool mutual) {
    return mutual ? 600 + 1150 * S : 300 + 900 * S;
}
__host__ __device__ __forceinline__ long long tile_cost(int S) { return 2500 + 500 * S; }

struct PlanSums {
    unsigned long long pairs, slots;  // interactions, and slots evaluated for them
    unsigned long long cost;          // whole cycles: the same for any order of the additions
    int max_sources, max_sinks;  // of a pencil
    unsigned hist[NCLASS];
    unsigned cursor[NCLASS];
};

struct PlanArgs {
    Geometry g;
    int smax, forced;
    long long cap;  // largest cost of a piece
    PlanSums *sums;
    MutualItem *items;
};

// Order of the list: tiles of one S together, longest first within them.
// Warps that run at the same time then run the same loops (an unrolled loop
// is 3-6 KB of code; with S mixed by cost alone, clustered 128^3 took 8.2 ms
// in the unroll-8 shape instead of 6.9, clustered 60^3 0.81 instead of 0.76).
__device__ __forceinline__ int cost_class(int S, long long cost) {
    const int octave = 31 - __clz((int)min(max(cost, 1LL), 1LL << 24));  // 2^10 .. 2^24 told apart
    return (S >= 8 ? 0 : S == 4 ? 16 : S == 2 ? 32 : 48) + min(max(24 - octave, 0), 15);
}

// Pieces of a tile: none above `cap`, in proportion for tiles of few sinks,
// which come last; at least four chunks each.
__host__ __device__ __forceinline__ int tile_pieces(int S, int chunks, long long cost, long long cap) {
    if (S < 4) cap = cap * S / 4;
    const long long want = cap > 0 ? (cost + cap - 1) / cap : chunks, most = chunks / 4;
    const long long n = want < most ? want : most;
    return n > 1 ? (int)n : 1;
}

// Sinks per lane of the next tile of a pencil with `rem` sinks left: the
// smallest tile that holds them, but 65-96 take 64 + 32 slots instead of 128
// and 129-192 take 128 + 32 or 128 + 64 instead of 256 (by chunk_cost).
__host__ __device__ __forceinline__ int tile_S(int rem, int smax, int forced) {
    if (forced) return min(forced, smax);
    return rem <= 32 ? 1 : rem <= 96 ? 2 : (rem <= 192 || smax == 4) ? 4 : 8;
}

// One warp per pencil.  PASS 0: sums.  1: pieces per cost class.  2: emit.
template <int PASS>
__global__ void plan_kernel(PlanArgs p) {
    const Geometry &g = p.g;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int R = g.R, W = 2 * R + 1, cpd = g.cpd;
    __shared__ int s_pre[8][MAXW + 1];
    __shared__ unsigned s_hist[NCLASS];
    int *spre = s_pre[wib];
    if (PASS == 1) {
        for (int i = threadIdx.x; i < NCLASS; i += blockDim.x) s_hist[i] = 0;
        __syncthreads();
    }
    unsigned long long pairs = 0, slots = 0, cost = 0;
    int max_m = 0, max_s = 0;
    const int64_t c2 = (int64_t)cpd * cpd;
    const int64_t n_pencils = (int64_t)(g.hi - g.lo) * c2;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t q = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib; q < n_pencils; q += nw) {
        const int64_t pencil = q + g.lo * c2;
        const int cz = (int)(pencil % cpd), cy = (int)(pencil / cpd % cpd), cx = (int)(pencil / c2);
        int cls = 3, cnt = 0;
        if (lane < W * W) {
            const int dx = lane / W - R, dy = lane % W - R;
            const int64_t c = ((int64_t)wrapc(cx + dx, cpd) * cpd + wrapc(cy + dy, cpd)) * cpd + cz;
            cnt = (int)(g.cs[c + 1] - g.cs[c]);
            cls = column_class(g, cx, dx, dy);
        }
        int ms = cls == 0 ? cnt : 0, mo = cls == 2 ? cnt : 0, mt = cnt;
        for (int o = 16; o; o >>= 1) {
            ms += __shfl_xor_sync(FULL, ms, o);
            mo += __shfl_xor_sync(FULL, mo, o);
            mt += __shfl_xor_sync(FULL, mt, o);
        }
        int scnt = 0;
        if (lane < W) {
            const int64_t c = ((int64_t)cx * cpd + cy) * cpd + wrapc(cz + lane - R, cpd);
            scnt = (int)(g.cs[c + 1] - g.cs[c]);
        }
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, scnt, o);
            if (lane >= o) scnt += t;
        }
        __syncwarp();
        if (lane < W) spre[lane + 1] = scnt;
        if (lane == 0) spre[0] = 0;
        __syncwarp();
        const int np = spre[W];
        if (np == 0) continue;
        max_m = max(max_m, mt);
        max_s = max(max_s, np);
        if (PASS == 0 && lane == 0) pairs += (unsigned long long)np * mt;
        Stream s;
        s.Ms = ms;
        own_column(s, spre, R, g.onesided);
        s.M = ms + s.own + mo;
        // full tiles of smax * 32 sinks, then the rest in smaller ones
        const int Sf = p.forced ? min(p.forced, p.smax) : p.smax;
        const int nfull = np / (32 * Sf);
        const int rest = np - nfull * 32 * Sf;
        // the rest: at most two tiles
        for (int t = lane; t < nfull + 4; t += 32) {
            int s0, S;
            if (t < nfull) {
                s0 = t * 32 * Sf;
                S = Sf;
            } else {
                int left = rest, k = t - nfull;
                s0 = nfull * 32 * Sf;
                S = tile_S(left, p.smax, p.forced);
                while (k > 0 && left > 0) {
                    s0 += 32 * S;
                    left -= 32 * S;
                    S = tile_S(left, p.smax, p.forced);
                    k--;
                }
                if (left <= 0) continue;
            }
            const int s1 = min(np, s0 + 32 * S);
            own_tile(s, spre, R, s0, s1);
            int chunks = 0;
            long long c = 0;
            for (int i = 0; i < NSEG; i++) {
                Seg sg;
                if (!segment(s, R, i, sg)) continue;
                const int n = (sg.e - sg.b + CHUNK - 1) / CHUNK;
                chunks += n;
                c += n * chunk_cost(S, sg.mutual);
                slots += (unsigned long long)(32 * S) * n * CHUNK * (sg.mutual ? 2 : 1);
            }
            if (PASS == 0) {
                cost += c + tile_cost(S);
                continue;
            }
            const int pieces = tile_pieces(S, chunks, c, p.cap);
            const int cl = cost_class(S, c / pieces);
            if (PASS == 1) {
                atomicAdd(&s_hist[cl], (unsigned)pieces);
            } else {
                const unsigned at = atomicAdd(&p.sums->cursor[cl], (unsigned)pieces);
                for (int k = 0; k < pieces; k++)
                    p.items[at + k] =
                        MutualItem{(int)pencil, s0, s1 - s0, S, (int)((int64_t)chunks * k / pieces),
                                   (int)((int64_t)chunks * (k + 1) / pieces), 0, 0};
            }
        }
    }
    if (PASS == 0) {
        for (int o = 16; o; o >>= 1) {
            slots += __shfl_xor_sync(FULL, slots, o);
            cost += __shfl_xor_sync(FULL, cost, o);
        }
        if (lane == 0) {
            if (pairs) atomicAdd(&p.sums->pairs, pairs);
            atomicAdd(&p.sums->slots, slots);
            atomicAdd(&p.sums->cost, cost);
            atomicMax(&p.sums->max_sources, max_m);
            atomicMax(&p.sums->max_sinks, max_s);
        }
    }
    if (PASS == 1) {
        __syncthreads();
        for (int i = threadIdx.x; i < NCLASS; i += blockDim.x)
            if (s_hist[i]) atomicAdd(&p.sums->hist[i], s_hist[i]);
    }
}

// ------------------------------------------------------------------------
// the sweep
// ------------------------------------------------------------------------

struct MParams {
    const float4 *__restrict__ pos;
    Geometry g;
    const MutualItem *items;
    int n_items;
    int *counter;
    unsigned long long *acc;  // [3 or 4][n_range] fixed point
    unsigned char *bad;       // [n_range] a partial was not finite
    int64_t p0, n_range;
    float fscale, wscale;     // force and density sums to fixed point
    PairConst pc;
    float zshift[MAXW], xyshift[MAXW];
    float near_w;
};

struct WarpSmem {
    float4 bxy[2 * CHUNK];  // (-x, -x, -y, -y); group g of 32 at [64 g, 64 g + 64), twice
    float2 bz[2 * CHUNK];   // (-z, -z)
    int64_t cstart[MAXSRC];
    int32_t cpre[MAXSRC + 1];
    float csx[MAXSRC], csy[MAXSRC];
    float4 tbb;  // the tile's sink x and y range widened by near_w (single spline)
    int64_t sstart[MAXW];
    int32_t spre[MAXW + 1];
};

// Column and sink tables of a pencil: columns in stream order (mutual, own,
// one-sided).  Returns the number of mutual columns.
__device__ int setup_tables(const MParams &kp, int pencil, WarpSmem &ws, int lane, Stream &s) {
    const Geometry &g = kp.g;
    const int R = g.R, W = 2 * R + 1, cpd = g.cpd;
    const int cz = pencil % cpd, cy = (pencil / cpd) % cpd, cx = pencil / (cpd * cpd);
    int cls = 3, cnt = 0, dx = 0, dy = 0;
    int64_t st = 0;
    if (lane < W * W) {
        dx = lane / W - R;
        dy = lane % W - R;
        const int64_t c = ((int64_t)wrapc(cx + dx, cpd) * cpd + wrapc(cy + dy, cpd)) * cpd + cz;
        st = g.cs[c];
        cnt = (int)(g.cs[c + 1] - st);
        cls = column_class(g, cx, dx, dy);
    }
    const unsigned b0 = __ballot_sync(FULL, cls == 0), b2 = __ballot_sync(FULL, cls == 2);
    const unsigned below = (1u << lane) - 1;
    const int nm = __popc(b0);
    int slot = -1;
    if (cls == 0) slot = __popc(b0 & below);
    if (cls == 1) slot = nm;
    if (cls == 2) slot = nm + 1 + __popc(b2 & below);
    __syncwarp();
    if (slot >= 0) {
        ws.cstart[slot] = st;
        ws.cpre[slot + 1] = cnt;
        ws.csx[slot] = kp.xyshift[dx + R];
        ws.csy[slot] = kp.xyshift[dy + R];
    }
    __syncwarp();
    const int ncol = nm + 1 + __popc(b2);
    int v = lane < ncol ? ws.cpre[lane + 1] : 0;
    int scnt = 0;
    if (lane < W) {
        const int64_t c = ((int64_t)cx * cpd + cy) * cpd + wrapc(cz + lane - R, cpd);
        st = g.cs[c];
        scnt = (int)(g.cs[c + 1] - st);
        ws.sstart[lane] = st;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL, v, o), u = __shfl_up_sync(FULL, scnt, o);
        if (lane >= o) {
            v += t;
            scnt += u;
        }
    }
    if (lane < ncol) ws.cpre[lane + 1] = v;
    if (lane < W) ws.spre[lane + 1] = scnt;
    if (lane == 0) ws.cpre[0] = ws.spre[0] = 0;
    __syncwarp();
    s.Ms = ws.cpre[nm];
    s.M = ws.cpre[ncol];
    own_column(s, ws.spre, R, g.onesided);
    return nm;
}

// Source record for stream index i (null record far away past the end), in
// the pencil frame; p: its particle.  FLAG: w = 1 if it lies inside the
// tile's sink box widened by near_w.
template <bool FLAG>
__device__ __forceinline__ float4 load_src(const MParams &kp, const WarpSmem &ws, int i, int end,
                                           int &k, float zlo, float zhi, int &p_out) {
    if (i >= end) {
        p_out = -1;
        return make_float4(1e18f, 1e18f, 1e18f, 0.f);
    }
    while (i >= ws.cpre[k + 1]) k++;
    const int64_t p = ws.cstart[k] + (i - ws.cpre[k]);
    p_out = (int)p;
    float4 t = __ldg(&kp.pos[p]);
    t.x += ws.csx[k];
    t.y += ws.csy[k];
    if (FLAG) t.w = inside(t, ws.tbb, zlo, zhi);
    return t;
}

// The lane's sinks and their sums.  Scalar form (S == 1) in one-element
// arrays of float, paired form (S >= 2) sinks 2q, 2q + 1 in the halves.
template <int S>
struct Sinks {
    static constexpr int N = S >= 2 ? S / 2 : 1;
    float2 x[N], y[N], z[N];     // positions (S == 1: .x only)
    float2 px[N], py[N], pz[N];  // FP32 partials
    float2 w[N];                 // density, FP32 partials
};

struct Reaction {
    float2 x, y, z, w;
};

// The lane's sinks against the source staged at bxy[j], bz[j].
template <int SOFT, bool DENS, int S, bool NEAR, bool MUTUAL>
__device__ __forceinline__ void meet(const float4 &t, const float2 &tz, Sinks<S> &k, Reaction &r,
                                     const PairConst &pc) {
    const float2 tx = make_float2(t.x, t.y), ty = make_float2(t.z, t.w);
    // density terms b2 - |d|^2: from r^2 where its r2_add is below the rounding
    // of b2 (mutual_bits); Plummer's eps^2 is not, and would leave its own
    // rounding in every term, so there |d|^2 is formed for itself (uniform
    // n = 6000, b2 = 32 eps^2: density error 1.6e-7 from r^2, 1.4e-7 so).  The
    // sum rounds to b2, but as a register: read from the parameters each time,
    // density 100^3 took 4.17 ms instead of 4.10
    const float b2 = SOFT == SOFT_PLUMMER ? pc.b2 : pc.b2 + r2_add<SOFT>(pc);
#pragma unroll
    for (int q = 0; q < Sinks<S>::N; q++) {
        if constexpr (S == 1) {
            const float dx = k.x[0].x + tx.x, dy = k.y[0].x + ty.x, dz = k.z[0].x + tz.x;
            const float r2 = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, r2_add<SOFT>(pc))));
            const float g = pair_g<SOFT, NEAR, Step::SHORT>(r2, pc);
            k.px[0].x = fmaf(g, dx, k.px[0].x);
            k.py[0].x = fmaf(g, dy, k.py[0].x);
            k.pz[0].x = fmaf(g, dz, k.pz[0].x);
            if (MUTUAL) {
                r.x.x = fmaf(g, dx, r.x.x);
                r.y.x = fmaf(g, dy, r.y.x);
                r.z.x = fmaf(g, dz, r.z.x);
            }
            if (DENS) {
                const float d = SOFT == SOFT_PLUMMER ? dens_term(dx, dy, dz, pc.b2) : fmaxf(b2 - r2, 0.f);
                k.w[0].x += d;
                if (MUTUAL) r.w.x += d;
            }
        } else {
            const float2 dx = add2(k.x[q], tx), dy = add2(k.y[q], ty), dz = add2(k.z[q], tz);
            const float2 r2 = r2_x2(dx, dy, dz, r2_add<SOFT>(pc));
            const float2 g = pair_g_x2<SOFT, NEAR, Step::SHORT>(r2, pc);
            k.px[q] = fma2(g, dx, k.px[q]);
            k.py[q] = fma2(g, dy, k.py[q]);
            k.pz[q] = fma2(g, dz, k.pz[q]);
            if (MUTUAL) {
                r.x = fma2(g, dx, r.x);
                r.y = fma2(g, dy, r.y);
                r.z = fma2(g, dz, r.z);
            }
            if (DENS) {
                const float2 s2 = SOFT == SOFT_PLUMMER ? fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))) : r2;
                const float2 e = fma2(s2, dup2(-1.f), dup2(b2));
                const float2 d = make_float2(fmaxf(e.x, 0.f), fmaxf(e.y, 0.f));
                k.w[q] = add2(k.w[q], d);
                if (MUTUAL) r.w = add2(r.w, d);
            }
        }
    }
}

// One-sided: m (a multiple of UNR) staged sources of a group, broadcast.
template <int SOFT, bool DENS, int S, bool NEAR, int UNR>
__device__ __forceinline__ void group_onesided(const float4 *bxy, const float2 *bz, int m,
                                               Sinks<S> &k, const PairConst &pc) {
    Reaction none;
#pragma unroll 1
    for (int j = 0; j < m; j += UNR) {
#pragma unroll
        for (int u = 0; u < UNR; u++)
            meet<SOFT, DENS, S, NEAR, false>(bxy[j + u], bz[j + u], k, none, pc);
    }
}

// Mutual: the 32 sources of a group, lane l meeting source (l + t) mod 32 in
// step t (bxy and bz at the lane's own slot).  Returns the reaction of the
// lane's own source.
template <int SOFT, bool DENS, int S, bool NEAR, int UNR>
__device__ __forceinline__ float4 group_mutual(const float4 *bxy, const float2 *bz, int from,
                                               Sinks<S> &k, const PairConst &pc) {
    Reaction r;
    r.x = r.y = r.z = r.w = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int t = 0; t < GROUP; t += UNR) {
#pragma unroll
        for (int u = 0; u < UNR; u++) {
            meet<SOFT, DENS, S, NEAR, true>(bxy[t + u], bz[t + u], k, r, pc);
            r.x.x = __shfl_sync(FULL, r.x.x, from);
            r.y.x = __shfl_sync(FULL, r.y.x, from);
            r.z.x = __shfl_sync(FULL, r.z.x, from);
            if (S > 1) {
                r.x.y = __shfl_sync(FULL, r.x.y, from);
                r.y.y = __shfl_sync(FULL, r.y.y, from);
                r.z.y = __shfl_sync(FULL, r.z.y, from);
            }
            if (DENS) {
                r.w.x = __shfl_sync(FULL, r.w.x, from);
                if (S > 1) r.w.y = __shfl_sync(FULL, r.w.y, from);
            }
        }
    }
    return make_float4(r.x.x + r.x.y, r.y.x + r.y.y, r.z.x + r.z.y, r.w.x + r.w.y);
}

__device__ __forceinline__ void add_fixed(unsigned long long *a, long long v) {
    atomicAdd(a, (unsigned long long)v);
}

__device__ __forceinline__ bool finite3(float x, float y, float z) {
    return fabsf(x) <= 3.4e38f && fabsf(y) <= 3.4e38f && fabsf(z) <= 3.4e38f;
}

template <int S>
__device__ __forceinline__ void load_sinks(const MParams &kp, const WarpSmem &ws,
                                           const MutualItem &it, int lane, unsigned mask,
                                           Sinks<S> &k) {
#pragma unroll
    for (int s = 0; s < S; s++) {
        const int j = s * 32 + lane;
        float x = -1e18f, y = -1e18f, z = -1e18f;  // taking no part: far from every source
        if (j < it.nsink) {
            const int i = it.sink_begin + j;
            int a = 0;
            while (i >= ws.spre[a + 1]) a++;
            if (mask >> a & 1) {
                const float4 q = __ldg(&kp.pos[ws.sstart[a] + (i - ws.spre[a])]);
                x = q.x;
                y = q.y;
                z = q.z + kp.zshift[a];
            }
        }
        if (s & 1) {
            k.x[s / 2].y = x;
            k.y[s / 2].y = y;
            k.z[s / 2].y = z;
        } else {
            k.x[s / 2].x = x;
            k.y[s / 2].x = y;
            k.z[s / 2].x = z;
        }
    }
}

// Fold a pair's partial into its compensated sums (hx, hy, lx, ly) and clear it.
__device__ __forceinline__ void fold_smem(float4 &v, float2 &p) {
    float2 h = make_float2(v.x, v.y), l = make_float2(v.z, v.w);
    fold2(h, l, p, false);
    v = make_float4(h.x, h.y, l.x, l.y);
}

// hl: the lane's compensated sums of its sinks, in shared memory.
template <int SOFT, bool DENS, int S, int UNR>
__device__ void run_item(const MParams &kp, WarpSmem &ws, float4 *hl, const MutualItem &it, int lane,
                         Stream &s, int nm) {
    constexpr bool FLAG = has_near(SOFT);
    constexpr int N = Sinks<S>::N;
    constexpr int SIDE = S == 8 && UNR > 2 ? 2 : UNR;  // unroll of the less used loops
    const int R = kp.g.R;
    Sinks<S> k;
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < N; q++) {
        k.px[q] = k.py[q] = k.pz[q] = k.w[q] = zero;
#pragma unroll
        for (int c = 0; c < (DENS ? 4 : 3); c++) hl[(c * N + q) * 32] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    own_tile(s, ws.spre, R, it.sink_begin, it.sink_begin + it.nsink);
    unsigned loaded = s.present;
    load_sinks<S>(kp, ws, it, lane, loaded, k);
    float zlo = 3.0e38f, zhi = -3.0e38f;
    if (FLAG) {  // the tile's sink bounding box, widened
        float xlo = 3.0e38f, xhi = -3.0e38f, ylo = 3.0e38f, yhi = -3.0e38f;
#pragma unroll
        for (int i = 0; i < S; i++)
            if (i * 32 + lane < it.nsink) {
                const float x = i & 1 ? k.x[i / 2].y : k.x[i / 2].x;
                const float y = i & 1 ? k.y[i / 2].y : k.y[i / 2].x;
                const float z = i & 1 ? k.z[i / 2].y : k.z[i / 2].x;
                xlo = fminf(xlo, x);
                xhi = fmaxf(xhi, x);
                ylo = fminf(ylo, y);
                yhi = fmaxf(yhi, y);
                zlo = fminf(zlo, z);
                zhi = fmaxf(zhi, z);
            }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            xlo = fminf(xlo, __shfl_xor_sync(FULL, xlo, off));
            xhi = fmaxf(xhi, __shfl_xor_sync(FULL, xhi, off));
            ylo = fminf(ylo, __shfl_xor_sync(FULL, ylo, off));
            yhi = fmaxf(yhi, __shfl_xor_sync(FULL, yhi, off));
            zlo = fminf(zlo, __shfl_xor_sync(FULL, zlo, off));
            zhi = fmaxf(zhi, __shfl_xor_sync(FULL, zhi, off));
        }
        const float w = kp.near_w;
        __syncwarp();
        if (lane == 0) ws.tbb = make_float4(xlo - w, xhi + w, ylo - w, yhi + w);
        __syncwarp();
        zlo -= w;
        zhi += w;
    }
    auto fold_all = [&]() {
#pragma unroll
        for (int q = 0; q < N; q++) {
            fold_smem(hl[q * 32], k.px[q]);
            fold_smem(hl[(N + q) * 32], k.py[q]);
            fold_smem(hl[(2 * N + q) * 32], k.pz[q]);
            if (DENS) fold_smem(hl[(3 * N + q) * 32], k.w[q]);
        }
    };
    // drop-in SICs fold every chunk (+1 %): their long one-sided streams, split
    // less finely than the former 64-sink tiles, would otherwise have raised
    // the error of uniform 64^3 from 2.1e-7 to 3.0e-7
    const int fold_every = kp.g.onesided ? 1 : FOLD;
    int vc = 0, since_fold = 0;  // chunks before this segment; chunks since the last fold
#pragma unroll 1
    for (int i = 0; i < NSEG; i++) {
        Seg sg;
        if (!segment(s, R, i, sg)) continue;
        const int nch = (sg.e - sg.b + CHUNK - 1) / CHUNK;
        const int ch0 = max(it.c0 - vc, 0), ch1 = min(it.c1 - vc, nch);
        vc += nch;
        if (ch0 >= ch1) continue;
        if (sg.mask != loaded) {
            loaded = sg.mask;
            load_sinks<S>(kp, ws, it, lane, loaded, k);
        }
        const int end = min(sg.e, sg.b + ch1 * CHUNK);
        int base = sg.b + ch0 * CHUNK;
        int k0 = sg.kind == 0 ? 0 : nm + (sg.kind - 1), k1 = k0, n0, n1;
        float4 pre0 = load_src<FLAG>(kp, ws, base + lane, end, k0, zlo, zhi, n0);
        float4 pre1 = load_src<FLAG>(kp, ws, base + GROUP + lane, end, k1, zlo, zhi, n1);
#pragma unroll 1
        for (; base < end; base += CHUNK) {
            // both branches only if a source may lie within eps of a sink of the tile
            const bool near = FLAG && __any_sync(FULL, pre0.w + pre1.w != 0.f);
            const int src0 = n0, src1 = n1;
            __syncwarp();
            const float4 v0 = make_float4(-pre0.x, -pre0.x, -pre0.y, -pre0.y);
            const float4 v1 = make_float4(-pre1.x, -pre1.x, -pre1.y, -pre1.y);
            const float2 w0 = make_float2(-pre0.z, -pre0.z), w1 = make_float2(-pre1.z, -pre1.z);
            ws.bxy[lane] = v0;
            ws.bz[lane] = w0;
            ws.bxy[CHUNK + lane] = v1;
            ws.bz[CHUNK + lane] = w1;
            if (sg.mutual) {
                ws.bxy[GROUP + lane] = v0;
                ws.bz[GROUP + lane] = w0;
                ws.bxy[CHUNK + GROUP + lane] = v1;
                ws.bz[CHUNK + GROUP + lane] = w1;
            }
            __syncwarp();
            if (base + CHUNK < end) {
                pre0 = load_src<FLAG>(kp, ws, base + CHUNK + lane, end, k0, zlo, zhi, n0);
                pre1 = load_src<FLAG>(kp, ws, base + CHUNK + GROUP + lane, end, k1, zlo, zhi, n1);
            }
            const int m = min(CHUNK, end - base);
#pragma unroll 1
            for (int gr = 0; gr * GROUP < m; gr++) {
                const float4 *bxy = ws.bxy + gr * CHUNK;
                const float2 *bz = ws.bz + gr * CHUNK;
                if (sg.mutual) {
                    const int from = (lane + 1) & 31;
                    float4 r;
                    if (FLAG && near)
                        r = group_mutual<SOFT, DENS, S, true, SIDE>(bxy + lane, bz + lane, from, k,
                                                                   kp.pc);
                    else
                        r = group_mutual<SOFT, DENS, S, false, UNR>(bxy + lane, bz + lane, from, k,
                                                                    kp.pc);
                    const int src = gr ? src1 : src0;
                    if (src >= 0) {
                        const int64_t idx = src - kp.p0;
                        unsigned long long *a = kp.acc + idx;
                        add_fixed(a, __float2ll_rn(-r.x * kp.fscale));
                        add_fixed(a + kp.n_range, __float2ll_rn(-r.y * kp.fscale));
                        add_fixed(a + 2 * kp.n_range, __float2ll_rn(-r.z * kp.fscale));
                        if (DENS) add_fixed(a + 3 * kp.n_range, __float2ll_rn(r.w * kp.wscale));
                        if (!finite3(r.x, r.y, r.z)) kp.bad[idx] = 1;
                    }
                } else {
                    const int mg = min(GROUP, m - gr * GROUP);
                    const int mp = (mg + SIDE - 1) / SIDE * SIDE;  // padding reads null records
                    if (FLAG && near)
                        group_onesided<SOFT, DENS, S, true, SIDE>(bxy, bz, mp, k, kp.pc);
                    else
                        group_onesided<SOFT, DENS, S, false, SIDE>(bxy, bz, mp, k, kp.pc);
                }
            }
            if (++since_fold >= fold_every) {
                fold_all();
                since_fold = 0;
            }
        }
    }
    fold_all();
#pragma unroll
    for (int i = 0; i < S; i++) {
        const int j = i * 32 + lane;
        if (j >= it.nsink) continue;
        const int q = i / 2;
        const bool odd = i & 1;
        const float4 vx = hl[q * 32], vy = hl[(N + q) * 32], vz = hl[(2 * N + q) * 32];
        const float hx = odd ? vx.y : vx.x, lx = odd ? vx.w : vx.z;
        const float hy = odd ? vy.y : vy.x, ly = odd ? vy.w : vy.z;
        const float hz = odd ? vz.y : vz.x, lz = odd ? vz.w : vz.z;
        const int si = it.sink_begin + j;
        int a = 0;
        while (si >= ws.spre[a + 1]) a++;
        const int64_t idx = ws.sstart[a] + (si - ws.spre[a]) - kp.p0;
        unsigned long long *o = kp.acc + idx;
        const float f = kp.fscale;
        add_fixed(o, __float2ll_rn(hx * f) + __float2ll_rn(lx * f));
        add_fixed(o + kp.n_range, __float2ll_rn(hy * f) + __float2ll_rn(ly * f));
        add_fixed(o + 2 * kp.n_range, __float2ll_rn(hz * f) + __float2ll_rn(lz * f));
        if (DENS) {
            const float4 vw = hl[(3 * N + q) * 32];
            add_fixed(o + 3 * kp.n_range, __float2ll_rn((odd ? vw.y : vw.x) * kp.wscale) +
                                              __float2ll_rn((odd ? vw.w : vw.z) * kp.wscale));
        }
        if (!finite3(hx, hy, hz)) kp.bad[idx] = 1;
    }
}

// What was tried in the loop, uniform 160^3: the reaction moved as two halves
// (six shuffles, no addition) 12.15 ms, as one (three shuffles, three FADD)
// 12.46; sources prefetched a step ahead 12.56; 3 CTAs an SM 12.9; unroll 4
// of the less used loops of 8-sink tiles instead of 2: clustered 128^3 9.1 ms
// instead of 8.0 (instruction fetch), so they stay at 2.
//
// Shape knobs as in the one-sided kernel: SMAX largest tile 32*SMAX sinks,
// UNR sources per unrolled step, MINB CTAs per SM.
template <int SOFT, bool DENS, int SMAX, int UNR, int MINB>
__global__ void __launch_bounds__(WPC * 32, MINB) mutual_kernel(const __grid_constant__ MParams kp) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpSmem &ws = reinterpret_cast<WarpSmem *>(smem_raw)[warp];
    float4 *hl = reinterpret_cast<float4 *>(smem_raw + sizeof(WarpSmem) * WPC) +
                 warp * ((DENS ? 4 : 3) * (SMAX / 2) * 32) + lane;
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(kp.counter, 1);
        i = __shfl_sync(FULL, i, 0);
        if (i >= kp.n_items) break;
        const MutualItem it = kp.items[i];
        Stream s;
        const int nm = setup_tables(kp, it.pencil, ws, lane, s);
        if (it.S == 1)
            run_item<SOFT, DENS, 1, UNR>(kp, ws, hl, it, lane, s, nm);
        else if (it.S == 2)
            run_item<SOFT, DENS, 2, UNR>(kp, ws, hl, it, lane, s, nm);
        else if (SMAX == 4 || it.S == 4)
            run_item<SOFT, DENS, 4, UNR>(kp, ws, hl, it, lane, s, nm);
        else
            run_item<SOFT, DENS, (SMAX >= 8 ? 8 : 4), UNR>(kp, ws, hl, it, lane, s, nm);
    }
}

// The sweep without a work list (allocation-free entry point): warps take
// (pencil, piece) pairs from the counter; a piece is every pieces-th part of
// each of the pencil's tiles.
template <int SOFT, bool DENS>
__global__ void __launch_bounds__(WPC * 32, 2)
    mutual_noalloc_kernel(const __grid_constant__ MParams kp, int pencil0, int n_pencils, int pieces) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpSmem &ws = reinterpret_cast<WarpSmem *>(smem_raw)[warp];
    float4 *hl = reinterpret_cast<float4 *>(smem_raw + sizeof(WarpSmem) * WPC) + warp * ((DENS ? 4 : 3) * 2 * 32) + lane;
    const int W = 2 * kp.g.R + 1;
    for (;;) {
        int q = 0;
        if (lane == 0) q = atomicAdd(kp.counter, 1);
        q = __shfl_sync(FULL, q, 0);
        if (q >= n_pencils * pieces) break;
        const int piece = q % pieces;
        MutualItem it{pencil0 + q / pieces, 0, 0, 0, 0, 0, 0, 0};
        Stream s;
        const int nm = setup_tables(kp, it.pencil, ws, lane, s);
        const int np = ws.spre[W];
        while (it.sink_begin < np) {
            it.S = tile_S(np - it.sink_begin, 4, 0);
            it.nsink = min(np - it.sink_begin, 32 * it.S);
            own_tile(s, ws.spre, kp.g.R, it.sink_begin, it.sink_begin + it.nsink);
            int chunks = 0;
            for (int i = 0; i < NSEG; i++) {
                Seg sg;
                if (segment(s, kp.g.R, i, sg)) chunks += (sg.e - sg.b + CHUNK - 1) / CHUNK;
            }
            it.c0 = (int)((int64_t)chunks * piece / pieces);
            it.c1 = (int)((int64_t)chunks * (piece + 1) / pieces);
            if (it.c0 < it.c1) {
                if (it.S == 1)
                    run_item<SOFT, DENS, 1, 4>(kp, ws, hl, it, lane, s, nm);
                else if (it.S == 2)
                    run_item<SOFT, DENS, 2, 4>(kp, ws, hl, it, lane, s, nm);
                else
                    run_item<SOFT, DENS, 4, 4>(kp, ws, hl, it, lane, s, nm);
            }
            it.sink_begin += it.nsink;
        }
    }
}

typedef void (*NoallocFn)(MParams, int, int, int);

NoallocFn noalloc_fn(int soft, bool dens) {
    switch (soft) {
    case SOFT_PLUMMER: return dens ? mutual_noalloc_kernel<SOFT_PLUMMER, true> : mutual_noalloc_kernel<SOFT_PLUMMER, false>;
    case SOFT_SINGLE_SPLINE:
        return dens ? mutual_noalloc_kernel<SOFT_SINGLE_SPLINE, true> : mutual_noalloc_kernel<SOFT_SINGLE_SPLINE, false>;
    case SOFT_CUBIC_SPLINE:
        return dens ? mutual_noalloc_kernel<SOFT_CUBIC_SPLINE, true> : mutual_noalloc_kernel<SOFT_CUBIC_SPLINE, false>;
    default:
        return dens ? mutual_noalloc_kernel<SOFT_CUBIC_PLUMMER, true> : mutual_noalloc_kernel<SOFT_CUBIC_PLUMMER, false>;
    }
}

typedef void (*MutualFn)(MParams);

struct Shape {
    int smax, unr, minb;
    const char *name;
};
constexpr Shape SHAPES[MUTUAL_SHAPES] = {
    {4, 4, 2, "sinks/lane<=4 unroll 4, 2 CTAs/SM"},
    {8, 4, 2, "sinks/lane<=8 unroll 4, 2 CTAs/SM"},
    {4, 8, 2, "sinks/lane<=4 unroll 8, 2 CTAs/SM"},
    {4, 2, 3, "sinks/lane<=4 unroll 2, 3 CTAs/SM"},
    {8, 2, 2, "sinks/lane<=8 unroll 2, 2 CTAs/SM"},
};

template <int SOFT, bool DENS, int I>
MutualFn shape_fn() {
    return mutual_kernel<SOFT, DENS, SHAPES[I].smax, SHAPES[I].unr, SHAPES[I].minb>;
}

template <int SOFT>
MutualFn shape(int v) {
    switch (v) {
    case 1: return shape_fn<SOFT, false, 1>();
    case 2: return shape_fn<SOFT, false, 2>();
    case 3: return shape_fn<SOFT, false, 3>();
    case 4: return shape_fn<SOFT, false, 4>();
    default: return shape_fn<SOFT, false, 0>();
    }
}

MutualFn pick(int soft, bool dens, int v) {
    switch (soft) {
    case SOFT_PLUMMER: return dens ? shape_fn<SOFT_PLUMMER, true, 0>() : shape<SOFT_PLUMMER>(v);
    case SOFT_SINGLE_SPLINE:
        return dens ? shape_fn<SOFT_SINGLE_SPLINE, true, 0>() : shape<SOFT_SINGLE_SPLINE>(v);
    case SOFT_CUBIC_SPLINE:
        return dens ? shape_fn<SOFT_CUBIC_SPLINE, true, 0>() : shape_fn<SOFT_CUBIC_SPLINE, false, 0>();
    default:
        return dens ? shape_fn<SOFT_CUBIC_PLUMMER, true, 0>() : shape_fn<SOFT_CUBIC_PLUMMER, false, 0>();
    }
}

int smax_of(const nf_config &cfg, int v) {
    return SHAPES[tunable(cfg.softening, cfg.b2 > 0.f) ? v : 0].smax;
}

size_t smem_bytes(int smax, bool dens) {
    return (sizeof(WarpSmem) + (dens ? 4 : 3) * (smax / 2) * 32 * sizeof(float4)) * WPC;
}

}  // namespace

// Fixed-point bits of the force (and density) unit for softening parameter
// eps, b2 and at most n_max sources a sink; false where the engine does not
// apply.  Largest pair force g d in the kernel's units, with softening length
// e: Plummer 2/(3 sqrt 3) e^-2; single spline (far units) the maximum of
// u (10 - 15 u + 6 u^2) = 2.01 e^-2; cubic spline < 1.4 e^-2; cubic Plummer
// 2^(2/3)/3 e^-2 (the unit of the Newton step, 2/3, is left in as margin).
// n_max times that is put at 2^62 at most.  The engine applies where the unit
// is at most 2^-25 h^-2 (h the cell width: the force of a pair a cell apart):
// the rounding of the few hundred additions to a sink is then several times
// below the FP32 rounding of its partials, whose terms are that size.
static bool mutual_bits(int soft, double eps, double b2, int cpd, double n_max, int *fbits,
                        int *wbits) {
    double e, a;
    switch (soft) {
    case SOFT_PLUMMER: e = sqrt(eps), a = 0.39; break;
    case SOFT_SINGLE_SPLINE: e = 1.0 / sqrt(eps), a = 2.1; break;
    case SOFT_CUBIC_SPLINE: e = 1.0 / eps, a = 1.4; break;
    default: e = cbrt(eps), a = 0.54; break;
    }
    n_max = std::max(n_max, 1.0);
    const double bound = 1.02 * a / (e * e) * n_max;
    if (!(bound > 0.0) || !std::isfinite(bound)) return false;
    *fbits = 62 - (int)std::ceil(std::log2(bound));
    const double h = 1.0 / (double)cpd;
    if (std::ldexp(1.0, -*fbits) * h * h > std::ldexp(1.0, -25)) return false;
    // the density sum, at most n_max b2; taken from r^2 (Plummer: from |d|^2)
    // with its r2_add, which must be below half a unit of b2's last place
    const double add = soft == SOFT_PLUMMER ? 0.0 : soft == SOFT_CUBIC_PLUMMER ? 1e-16 : 1e-25;
    if (b2 > 0.0 && b2 < std::ldexp(add, 25)) return false;
    *wbits = b2 > 0.0 ? 62 - (int)std::ceil(std::log2(1.02 * b2 * n_max)) : 0;
    // both scales are floats
    return std::abs(*fbits) <= 100 && std::abs(*wbits) <= 100;
}

size_t mutual_scratch_bytes(int64_t n_range, int nc) { return (size_t)n_range * (8 * nc + 1); }

const char *mutual_shape_name(int v) { return SHAPES[v].name; }

int mutual_grid(nf_ctx *ctx, int variant) {
    MutualFn fn = pick(ctx->cfg.softening, ctx->cfg.b2 > 0.f, variant);
    const size_t smem = smem_bytes(smax_of(ctx->cfg, variant), ctx->cfg.b2 > 0.f);
    int per_sm = 0;
    if (cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)fn, WPC * 32, smem) !=
            cudaSuccess) {
        cudaGetLastError();
        per_sm = 1;
    }
    return ctx->sms * std::max(per_sm, 1);
}

// The work list of sink pencils of the middle slab of a drop-in SIC's mini box
// (2R+1 slabs, cell table cs on the host), made on the host: a SIC is a few
// hundred pencils, and its list travels with its positions.  Every pair is
// met one-sided.  Fills pl's units and counts and `items`; false where the
// engine does not apply.  `warps`: of a full launch.
bool mutual_sic_list(const nf_config &cfg, int cpd, const std::vector<SicPencil> &pencils, const int64_t *cs,
                     int warps, Plan &pl, std::vector<MutualItem> &items) {
    if (cfg.accumulation != NF_ACC_COMPENSATED) return false;
    const int R = cfg.near_field_radius, W = 2 * R + 1;
    const int smax = smax_of(cfg, 0);
    struct Tile {
        MutualItem it;
        int chunks, pieces;
        long long cost;  // of the tile, then of a piece
    };
    std::vector<Tile> tiles;
    tiles.reserve(4 * pencils.size());
    int64_t max_sources = 0;
    long long total = 0;
    pl.pairs = 0;
    for (const SicPencil &p : pencils) {
        if (p.sources > INT32_MAX / 8 || p.first + p.n > INT32_MAX / 8) return false;
        max_sources = std::max(max_sources, p.sources);
        pl.pairs += (uint64_t)p.n * (uint64_t)p.sources;
        const int64_t centre = ((int64_t)R * cpd + p.y) * cpd + p.z;
        const int own = (int)(cs[centre + 1] - cs[centre]);
        // the stream: the centre cell, then all other columns
        const int chunks = (own + CHUNK - 1) / CHUNK + ((int)p.sources - own + CHUNK - 1) / CHUNK;
        for (int64_t s0 = p.first, end = p.first + p.n; s0 < end;) {
            const int S = tile_S((int)(end - s0), smax, cfg.sinks_per_lane);
            const int n = (int)std::min<int64_t>(end - s0, 32 * S);
            const long long cost = chunks * chunk_cost(S, false);
            tiles.push_back(Tile{MutualItem{(int)centre, (int)s0, n, S, 0, 0, 0, 0}, chunks, 1, cost});
            total += cost + tile_cost(S);
            s0 += n;
        }
    }
    if (!mutual_bits(cfg.softening, cfg.eps, cfg.b2, cpd, (double)W * max_sources, &pl.fbits, &pl.wbits))
        return false;
    // pieces of two warps' share: several SICs run side by side (driver over
    // uniform 160^3: 31 ms, with one warp's share 36, clustered 96^3 9.0 and 10.1)
    const long long cap = std::max(1LL, 2 * total / warps);
    for (Tile &t : tiles) {
        t.pieces = tile_pieces(t.it.S, t.chunks, t.cost, cap);
        t.cost /= t.pieces;
    }
    std::sort(tiles.begin(), tiles.end(), [](const Tile &a, const Tile &b) {
        return a.it.S != b.it.S ? a.it.S > b.it.S : a.cost > b.cost;
    });
    items.clear();
    for (const Tile &t : tiles)
        for (int k = 0; k < t.pieces; k++) {
            MutualItem it = t.it;
            it.c0 = (int)((int64_t)t.chunks * k / t.pieces);
            it.c1 = (int)((int64_t)t.chunks * (k + 1) / t.pieces);
            items.push_back(it);
        }
    pl.mutual = true;
    pl.variant = 0;
    pl.lo = R;
    pl.hi = R + 1;
    pl.onesided = true;
    pl.n_mutual = (int)items.size();
    return true;
}

// The work list of slabs [lo, hi): NF_OK with pl.mutual false where the engine
// does not apply (the caller then plans the one-sided sweep).
nf_status mutual_plan(nf_ctx *ctx, const nf_box *box, int lo, int hi, int variant, Plan &pl) {
    cudaStream_t st = ctx->stream;
    pl.mutual = false;
    const nf_config &cfg = ctx->cfg;
    if (cfg.accumulation != NF_ACC_COMPENSATED) return NF_OK;
    const int R = cfg.near_field_radius, W = 2 * R + 1;
    PlanArgs a{};
    a.g = Geometry{box->d_cs, box->cpd, R, lo, hi, false};
    a.smax = smax_of(cfg, variant);
    a.forced = cfg.sinks_per_lane;
    NF_CUDA(pool_alloc(ctx, &a.sums, sizeof(PlanSums)));
    PlanSums h;
    const int64_t pencils = (int64_t)(hi - lo) * box->cpd * box->cpd;
    const int blocks = (int)std::min<int64_t>((pencils + 7) / 8, (int64_t)ctx->sms * 16);
    cudaError_t e = cudaMemsetAsync(a.sums, 0, sizeof(PlanSums), st);
    if (e == cudaSuccess) {
        plan_kernel<0><<<blocks, 256, 0, st>>>(a);
        e = cudaMemcpyAsync(&h, a.sums, sizeof(h), cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    const float eps = box->eps > 0.f ? box->eps : cfg.eps;
    if (e != cudaSuccess || h.max_sources > INT32_MAX / 8 || h.max_sinks > INT32_MAX / 8 ||
        !mutual_bits(cfg.softening, eps, cfg.b2, box->cpd, (double)W * h.max_sources, &pl.fbits,
                     &pl.wbits)) {
        pool_free(ctx, a.sums);
        return e != cudaSuccess ? cuda_fail(e, "work list (sums)") : NF_OK;
    }
    pl.grid = mutual_grid(ctx, variant);
    pl.warps = pl.grid * WPC;
    // an eighth of a warp's share: 6, 12 and 20 parts were within 2 % on large
    // sweeps, 3-6 % slower on ones of a millisecond
    a.cap = std::max<long long>(1, (long long)(h.cost / ((unsigned long long)pl.warps * 8)));
    plan_kernel<1><<<blocks, 256, 0, st>>>(a);
    e = cudaMemcpyAsync(h.hist, a.sums->hist, sizeof(h.hist), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    uint64_t n = 0;
    if (e == cudaSuccess) {
        for (int i = 0; i < NCLASS; i++) {
            h.cursor[i] = (unsigned)n;
            n += h.hist[i];
        }
        if (n > (uint64_t)INT32_MAX / 2) {
            pool_free(ctx, a.sums);
            return NF_OK;
        }
        e = pool_alloc(ctx, &pl.d_mutual, n * sizeof(MutualItem));
    }
    if (e == cudaSuccess) {
        a.items = pl.d_mutual;
        e = cudaMemcpyAsync(a.sums->cursor, h.cursor, sizeof(h.cursor), cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess) {
        plan_kernel<2><<<blocks, 256, 0, st>>>(a);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    pool_free(ctx, a.sums);
    if (e != cudaSuccess) return cuda_fail(e, "work list");
    pl.mutual = true;
    pl.n_mutual = (int)n;
    pl.pairs = h.pairs;
    pl.padded_pairs = h.slots;
    return NF_OK;
}

struct ZeroArgs {
    uint4 *a;
    size_t n16;
    unsigned char *tail;
    int tail_bytes;
    int *counter;
};

static ZeroArgs zero_args(nf_ctx *ctx, const Plan &pl, void *scratch, int *counter) {
    const size_t bytes = mutual_scratch_bytes(pl.n_range, ctx->cfg.b2 > 0.f ? 4 : 3);
    return ZeroArgs{(uint4 *)scratch, bytes / 16, (unsigned char *)scratch + bytes / 16 * 16,
                    (int)(bytes % 16), counter};
}

static __device__ __forceinline__ void zero_range(const ZeroArgs &z, int64_t i0, int64_t stride) {
    for (int64_t i = i0; i < (int64_t)z.n16; i += stride) z.a[i] = make_uint4(0, 0, 0, 0);
    if (i0 < z.tail_bytes) z.tail[i0] = 0;
    if (i0 == 0) *z.counter = 0;
}

static __global__ void zero_kernel(ZeroArgs z) {
    zero_range(z, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// A SIC's start on the device in one launch: positions packed from SoA to
// float4 records, four to a thread (n4, a multiple of four, in each of x, y,
// z), and the sums zeroed.  (Reading the positions from pinned host memory
// here, without the copy before it, was slower: uniform 64^3 driver sweep 3.80
// against 3.30 ms, clustered 96^3 11.4 against 10.1.)
static __global__ void unpack_kernel(const float4 *__restrict__ x, const float4 *__restrict__ y,
                                     const float4 *__restrict__ z, int64_t n4, float4 *pos,
                                     ZeroArgs zero) {
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = i0; i < n4 / 4; i += stride) {
        const float4 a = x[i], b = y[i], c = z[i];
        pos[4 * i] = make_float4(a.x, b.x, c.x, 0.f);
        pos[4 * i + 1] = make_float4(a.y, b.y, c.y, 0.f);
        pos[4 * i + 2] = make_float4(a.z, b.z, c.z, 0.f);
        pos[4 * i + 3] = make_float4(a.w, b.w, c.w, 0.f);
    }
    zero_range(zero, i0, stride);
}

nf_status mutual_unpack(nf_ctx *ctx, const Plan &pl, const float *xyz, int64_t n4, float4 *pos,
                        void *scratch, int *counter, cudaStream_t st) {
    const ZeroArgs zero = zero_args(ctx, pl, scratch, counter);
    const int64_t work = std::max<int64_t>(n4 / 4, (int64_t)zero.n16);
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((work + 255) / 256, ctx->sms * 4));
    unpack_kernel<<<blocks, 256, 0, st>>>((const float4 *)xyz, (const float4 *)(xyz + n4),
                                          (const float4 *)(xyz + 2 * n4), n4, pos, zero);
    NF_CUDA(cudaGetLastError());
    return NF_OK;
}

static MParams mutual_params(const nf_config &cfg, const MutualLaunch &L) {
    const Plan &pl = *L.plan;
    const int nc = cfg.b2 > 0.f ? 4 : 3;
    MParams kp;
    memset(&kp, 0, sizeof(kp));
    kp.pos = L.pos;
    kp.g = Geometry{L.cs, L.cpd, cfg.near_field_radius, pl.lo, pl.hi, pl.onesided};
    kp.items = pl.d_mutual;
    kp.n_items = pl.n_mutual;
    kp.counter = L.counter;
    kp.acc = (unsigned long long *)L.scratch;
    kp.bad = (unsigned char *)L.scratch + (size_t)pl.n_range * 8 * nc;
    kp.p0 = pl.p0;
    kp.n_range = pl.n_range;
    kp.fscale = (float)std::ldexp(1.0, pl.fbits);
    kp.wscale = (float)std::ldexp(1.0, pl.wbits);
    kp.pc = pair_const(cfg, L.eps, Step::SHORT);
    kp.near_w = near_width(cfg, L.eps, L.cpd);
    for (int a = 0; a < 2 * kp.g.R + 1; a++)
        kp.zshift[a] = kp.xyshift[a] = (float)((a - kp.g.R) * (1.0 / (double)L.cpd));
    return kp;
}

// Zero the sums (unless mutual_unpack has) and run the sweep of a plan.
nf_status mutual_launch(nf_ctx *ctx, const MutualLaunch &L, cudaStream_t st) {
    ctx->engine = NF_ENGINE_MUTUAL;
    const nf_config &cfg = ctx->cfg;
    const Plan &pl = *L.plan;
    if (!L.zeroed) {
        zero_kernel<<<ctx->sms * 4, 256, 0, st>>>(zero_args(ctx, pl, L.scratch, L.counter));
        NF_CUDA(cudaGetLastError());
    }
    if (L.before) NF_CUDA(cudaEventRecordWithFlags(L.before, st, L.event_flags));
    if (pl.n_mutual == 0) return NF_OK;
    MParams kp = mutual_params(cfg, L);
    MutualFn fn = pick(cfg.softening, cfg.b2 > 0.f, pl.variant);
    void *args[] = {&kp};
    NF_CUDA(cudaLaunchKernel((const void *)fn, dim3(pl.grid), dim3(WPC * 32), args,
                             smem_bytes(smax_of(cfg, pl.variant), cfg.b2 > 0.f), st));
    return NF_OK;
}

// First launch of an allocation-free call: the slab range's particle bounds and
// the box's particle count to bounds[0..2], and, where the range fits max_n,
// its sums and the counters zeroed.
static __global__ void noalloc_begin_kernel(const int64_t *__restrict__ cs, int64_t c_lo, int64_t c_hi,
                                            int64_t ncell, int64_t max_n, int bytes_per, uint4 *acc,
                                            int *counters, int64_t *bounds) {
    const int64_t p0 = cs[c_lo], p1 = cs[c_hi];
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 < 4) counters[i0] = 0;
    if (i0 == 0) {
        bounds[0] = p0;
        bounds[1] = p1;
        bounds[2] = cs[ncell];
    }
    if (p1 - p0 > max_n || p1 < p0) return;
    // whole 16-byte words: the scratch is larger than any range's sums
    const int64_t n16 = ((p1 - p0) * bytes_per + 15) / 16;
    for (int64_t i = i0; i < n16; i += (int64_t)gridDim.x * blockDim.x) acc[i] = make_uint4(0, 0, 0, 0);
}

nf_status mutual_noalloc_begin(int sms, const nf_config &cfg, int cpd, const int64_t *cs, int lo, int hi,
                               int64_t max_n, void *acc, int *counters, int64_t *bounds,
                               cudaStream_t st) {
    const int64_t c2 = (int64_t)cpd * cpd;
    noalloc_begin_kernel<<<sms, 256, 0, st>>>(cs, lo * c2, hi * c2, c2 * cpd, max_n,
                                              8 * (cfg.b2 > 0.f ? 4 : 3) + 1, (uint4 *)acc, counters, bounds);
    NF_CUDA(cudaGetLastError());
    return NF_OK;
}

// CTAs per SM of the allocation-free sweep, asked once per device and kernel.
static nf_status noalloc_grid(int dev, int sms, const nf_config &cfg, int *grid) {
    static std::atomic<int> per_sm[128][8];
    const bool dens = cfg.b2 > 0.f;
    std::atomic<int> &slot = per_sm[dev][2 * cfg.softening + dens];
    int n = slot.load();
    if (n == 0) {
        const void *fn = (const void *)noalloc_fn(cfg.softening, dens);
        NF_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(4, cfg.b2 > 0.f)));
        NF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, WPC * 32, smem_bytes(4, cfg.b2 > 0.f)));
        n = std::max(n, 1);
        slot.store(n);
    }
    *grid = sms * n;
    return NF_OK;
}

// The sweep of an allocation-free call (after mutual_noalloc_begin): pl holds
// the range; its units are set here.  *done stays false where the engine does
// not apply.
nf_status mutual_noalloc(int dev, int sms, const nf_config &cfg, const MutualLaunch &L, Plan &pl,
                         int64_t np_total, bool *done, cudaStream_t st) {
    *done = false;
    if (cfg.accumulation != NF_ACC_COMPENSATED || np_total > INT32_MAX / 8 ||
        !mutual_bits(cfg.softening, cfg.eps, cfg.b2, L.cpd, (double)np_total, &pl.fbits, &pl.wbits))
        return NF_OK;
    int grid = 0;
    nf_status s = noalloc_grid(dev, sms, cfg, &grid);
    if (s != NF_OK) return s;
    MParams kp = mutual_params(cfg, L);
    const int64_t c2 = (int64_t)L.cpd * L.cpd;
    int pencil0 = (int)(pl.lo * c2), n_pencils = (int)((pl.hi - pl.lo) * c2);
    // few pencils are cut into pieces, two a warp
    int pieces = (int)std::max<int64_t>(1, std::min<int64_t>(8, 2 * (int64_t)grid * WPC / n_pencils));
    if ((int64_t)n_pencils * pieces > INT32_MAX / 2) pieces = 1;
    void *args[] = {&kp, &pencil0, &n_pencils, &pieces};
    NF_CUDA(cudaLaunchKernel((const void *)noalloc_fn(cfg.softening, cfg.b2 > 0.f), dim3(grid),
                             dim3(WPC * 32), args, smem_bytes(4, cfg.b2 > 0.f), st));
    pl.mutual = true;
    *done = true;
    return NF_OK;
}

}  // namespace nf
