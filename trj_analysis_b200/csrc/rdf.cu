// rdf.cu -- species-resolved pair-distance histogram g_ab(r) on sm_100a.
//
// Restates the arithmetic of the reference kernel rdf_sh (src/modules/rdf.cuf:426-487):
// per unordered pair, FP32 minimum image xd -= L*nint(xd/L) per axis, rr2 = (xd^2+yd^2)+zd^2,
// counted when rr2 < side2 into bin nint(sqrt_rn(rr2)/deltar) if 1 <= bin <= lsmax, row
// ind_ij(species_i, species_j).  Every FP32 operation is the explicitly rounded intrinsic
// (__fsub_rn/__fmul_rn/__fadd_rn/__fsqrt_rn/__fdiv_rn), so no FMA contraction changes it.
//
// Unlike the reference's O(N^2) sweep, candidate pairs come from a linked-cell grid:
// cells of edge >= rcut*(1+2^-10), a half-shell stencil (13 neighbour cells + self) so each
// pair is tested once.  The per-pair arithmetic is sign-symmetric (IEEE subtraction, NINT
// half-away-from-zero), so the order (i,j) or (j,i) gives the same rr2 and the same bin;
// the counts equal the all-pairs sweep exactly.  Axes with fewer than 3 cells are not split
// (one cell along that axis); a frame with no split axis is the all-pairs case.
//
// Each cell is divided into boxes of about 28 atoms ("groups"), and the atoms are sorted by
// (cell, group).  A warp takes the up to 32 atoms of one group as homes, one per lane, and walks the
// groups of the neighbour cells: groups, then single atoms, farther from the homes' bounding box than
// the cutoff are skipped (conservatively: the counts are those of the full stencil), and the survivors
// are compacted into a buffer of the warp in shared memory, from which the exact pair test runs with
// every lane busy, two neighbours per packed FP32 instruction.
#include <curand_kernel.h>
#include <math.h>

#include <algorithm>

#include "batch.cuh"
#include "pairs.cuh"
#include "trj_common.cuh"

namespace {

constexpr int kGroup = 32;            // home atoms of a round, one per lane
constexpr double kGroupFill = 28.0;   // average atoms per group aimed at: few groups then exceed 32
constexpr int kRing = 128;            // surviving neighbours buffered per warp (arrays x, y, z, w)
constexpr int kRingRun = 64;          // survivors tested per run
constexpr int kMaxWarps = 32;         // per SM: 64 registers a thread (24 warps of 80 registers: 4 % slower at 1e6 atoms)

// A frame's words of work state (in a fused turn: an item's): work counter, frame flags, then one 64-bit sum of the
// atoms placed (low half) and the rounds of homes (high half).
enum { kWorkNext = 0, kWorkFlags = 1, kWorkAtoms = 2, kWorkRounds = 3, kWorkWords = 4 };

// Frame flags raised by cell_assign_kernel: how far coordinates reach outside [0, L).  They decide
// whether |d| < 3L/2 holds for every pair of the frame (see frame_within).
enum : unsigned { kFrameLow = 1u, kFrameVeryLow = 2u, kFrameHigh = 4u };

__device__ __forceinline__ int fast_div(int n, const FastDiv& f) {
    return f.d == 1u ? n : (int)(__umulhi((unsigned)n, f.mul) >> f.shift);
}

__device__ __forceinline__ float fast_sqrt(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float min_image_exact(float d, float L) {
    float n = roundf(__fdiv_rn(d, L));
    return __fsub_rn(d, __fmul_rn(L, n));
}

// Minimum image of the reference, d - L*nint(fl(d/L)), without the division below 3L/2: h1 (h2) is the
// least float x >= 0 whose quotient fl(x/L) is >= 1/2 (>= 3/2), found on the host with the same FP32
// division.  Correctly rounded division is monotonic in x, so |d| < h1 <=> nint = 0 and
// h1 <= |d| < h2 <=> nint = +-1 (sign of d): the result is the reference's, bit for bit.
__device__ __forceinline__ float min_image(float d, float L, float h1, float h2) {
    const float a = fabsf(d);
    if (a < h1) return d;
    if (a < h2) return __fsub_rn(d, __fmul_rn(L, copysignf(1.0f, d)));
    return min_image_exact(d, L);  // also NaN
}

// Bin of a pair by the reference's arithmetic (0: not counted).
__device__ __forceinline__ int outcome(float rr2, float side2, float deltar, int lsmax, int floor_bins) {
    if (!(rr2 < side2)) return 0;
    float rr = __fsqrt_rn(rr2);
    float q = __fdiv_rn(rr, deltar);
    int ind = floor_bins ? (int)floorf(q) + 1 : (int)roundf(q);
    return (ind <= lsmax && ind > 0) ? ind : 0;
}

__device__ __forceinline__ int wrapc(int c, int n) { return c < 0 ? c + n : (c >= n ? c - n : c); }

struct PairCounters {
    unsigned ulp = 0, fma = 0;
    u64 counted = 0;
};

// Exact reference outcome of a pair near a bin edge or the cutoff, with its edge statistics when wanted:
// returns the bin | 2^29 if a one-ulp change of rr2 changes it | 2^30 if the FMA-contracted rr2
// does.  Scalars by value: nothing of the caller's needs an address (no local-memory copies).
__device__ __noinline__ int exact_bin(float rr2, float x2, float dy, float dz, float side2, float deltar, int lsmax,
                                      int floor_bins, int want_edge = 1) {
    const int ind = outcome(rr2, side2, deltar, lsmax, floor_bins);
    if (!want_edge) return ind;
    const int olo = outcome(nextafterf(rr2, -INFINITY), side2, deltar, lsmax, floor_bins);
    const int ohi = outcome(nextafterf(rr2, INFINITY), side2, deltar, lsmax, floor_bins);
    const float rr2f = fmaf(dz, dz, fmaf(dy, dy, x2));
    const int fma = outcome(rr2f, side2, deltar, lsmax, floor_bins) != ind;
    return ind | ((olo != ind || ohi != ind) ? (1 << 29) : 0) | (fma ? (1 << 30) : 0);
}

// How the minimum image of a pair is formed.  All forms give the reference's d - L*nint(fl(d/L)) for
// every pair that can be in range, up to its sign, which drops out in the squares.
//   kImgNone   d: both cells hold only coordinates in [0, L), every axis is split (>= 3 cells of edge >=
//              cutoff) and the task does not wrap: a pair with another image is beyond the cutoff in
//              either one (its |d| here is >= L/2 >= 1.5 cutoffs, its true image >= one cell edge).
//   kImgShift  the same on tasks that wrap: nint = -+1 on the wrapped axes, d + img with img = +-L or 0
//              (adding 0 leaves d as it is).
//   kImgRound  d - L*n with n = d/L rounded by the 1.5*2^23 trick: every axis split, coordinates in [-L, L)
//              (|n| <= 2, so L*n is exact).  A pair in range has |d - L*n| <= L/3, far from where the
//              approximate quotient could round to another integer; a pair near there is >= L/2 away.
//   kImgFold   min(|d|, ||d| - L|) per axis, for frames in which |d| < 3L/2 (frame_within): below L/2 it
//              is |d| (the rounded L - |d| is >= L/2), from L/2 on |d| - L is exact (Sterbenz) and the
//              smaller one; h1 is L/2 itself, so this is the reference's choice, ties included.
//   kImgAny    the thresholds h1, h2 and the division beyond them.
enum { kImgNone = 0, kImgShift = 1, kImgRound = 2, kImgFold = 3, kImgAny = 4 };

// Constants of one axis: img (kImgShift), or 1/L (kImgRound).
template <int MODE>
__device__ __forceinline__ float image_1(float b, float na, float cst, float L, float h1, float h2) {
    const float d = __fadd_rn(b, na);
    if (MODE == kImgShift) return __fadd_rn(d, cst);
    if (MODE == kImgRound) return __fmaf_rn(__fsub_rn(__fmaf_rn(d, cst, 12582912.0f), 12582912.0f), -L, d);
    if (MODE == kImgFold) {
        const float a = fabsf(d);
        return fminf(a, fabsf(__fsub_rn(a, L)));
    }
    if (MODE == kImgAny) return min_image(d, L, h1, h2);
    return d;
}

template <int MODE>
__device__ __forceinline__ u64 image_2(u64 b, u64 na, u64 cst, float L, float h1, float h2) {
    u64 d = add2(b, na);
    if (MODE == kImgShift) return add2(d, cst);
    if (MODE == kImgRound) {
        const u64 magic = pack2(12582912.0f, 12582912.0f), nmagic = pack2(-12582912.0f, -12582912.0f);
        return fma2(add2(fma2(d, cst, magic), nmagic), pack2(-L, -L), d);
    }
    if (MODE == kImgFold || MODE == kImgAny) {
        float lo, hi;
        unpack2(d, lo, hi);
        if (MODE == kImgFold) {
            lo = fabsf(lo);
            hi = fabsf(hi);
            lo = fminf(lo, fabsf(__fsub_rn(lo, L)));
            hi = fminf(hi, fabsf(__fsub_rn(hi, L)));
        } else {
            lo = min_image(lo, L, h1, h2);
            hi = min_image(hi, L, h1, h2);
        }
        d = pack2(lo, hi);
    }
    return d;
}

__device__ __forceinline__ float max3_abs(float a, float b, float c) { return fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c)); }

// Low bits of 1.5*2^23: an FP32 sum of it and q < 2^22 holds kBinBias + nint(q) as an integer.
constexpr unsigned kBinBias = 0x4B400000u;

// A lane's home atom against the survivors in its warp's buffer.
struct Home {
    float nx, ny, nz;   // negated coordinates
    unsigned hist;      // square layout: shared-memory address of its species' first row of bins, minus 4 *
                        // kBinBias; triangular layout: address of its species' entry in the row table
    float q;            // charge
};

// What a warp keeps between the culling and the tests, in shared memory so that neither loop holds the other's
// registers.
struct WarpState {
    float4 home[kGroup];        // negated coordinates, Home::hist (bits) of every lane
    int gs[32], gn[32];         // start and atoms of the neighbour groups of the current 32
    float home_q[kGroup];
    float4 box, half;           // the group's box: centre and half-widths
    float4 cut;                 // its centre less the neighbour cell's image
    float4 img;
    int4 walk;                  // j, je, m, e0 of the neighbour walk
    int4 outer;                 // position in the neighbour list, cell of the homes and its flags, first home
    int nh;
    unsigned since;             // clock when the CTA's rows were last merged
};

constexpr size_t kWarpBytes = 16 * kRing + (sizeof(WarpState) + 15) / 16 * 16;  // buffer and state of a warp

// Tests `n4` blocks of four survivors from ring position `head` (SELF: the round's own atoms in lane order
// from position 0, pairs j > i).  w of a survivor: bytes to add to Home::hist (square layout: species * row
// bytes; triangular layout: species * 64, a row of the 16 x 16 table).
//
// Per survivor and home: the reference's rr2 with every operation rounded once (two survivors per packed
// instruction), then the bin from an approximate root.  q = r/deltar is off by less than 0.32 q 2^-20
// (sqrt.approx 2^-23, 1/deltar 2^-24, the reference's own root and quotient 2^-24 each), and less than
// 0.47 q 2^-20 after a change of rr2 by one ulp (2^-24) or to its FMA-contracted value (1.25*2^-23); so a
// pair whose q is farther than edge_thr allows from any bin edge has the reference's bin, and no edge
// statistic.  rr2 < side2 is exact.  FLOOR: floor(q) + 1 = the integer nearest to q + 1/2, whose sum is rounded
// once more (2^-24: 0.38 and 0.53 in all).
// Every pair in range is counted at once in its approximate bin; a block in which some test lies in the
// window of an edge (or, with EDGE, within 2^-20 of the cutoff, where one-ulp changes decide) is looked at
// again and the few wrong counts are moved.  QMODE instead leaves those out of the first count, since a
// charge product cannot be taken back exactly.
template <int MODE, bool SELF, bool FLOOR, bool QMODE, bool SQUARE, bool EDGE, int UNROLL>
__device__ __forceinline__ void test_run(const float* __restrict__ ring, const double* __restrict__ ring_q, int head,
                                         int n4, const WarpState* __restrict__ ws, const PairGeom& g,
                                         PairCounters& pc, double* myq) {
    const int lane = (int)(threadIdx.x & 31u);
    Home h;
    {
        const float4 a = ws->home[lane];
        h.nx = a.x;
        h.ny = a.y;
        h.nz = a.z;
        h.hist = __float_as_uint(a.w);
        if (QMODE) h.q = ws->home_q[lane];
    }
    const bool has = lane < ws->nh;
    float cx = 0.f, cy = 0.f, cz = 0.f;
    if (MODE == kImgShift) {
        const float4 v = ws->img;
        cx = v.x;
        cy = v.y;
        cz = v.z;
    } else if (MODE == kImgRound) {
        cx = g.inv_L[0];
        cy = g.inv_L[1];
        cz = g.inv_L[2];
    }
    const u64 nx = pack2(h.nx, h.nx), ny = pack2(h.ny, h.ny), nz = pack2(h.nz, h.nz);
    const u64 jx = pack2(cx, cx), jy = pack2(cy, cy), jz = pack2(cz, cz);
    const u64 inv = pack2(g.inv_deltar, g.inv_deltar);
    const u64 magic = pack2(12582912.0f, 12582912.0f);  // 1.5*2^23: its sum with q holds nint(q) in the low bits
    const u64 one = pack2(g.one, g.one);
    const u64 neg1 = pack2(-1.0f, -1.0f), half = pack2(0.5f, 0.5f);
    const float thr = g.edge_thr;
    const float lo = has ? (QMODE ? g.side2_lo : g.side2) : 0.0f, hi = has ? g.side2_hi : 0.0f;
#pragma unroll UNROLL
    for (int k = 0; k < n4; ++k) {
        const int e = (head + 4 * k) & (kRing - 1);
        const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(ring + e);
        const ulonglong2 Y = *reinterpret_cast<const ulonglong2*>(ring + kRing + e);
        const ulonglong2 Z = *reinterpret_cast<const ulonglong2*>(ring + 2 * kRing + e);
        const uint4 W = *reinterpret_cast<const uint4*>(ring + 3 * kRing + e);
        float r[4];
        unsigned bits[4];
        float d[4];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const u64 dx = image_2<MODE>(p ? X.y : X.x, nx, jx, g.L[0], g.h1[0], g.h2[0]);
            const u64 dy = image_2<MODE>(p ? Y.y : Y.x, ny, jy, g.L[1], g.h1[1], g.h2[1]);
            const u64 dz = image_2<MODE>(p ? Z.y : Z.x, nz, jz, g.L[2], g.h1[2], g.h2[2]);
            // the two sums as a*1 + b: the assembler contracts a packed product and sum into an fma
            const u64 rr = fma2(fma2(mul2(dx, dx), one, mul2(dy, dy)), one, mul2(dz, dz));
            unpack2(rr, r[2 * p], r[2 * p + 1]);
            const u64 s = pack2(fast_sqrt(r[2 * p]), fast_sqrt(r[2 * p + 1]));
            u64 t, dd;
            if (FLOOR) {
                const u64 q = fma2(s, inv, half);
                t = add2(q, magic);
                dd = add2(q, fma2(t, neg1, magic));
            } else {
                t = fma2(s, inv, magic);
                dd = fma2(s, inv, fma2(t, neg1, magic));
            }
            unpack2(dd, d[2 * p], d[2 * p + 1]);
            bits[2 * p] = (unsigned)t;
            bits[2 * p + 1] = (unsigned)(t >> 32);
        }
        const unsigned w[4] = {W.x, W.y, W.z, W.w};
        auto row_of = [&](unsigned wt) {
            unsigned row = h.hist + wt;
            if (!SQUARE) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(row) : "r"(row));
            return row;
        };
        bool again;
        if constexpr (QMODE) {
            again = false;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const bool in = (!SELF || 4 * k + t > lane) && r[t] < hi;
                const bool fast = in && r[t] < lo && fabsf(d[t]) <= thr;
                if (fast) {
                    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(row_of(w[t]) + (bits[t] << 2)) : "memory");
                    atomicAdd(&myq[bits[t] - kBinBias], (double)h.q * ring_q[e + t]);
                }
                again = again || (in && !fast);
            }
        } else {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                // predicated, not branched over: a branch per test costs more than the idle lanes
                const float top = (SELF && 4 * k + t <= lane) ? 0.0f : lo;
                asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %0, %1;\n\t@p red.shared.add.u32 [%2], 1;\n\t}" ::"f"(r[t]),
                             "f"(top), "r"(row_of(w[t]) + (bits[t] << 2))
                             : "memory");
            }
            again = fmaxf(max3_abs(d[0], d[1], d[2]), fabsf(d[3])) > thr;
            if (EDGE) {
                const u64 m = pack2(-g.side2, -g.side2);
                float z[4];
                unpack2(add2(pack2(r[0], r[1]), m), z[0], z[1]);
                unpack2(add2(pack2(r[2], r[3]), m), z[2], z[3]);
                const float zm = fminf(fminf(fabsf(z[0]), fabsf(z[1])), fminf(fabsf(z[2]), fabsf(z[3])));
                again = again || zm <= g.side2_win;
            }
        }
        if (again) {
            const float lo2 = (EDGE || QMODE) ? g.side2_lo : INFINITY;
            unsigned which = 0;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if ((!SELF || 4 * k + t > lane) && r[t] < (EDGE || QMODE ? hi : lo) && (fabsf(d[t]) > thr || r[t] >= lo2))
                    which |= 1u << t;
#pragma unroll 1
            while (which) {
                const int t = __ffs(which) - 1;
                which &= which - 1u;
                const float rr2 = t < 2 ? (t == 0 ? r[0] : r[1]) : (t == 2 ? r[2] : r[3]);
                const unsigned was = (t < 2 ? (t == 0 ? bits[0] : bits[1]) : (t == 2 ? bits[2] : bits[3]));
                float x2 = 0.f, dy = 0.f, dz = 0.f;
                if (EDGE || QMODE) {  // the statistics look at the FMA-contracted rr2 as well
                    const float dx = image_1<MODE>(ring[e + t], h.nx, cx, g.L[0], g.h1[0], g.h2[0]);
                    dy = image_1<MODE>(ring[kRing + e + t], h.ny, cy, g.L[1], g.h1[1], g.h2[1]);
                    dz = image_1<MODE>(ring[2 * kRing + e + t], h.nz, cz, g.L[2], g.h1[2], g.h2[2]);
                    x2 = __fmul_rn(dx, dx);
                }
                const int x = exact_bin(rr2, x2, dy, dz, g.side2, g.deltar, g.lsmax, g.floor_bins,
                                        (EDGE || QMODE) && g.want_edge);
                pc.ulp += (x >> 29) & 1;
                pc.fma += (x >> 30) & 1;
                const unsigned ind = (x & ((1 << 29) - 1)) + kBinBias;
                const unsigned row = row_of(__float_as_uint(ring[3 * kRing + e + t]));
                if (QMODE) {
                    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(row + (ind << 2)) : "memory");
                    atomicAdd(&myq[ind - kBinBias], (double)h.q * ring_q[e + t]);
                } else if (rr2 < g.side2 && ind != was) {
                    asm volatile("red.shared.add.u32 [%0], 0xffffffff;" ::"r"(row + (was << 2)) : "memory");
                    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(row + (ind << 2)) : "memory");
                }
            }
        }
    }
}

// Wrapped coordinate of a folded one in [-L, L): x, or x + L for x < 0 (the same FP32 value the cell
// assignment computes, so the atom lies in its cell's range).  The fold of select_ncdfinput keeps
// negative coordinates negative; the cull works on the wrapped values.
__device__ __forceinline__ float wrap_cull(float x, float L) { return x < 0.f ? __fadd_rn(x, L) : x; }

// Distance along one axis from a point (or box centre) to the homes' box, clipped at 0.  PERIODIC: of the
// nearest image.
template <bool PERIODIC>
__device__ __forceinline__ float axis_gap(float b, float c, float h, float L) {
    float t = fabsf(b - c);
    if (PERIODIC) t = fminf(t, L - t);
    return fmaxf(t - h, 0.f);
}

// A group's bounding box along one axis from the lanes' least and largest wrapped coordinates (in [0, L]: their
// bit patterns order like the values).
__device__ __forceinline__ void axis_box(unsigned lo, unsigned hi, float pad, float& c, float& h) {
    const float mn = __uint_as_float(__reduce_min_sync(0xffffffffu, lo));
    const float mx = __uint_as_float(__reduce_max_sync(0xffffffffu, hi));
    c = 0.5f * (mn + mx);
    h = 0.5f * (mx - mn) + pad;
}

// |d| < 3L/2 for every pair of the frame: no coordinate below -0.499 L, or none below -0.749 L while none
// reaches 0.749 L (frames centred on the origin).  (Coordinates outside [-L, L) are flagged per cell.)
__device__ __forceinline__ bool frame_within(unsigned f) {
    return !(f & kFrameLow) || !(f & (kFrameVeryLow | kFrameHigh));
}

// One work item of a frame: round item / nseg (up to 32 atoms of one group, see emit_rounds) against segment
// item % nseg of its group's neighbour list.  hist: shared-memory address of the bin rows (SQUARE), rowtab: of the
// row table (otherwise).
template <bool FLOOR, bool QMODE, bool SQUARE, bool EDGE, int UNROLL>
__device__ __forceinline__ void pair_item(const RdfParams& p, int item, const int4* __restrict__ rounds,
                                          const float4* __restrict__ sorted,
                                          const int32_t* __restrict__ fstart, const int32_t* __restrict__ fcount,
                                          const int32_t* __restrict__ cflag, bool frame_ok,
                                          const float* __restrict__ sorted_q, float* ring, double* ring_q,
                                          WarpState* ws, unsigned hist_base, unsigned rowtab, double* qhist,
                                          PairCounters& pc, u64& n_tested) {
    const PairGeom& g = p.g;
    const int lane = (int)(threadIdx.x & 31u);
    const unsigned lt = (1u << lane) - 1u;
    const int round = fast_div(item, p.div_nseg), seg = item - round * p.nseg;
    // one 16-byte load wants four neighbouring registers, which the uncharged loops do not have (2.54 ms at 1e6 atoms
    // against 2.47); the charged ones gain from it (255,000 ions, cutoff 3.5: 394 -> 390 us)
    int4 rd;
    if constexpr (QMODE) {
        rd = rounds[round];
    } else {
        const int2* r2 = reinterpret_cast<const int2*>(rounds + round);
        const int2 lo = r2[0], hi = r2[1];
        rd = make_int4(lo.x, lo.y, hi.x, hi.y);
    }
    const int key = rd.x, h0 = rd.y, hbeg = rd.z, hend = rd.w;
    const int c = fast_div(key, p.div_nsub), own = key - c * p.nsub;
    const int cxy = fast_div(c, p.div_nc2), cz = c - cxy * p.nc[2];
    const int cx = fast_div(cxy, p.div_nc1), cy = cxy - cx * p.nc[1];
    const int fl = cflag[c];
    const int t0 = seg * p.per_seg, t1 = min(p.list, t0 + p.per_seg);
    // The group's box: centre and half-widths (of all its atoms, so that the pairs tested do not depend on their
    // order; + 0 turns -0 into +0).
    {
        unsigned lo[3] = {0x7f800000u, 0x7f800000u, 0x7f800000u}, hi[3] = {0u, 0u, 0u};
        for (int i = hbeg + lane; i < hend; i += kGroup) {
            const float4 a = sorted[i];
            const unsigned v[3] = {__float_as_uint(wrap_cull(a.x, g.L[0]) + 0.0f),
                                   __float_as_uint(wrap_cull(a.y, g.L[1]) + 0.0f),
                                   __float_as_uint(wrap_cull(a.z, g.L[2]) + 0.0f)};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                lo[d] = min(lo[d], v[d]);
                hi[d] = max(hi[d], v[d]);
            }
        }
        float4 c, w;
        c.w = w.w = 0.f;
        axis_box(lo[0], hi[0], p.cull_pad, c.x, w.x);
        axis_box(lo[1], hi[1], p.cull_pad, c.y, w.y);
        axis_box(lo[2], hi[2], p.cull_pad, c.z, w.z);
        if (lane == 0) {
            ws->box = c;
            ws->half = w;
        }
    }
    {
        const int nh = min(kGroup, hend - h0);
        const bool has = lane < nh;
        float4 a = has ? sorted[h0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        const unsigned wa = __float_as_uint(a.w);  // species * row bytes (64 with the row table)
        a.x = -a.x;
        a.y = -a.y;
        a.z = -a.z;
        a.w = __uint_as_float(SQUARE ? hist_base + wa * (unsigned)g.nsp - 4u * kBinBias : rowtab + (wa >> 4));
        ws->home[lane] = a;
        if (QMODE) ws->home_q[lane] = has ? sorted_q[h0 + lane] : 0.f;
        if (lane == 0) ws->nh = nh;
    }
    for (int t = t0; t < t1;) {
        // entries [e_lo, e_hi) of offset o: group e, or (own cell) the e-th after the homes' own
        const int o = t < p.nself ? 0 : 1 + fast_div(t - p.nself, p.div_nsub);
        const int first = o == 0 ? 0 : p.nself + (o - 1) * p.nsub;
        const int e_lo = t - first, e_hi = min(o == 0 ? p.nself : p.nsub, t1 - first);
        const int ex = cx + p.off[o][0], ey = cy + p.off[o][1], ez = cz + p.off[o][2];
        const int c2 = (wrapc(ex, p.nc[0]) * p.nc[1] + wrapc(ey, p.nc[1])) * p.nc[2] + wrapc(ez, p.nc[2]);
        const int f2 = fl | cflag[c2];
        const bool far = f2 & 2;
        const bool plain = p.split_all && !(f2 & 1);  // image known from the cells
        int mode;
        {
            const float4 img = make_float4(ex < 0 ? -g.L[0] : (ex >= p.nc[0] ? g.L[0] : 0.f),
                                           ey < 0 ? -g.L[1] : (ey >= p.nc[1] ? g.L[1] : 0.f),
                                           ez < 0 ? -g.L[2] : (ez >= p.nc[2] ? g.L[2] : 0.f), 0.f);
            mode = plain ? ((img.x != 0.f || img.y != 0.f || img.z != 0.f) ? kImgShift : kImgNone)
                         : far ? kImgAny : p.split_all ? kImgRound : frame_ok ? kImgFold : kImgAny;
            __syncwarp();  // the group's box, homes and the last offset's readers
            if (lane == 0) {
                const float4 c = ws->box;
                ws->img = img;
                ws->cut = plain ? make_float4(c.x - img.x, c.y - img.y, c.z - img.z, 0.f) : c;
                ws->outer = make_int4(first + e_hi, c2 * p.nsub, own, h0);
            }
            __syncwarp();
        }
        int head = 0, tail = 0;
        auto append = [&](float x, float y, float z, float w, float qb, bool keep) {
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const int e = (tail + __popc(m & lt)) & (kRing - 1);
                ring[e] = x;
                ring[kRing + e] = y;
                ring[2 * kRing + e] = z;
                ring[3 * kRing + e] = w;
                if (QMODE) ring_q[e] = (double)qb;
            }
            tail += __popc(m);
        };
        // Fills the buffer up to a multiple of four with NaN entries (in no range, near no edge).
        auto pad = [&]() {
            const int n = tail - head, up = (n + 3) & ~3;
            if (lane < up - n) {
                const int e = (tail + lane) & (kRing - 1);
                ring[e] = ring[kRing + e] = ring[2 * kRing + e] = NAN;
                ring[3 * kRing + e] = 0.f;
                if (QMODE) ring_q[e] = 0.0;
            }
            return up >> 2;
        };
#define TRJ_RUN(M, S, N4) test_run<M, S, FLOOR, QMODE, SQUARE, EDGE, UNROLL>(ring, ring_q, head, N4, ws, g, pc, qhist)
        if (o == 0 && e_lo == 0) {
            // pairs j > i of the round's own atoms, through the buffer in lane order
            const int nh = ws->nh;
            const float4 a = lane < nh ? sorted[h0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
            append(a.x, a.y, a.z, a.w, QMODE ? ws->home_q[lane] : 0.f, lane < nh);
            const int n4 = pad();
            __syncwarp();
            if (plain) TRJ_RUN(kImgNone, true, n4);
            else if (mode == kImgRound) TRJ_RUN(kImgRound, true, n4);
            else if (mode == kImgFold) TRJ_RUN(kImgFold, true, n4);
            else TRJ_RUN(kImgAny, true, n4);
            __syncwarp();
            if (EDGE && lane < nh) n_tested += (unsigned)(nh - 1 - lane);
            tail = 0;
        }
        int e0 = e_lo - 32, j = 0, je = 0;
        unsigned m = 0;
        bool more = true;
        do {
            // survivors into the buffer until a run is full or the segment's groups are used up
            while (tail - head < kRingRun) {
                if (j >= je) {
                    if (!m) {
                        e0 += 32;
                        if (e0 >= e_hi) {
                            more = false;
                            break;
                        }
                        // lanes over the neighbour groups: which can hold an atom in range of the homes' box
                        const int4 out = ws->outer;
                        const int e = e0 + lane;
                        int s = o == 0 ? out.z + e : e;
                        if (s >= p.nsub) s -= p.nsub;
                        // half-way round an even number of groups each pair is met twice: the lower has it
                        bool near = e < e_hi && (o > 0 || 2 * e != p.nsub || 2 * out.z < p.nsub);
                        if (near && !far) {
                            const float4 b = ws->box, w = ws->half, img = ws->img;
                            const int q = (int)(((float)s + 0.5f) * p.inv_sub[2]), sz = s - q * p.sub[2];
                            const int sx = (int)(((float)q + 0.5f) * p.inv_sub[1]), sy = q - sx * p.sub[1];
                            const float gx = ((float)ex + ((float)sx + 0.5f) * p.inv_sub[0]) * p.edge[0];
                            const float gy = ((float)ey + ((float)sy + 0.5f) * p.inv_sub[1]) * p.edge[1];
                            const float gz = ((float)ez + ((float)sz + 0.5f) * p.inv_sub[2]) * p.edge[2];
                            float dx, dy, dz;
                            if (p.split_all) {
                                dx = axis_gap<false>(gx, b.x, w.x + p.half[0], 0.f);
                                dy = axis_gap<false>(gy, b.y, w.y + p.half[1], 0.f);
                                dz = axis_gap<false>(gz, b.z, w.z + p.half[2], 0.f);
                            } else {
                                dx = axis_gap<true>(gx - img.x, b.x, w.x + p.half[0], g.L[0]);
                                dy = axis_gap<true>(gy - img.y, b.y, w.y + p.half[1], g.L[1]);
                                dz = axis_gap<true>(gz - img.z, b.z, w.z + p.half[2], g.L[2]);
                            }
                            near = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= p.cull2;
                        }
                        m = __ballot_sync(0xffffffffu, near);
                        __syncwarp();  // the readers of the last 32 groups' starts (a ballot orders no memory)
                        if (near) {
                            ws->gs[lane] = fstart[out.y + s];
                            ws->gn[lane] = fcount[out.y + s];
                        }
                        __syncwarp();
                        continue;
                    }
                    const int k = __ffs(m) - 1;
                    m &= m - 1u;
                    j = ws->gs[k];
                    je = j + ws->gn[k];
                    if (o == 0 && e0 + k == 0) j = ws->outer.w + ws->nh;  // the round's own atoms are done
                    continue;
                }
                bool keep = j + lane < je;
                const float4 b = keep ? sorted[j + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
                const float qb = (QMODE && keep) ? sorted_q[j + lane] : 0.f;
                j += 32;
                if (keep && !far) {
                    const float4 c = ws->cut, w = ws->half;
                    float dx, dy, dz;
                    if (plain) {
                        dx = axis_gap<false>(b.x, c.x, w.x, 0.f);
                        dy = axis_gap<false>(b.y, c.y, w.y, 0.f);
                        dz = axis_gap<false>(b.z, c.z, w.z, 0.f);
                    } else {
                        dx = axis_gap<true>(wrap_cull(b.x, g.L[0]), c.x, w.x, g.L[0]);
                        dy = axis_gap<true>(wrap_cull(b.y, g.L[1]), c.y, w.y, g.L[1]);
                        dz = axis_gap<true>(wrap_cull(b.z, g.L[2]), c.z, w.z, g.L[2]);
                    }
                    keep = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= p.cull2;
                }
                const int before = tail;
                append(b.x, b.y, b.z, b.w, qb, keep);
                if (EDGE && lane < ws->nh) n_tested += (unsigned)(tail - before);
            }
            const int n4 = tail - head >= kRingRun ? kRingRun / 4 : pad();
            if (lane == 0) ws->walk = make_int4(j, je, (int)m, e0);
            __syncwarp();  // the other lanes' entries
            if (mode == kImgNone) TRJ_RUN(kImgNone, false, n4);
            else if (mode == kImgShift) TRJ_RUN(kImgShift, false, n4);
            else if (mode == kImgRound) TRJ_RUN(kImgRound, false, n4);
            else if (mode == kImgFold) TRJ_RUN(kImgFold, false, n4);
            else TRJ_RUN(kImgAny, false, n4);
            const int4 walk = ws->walk;
            __syncwarp();  // before the buffer and the state are written again
            j = walk.x;
            je = walk.y;
            m = (unsigned)walk.z;
            e0 = walk.w;
            head += 4 * n4;
        } while (more);
#undef TRJ_RUN
        t = ws->outer.x;
        __syncwarp();
    }
}

// The CTA's rows into the frame's uint64 histogram (their total is the counted pairs); they are cleared.
template <bool SQUARE>
__device__ __forceinline__ void merge_rows(const RdfParams& p, unsigned* hist, u64* __restrict__ hist_g,
                                           PairCounters& pc) {
    const int nsp = p.g.nsp, rw = p.g.row_words, lsmax = p.g.lsmax, hsz = p.nit * lsmax;
    auto take = [&](int row, int bin) {
        const u64 c = hist[row * rw + bin];
        hist[row * rw + bin] = 0u;
        return c;
    };
    int row = 0, sa = 0, sb = 0;  // species of the row of element k
#pragma unroll 1
    for (int k = threadIdx.x; k < hsz; k += blockDim.x) {
        while (row < k / lsmax) {
            ++row;
            if (++sb == nsp) sb = ++sa;
        }
        const int bin = k - row * lsmax + 1;
        u64 s;
        if (SQUARE) {
            s = take(sa * nsp + sb, bin);
            if (sa != sb) s += take(sb * nsp + sa, bin);
        } else {
            s = take(row, bin);
        }
        if (s) atomicAdd(&hist_g[k], s);
        pc.counted += s;
    }
}

__device__ __forceinline__ void add_edges(u64* __restrict__ edge_g, const PairCounters& pc, u64 n_tested) {
    u64 n_ulp = pc.ulp, n_fma = pc.fma, n_counted = pc.counted;
    for (int off = 16; off > 0; off >>= 1) {
        n_ulp += __shfl_down_sync(0xffffffffu, n_ulp, off);
        n_fma += __shfl_down_sync(0xffffffffu, n_fma, off);
        n_counted += __shfl_down_sync(0xffffffffu, n_counted, off);
        n_tested += __shfl_down_sync(0xffffffffu, n_tested, off);
    }
    if ((threadIdx.x & 31) == 0) {
        if (n_ulp) atomicAdd(&edge_g[TRJ_EDGE_ULP], n_ulp);
        if (n_fma) atomicAdd(&edge_g[TRJ_EDGE_FMA], n_fma);
        if (n_counted) atomicAdd(&edge_g[TRJ_EDGE_COUNTED], n_counted);
        if (n_tested) atomicAdd(&edge_g[TRJ_EDGE_TESTED], n_tested);
    }
}

// Rows hold 32 bits per bin.  2^26 clocks (35 ms) after its CTA last merged its rows a warp takes no further item, and
// once the CTA's other warps have come to that point (or to the end) the rows are merged and cleared.  An SM tests
// about eight pairs per clock, so that a bin stays below 2^32 as long as no item meets 1e7 atoms at one distance (eight
// warps per CTA; 3e6 with the 32 of CTAs that share a histogram of many bins).  Without it a CTA of a frame of 1e7
// atoms puts 4e9 pairs into a coarse bin at half the box.  It costs 1 % without and nothing with edge statistics (2.45
// -> 2.475 and 2.88 -> 2.875 ms at 1e6 atoms); the test loop's registers are tight: counting the tests instead, or
// merging by single warps, 2.55 and 3.04 to 3.19.
constexpr unsigned kMergeClocks = 1u << 26;

// The next work item, for a whole warp; past every item also when the rows are due to be merged.
__device__ __forceinline__ unsigned next_item(unsigned* next, const WarpState* ws) {
    unsigned item = 0xffffffffu;
    if ((threadIdx.x & 31u) == 0u && (unsigned)clock() - ws->since < kMergeClocks) item = atomicAdd(next, 1u);
    return __shfl_sync(0xffffffffu, item, 0);
}

// Work item = (round of homes, segment of their group's neighbour list), taken from a global counter by one warp at
// a time; no warp waits for another until the rows are merged.  Shared memory: bin rows (count), charge rows (QMODE, FP64 [row_words]),
// the warps' buffers.  SQUARE: a bin row per ordered species pair, so that a pair's row address is a sum of
// two registers; otherwise the rows of ind_ij through a 16 x 16 table of addresses.
//
// What bounds it: instruction issue, not the 22 MB it moves.  At 1e6 atoms (3 species, 0.86e9 pairs in range)
// 1.75e9 pairs are tested, in 17.6e6 blocks of four survivors x 32 homes of about 75 instructions each (packed
// FP32 alone takes 63 of the 80 issue slots of such a block), and 4.6e6 neighbour groups read and culled,
// together a quarter of the time.  With the culling's variables in registers across the tests 64 registers do
// not hold both (100 bytes spilled in the inner loop, 97 instructions a block): 2.95 ms at 1e6 atoms, 0.437 ms
// at 62,500 (cutoff 10, four cells per axis), 6.08 ms for the 4e6-atom slab, 1.83 ms for 256,000 ions; with
// them in WarpState and two blocks per turn of the loop 2.64, 0.394, 5.50 and 1.63 ms, with rounds for items
// 2.54, 0.370, 5.45 and 1.53 (layout and sort included).  (The ions' loop keeps one block per turn: two take
// 1.97 ms.)  64-atom homes, two per lane, that a CTA walks over staged neighbour cells with a branch per pair:
// 7.37, 1.69, 19.5 and 3.75 ms.
template <bool FLOOR, bool QMODE, bool SQUARE, bool EDGE>
__global__ void __launch_bounds__(kMaxWarps * 32, 1)
    rdf_pairs_kernel(const __grid_constant__ RdfParams p, const float4* __restrict__ sorted,
                     const int32_t* __restrict__ fstart, const int32_t* __restrict__ fcount,
                     const int32_t* __restrict__ cflag, const int4* __restrict__ rounds, unsigned* __restrict__ work,
                     u64* __restrict__ hist_g, u64* __restrict__ edge_g, unsigned* __restrict__ status,
                     const float* __restrict__ sorted_q, double* __restrict__ gqq_frame) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t never;  // no thread arrives on it: the target of the stall test
    __shared__ unsigned rowtab[SQUARE ? 1 : 256];
    __shared__ int stalled;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarp = blockDim.x >> 5;
    const PairGeom& g = p.g;
    const int nsp = g.nsp, rw = g.row_words;
    const int nrow = SQUARE ? nsp * nsp : p.nit;
    // [warps' buffers and states][QMODE: warps' charge buffers, FP64 rows][count rows]
    float* ring = reinterpret_cast<float*>(smem + (size_t)warp * kWarpBytes);
    WarpState* ws = reinterpret_cast<WarpState*>(smem + (size_t)warp * kWarpBytes + 16 * kRing);
    double* ring_q = reinterpret_cast<double*>(smem + (size_t)nwarp * kWarpBytes) + (QMODE ? warp * kRing : 0);
    double* qhist = reinterpret_cast<double*>(smem + (size_t)nwarp * kWarpBytes) + (QMODE ? nwarp * kRing : 0);
    unsigned* hist = reinterpret_cast<unsigned*>(qhist + (QMODE ? rw : 0));
    for (int k = tid; k < nrow * rw; k += blockDim.x) hist[k] = 0u;
    if (QMODE)
        for (int k = tid; k < rw; k += blockDim.x) qhist[k] = 0.0;
    const unsigned hist_base = trj_smem_addr(hist);
    if (!SQUARE)
        for (int k = tid; k < nsp * nsp; k += blockDim.x)
            rowtab[(k / nsp) * 16 + k % nsp] =
                hist_base + (unsigned)(trj_pair_row(k / nsp, k % nsp, nsp) * rw * 4) - 4u * kBinBias;
    if (lane == 0) ws->since = (unsigned)clock();
    if (tid == 0) {
        trj_mbar_init(&never, 1);
        trj_fence_mbar_init();
        stalled = 0;
    }
    __syncthreads();
    if (p.stall_test && !trj_mbar_wait_limit(&never, 0u, p.wait_clocks)) {
        if (lane == 0) trj_raise(status, TRJ_DEV_TIMEOUT);
        stalled = 1;
    }
    __syncthreads();
    if (stalled) return;

    const bool frame_ok = frame_within(work[kWorkFlags]);
    const unsigned nitems = work[kWorkRounds] * (unsigned)p.nseg;
#pragma unroll 1
    for (bool more = true; more;) {
        PairCounters pc;
        u64 n_tested = 0;
        for (;;) {
            const unsigned item = next_item(work, ws);
            if (item >= nitems) {
                more = item == 0xffffffffu;
                break;
            }
            pair_item<FLOOR, QMODE, SQUARE, EDGE, QMODE ? 1 : 2>(p, (int)item, rounds, sorted, fstart, fcount, cflag,
                                                                 frame_ok, sorted_q, ring, ring_q, ws, hist_base,
                                                                 trj_smem_addr(rowtab), qhist, pc, n_tested);
        }
        more = __syncthreads_or(more);
        merge_rows<SQUARE>(p, hist, hist_g, pc);
        if (edge_g) add_edges(edge_g, pc, n_tested);
        if (lane == 0) ws->since = (unsigned)clock();
        __syncthreads();
    }
    if (QMODE) {
        for (int k = tid; k < g.lsmax; k += blockDim.x) {
            const double s = qhist[k + 1];
            if (s != 0.0) atomicAdd(&gqq_frame[k], s);
        }
    }
}

// Group of a folded coordinate along one axis: cell, then box within the cell (NaN: the first ones).
__device__ __forceinline__ int cell_of(float r, float L, int nc, int nsub, int& box) {
    const float w = r - L * floorf(r / L);
    const float t = w * ((float)nc / L);
    int c = (int)t;
    c = c < 0 ? 0 : (c >= nc ? nc - 1 : c);
    const int sc = (int)((t - (float)c) * (float)nsub);
    box = sc < 0 ? 0 : (sc >= nsub ? nsub - 1 : sc);
    return c;
}

// Key, cell, cell flags (bit 0: a coordinate outside [0, L); bit 1: outside [-L, L) or NaN) and frame flags of
// an atom.
struct AtomCell {
    int key, cell;
    int flag;
    unsigned frame;
};
__device__ __forceinline__ AtomCell place(const float4& v, const RdfParams& p) {
    const float r[3] = {v.x, v.y, v.z};
    int k[3], sub[3];
    bool outside = false, far = false;
    AtomCell a;
    a.frame = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float L = p.g.L[d];
        outside |= !(r[d] >= 0.0f && r[d] < L);
        far |= !(r[d] >= -L && r[d] < L);
        a.frame |= (r[d] < -0.499f * L ? kFrameLow : 0u) | (r[d] < -0.749f * L ? kFrameVeryLow : 0u) |
                   (r[d] >= 0.749f * L ? kFrameHigh : 0u);
        k[d] = cell_of(r[d], L, p.nc[d], p.sub[d], sub[d]);
    }
    a.cell = (k[0] * p.nc[1] + k[1]) * p.nc[2] + k[2];
    a.key = a.cell * p.nsub + (sub[0] * p.sub[1] + sub[1]) * p.sub[2] + sub[2];
    a.flag = outside ? (far ? 3 : 1) : 0;
    return a;
}

// Cell of each atom from its wrapped coordinate, and its group: the cell is divided into sub[0] x sub[1] x
// sub[2] boxes numbered z fastest, so atoms sorted by key = cell * nsub + box are cell-contiguous and
// grouped by box.  Per-key counts and slots, cell and frame flags.
__global__ void cell_assign_kernel(const float4* __restrict__ packed, int64_t n, const __grid_constant__ RdfParams p,
                                   int32_t* __restrict__ fcount, int32_t* __restrict__ cflag,
                                   unsigned* __restrict__ fflag, int32_t* __restrict__ akey,
                                   int32_t* __restrict__ aslot) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned ff = 0;
    if (i < n) {
        const float4 v = packed[i];
        const AtomCell c = place(v, p);
        ff = c.frame;
        // A species outside 0..nsp-1 can only come from a frame already flagged as bad data: not placed.
        const bool ok = __float_as_uint(v.w) < (unsigned)p.g.nsp;
        akey[i] = ok ? c.key : -1;
        if (ok) aslot[i] = atomicAdd(&fcount[c.key], 1);
        if (c.flag) atomicOr(&cflag[c.cell], c.flag);
    }
    ff = __reduce_or_sync(0xffffffffu, ff);
    if ((threadIdx.x & 31) == 0 && (ff & ~*(volatile unsigned*)fflag)) atomicOr(fflag, ff);
}

// Atoms (low half) and rounds of homes (high half) of a group of v atoms: sums of both in one scan.
__device__ __forceinline__ u64 group_sums(int v) { return (u64)((v + kGroup - 1) / kGroup) << 32 | (unsigned)v; }

__device__ __forceinline__ u64 warp_scan(u64 x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// A group's rounds of homes: key and first atom of every 32 atoms, begin and end of the group.  The pair kernel's work goes by rounds, not by
// groups, because the groups of a frame of uneven density hold anything from no atom to all of them.  A ball of
// 62,500 atoms in a box 7.5 times as wide has groups of up to 3,900; with a warp for all homes of a group, and items
// for the empty ones too, 312 ms, with rounds 1.62; 20,000 atoms in one clump 343 and 1.33 ms.  Even frames gain as
// well, from items of one round instead of one or two: 62,500 atoms 0.36 -> 0.33 ms, 1e6 2.59 -> 2.43.
__device__ __forceinline__ void emit_rounds(int4* __restrict__ rounds, unsigned first, int key, int start, int v) {
    for (int i = 0; i * kGroup < v; ++i) rounds[first + i] = make_int4(key, start + i * kGroup, start, start + v);
}

// Start of every group in the sorted array, and its rounds.  Groups need only be contiguous, not in key order, so a
// block takes the room of its 256 groups from a counter instead of waiting for the sums before it: one short
// kernel in place of a scan over all keys.
__global__ void __launch_bounds__(256) group_offsets_kernel(const int32_t* __restrict__ fcount, int nkey,
                                                            u64* __restrict__ total, int32_t* __restrict__ fstart,
                                                            int4* __restrict__ rounds) {
    __shared__ u64 wsum[8], base;
    const int k = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int v = k < nkey ? fcount[k] : 0;
    const u64 x = warp_scan(group_sums(v), lane);
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        u64 sum = 0;
        for (int w = 0; w < 8; ++w) {
            const u64 y = wsum[w];
            wsum[w] = sum;
            sum += y;
        }
        base = atomicAdd(total, sum);
    }
    __syncthreads();
    if (k < nkey) {
        const u64 at = base + wsum[warp] + x - group_sums(v);
        fstart[k] = (int)(unsigned)at;
        emit_rounds(rounds, (unsigned)(at >> 32), k, (int)(unsigned)at, v);
    }
}

// Sum over a block of v (FP64, fixed order): warp shuffles, then warps in order; thread 0 has it.
__device__ __forceinline__ double block_sum(double v, double* red) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v += red[w];
    return v;
}

// q2[block]: sum of the block's squared charges (frames with charges).
__global__ void cell_scatter_kernel(const float4* __restrict__ packed, int64_t n,
                                    const int32_t* __restrict__ akey, const int32_t* __restrict__ aslot,
                                    const int32_t* __restrict__ fstart, unsigned wscale, float4* __restrict__ sorted,
                                    const float* __restrict__ q, float* __restrict__ sorted_q,
                                    double* __restrict__ q2) {
    __shared__ double red[32];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int key = i < n ? akey[i] : -1;
    const float qi = q && i < n ? q[i] : 0.f;
    if (key >= 0) {
        const int64_t d = fstart[key] + aslot[i];
        float4 v = packed[i];
        v.w = __uint_as_float(__float_as_uint(v.w) * wscale);  // species as the pair kernel adds it to addresses
        sorted[d] = v;
        if (q) sorted_q[d] = qi;
    }
    if (q) {
        const double s = block_sum((double)qi * (double)qi, red);
        if (threadIdx.x == 0) q2[blockIdx.x] = s;
    }
}

// The whole cell sort of a small frame in one CTA, counts in shared memory: one launch instead of a memset and
// three kernels, which between them cost more than the sort.  Each thread keeps its atoms' keys in registers.
constexpr int kSmallThreads = 1024, kSmallRounds = 8;
constexpr int kSmallAtoms = kSmallThreads * kSmallRounds;
constexpr int kSmallKeys = 4096;  // most groups, and most cells, of a frame sorted this way
__global__ void __launch_bounds__(kSmallThreads) cell_sort_small_kernel(
    const float4* __restrict__ packed, int n, const __grid_constant__ RdfParams p, int ncell, int nkey, unsigned wscale,
    unsigned* __restrict__ work, int32_t* __restrict__ cflag, int32_t* __restrict__ fcount,
    int32_t* __restrict__ fstart, int4* __restrict__ rounds, float4* __restrict__ sorted, const float* __restrict__ q,
    float* __restrict__ sorted_q, double* __restrict__ q2) {
    __shared__ double red[32];
    __shared__ int cnt[kSmallKeys], flag[kSmallKeys];
    __shared__ u64 wsum[32];
    __shared__ unsigned frame;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < nkey; k += kSmallThreads) cnt[k] = 0;
    for (int k = tid; k < ncell; k += kSmallThreads) flag[k] = 0;
    if (tid == 0) frame = 0u;
    __syncthreads();
    int key[kSmallRounds], slot[kSmallRounds];
    unsigned ff = 0;
#pragma unroll
    for (int r = 0; r < kSmallRounds; ++r) {
        const int i = r * kSmallThreads + tid;
        key[r] = -1;
        if (i < n) {
            const float4 v = packed[i];
            const AtomCell c = place(v, p);
            ff |= c.frame;
            if (__float_as_uint(v.w) < (unsigned)p.g.nsp) {
                key[r] = c.key;
                slot[r] = atomicAdd(&cnt[c.key], 1);
            }
            if (c.flag) atomicOr(&flag[c.cell], c.flag);
        }
    }
    if (ff) atomicOr(&frame, ff);
    __syncthreads();
    // starts: every thread scans kSmallKeys / kSmallThreads consecutive keys
    constexpr int kPer = kSmallKeys / kSmallThreads;
    int v[kPer];
    u64 sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int g = tid * kPer + k;
        v[k] = g < nkey ? cnt[g] : 0;
        sum += group_sums(v[k]);
    }
    const u64 x = warp_scan(sum, lane);
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    const u64 w = warp_scan(wsum[lane], lane);
    const u64 before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
    u64 run = (warp > 0 ? before : 0) + x - sum;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int g = tid * kPer + k;
        if (g < nkey) {
            const int at = (int)(unsigned)run;
            fstart[g] = at;
            fcount[g] = v[k];
            cnt[g] = at;
            emit_rounds(rounds, (unsigned)(run >> 32), g, at, v[k]);
        }
        run += group_sums(v[k]);
    }
    for (int k = tid; k < ncell; k += kSmallThreads) cflag[k] = flag[k];
    if (tid == kSmallThreads - 1) work[kWorkRounds] = (unsigned)(run >> 32);
    if (tid == 0) {
        work[kWorkNext] = 0u;
        work[kWorkFlags] = frame;
    }
    __syncthreads();
    double s2 = 0.0;
#pragma unroll
    for (int r = 0; r < kSmallRounds; ++r) {
        const int i = r * kSmallThreads + tid;
        const float qi = q && i < n ? q[i] : 0.f;
        s2 += (double)qi * (double)qi;
        if (key[r] >= 0) {
            const int d = cnt[key[r]] + slot[r];
            float4 a = packed[i];
            a.w = __uint_as_float(__float_as_uint(a.w) * wscale);
            sorted[d] = a;
            if (q) sorted_q[d] = qi;
        }
    }
    if (q) {
        s2 = block_sum(s2, red);
        if (tid == 0) q2[0] = s2;
    }
}

// One block, after the pair kernel: avq2 = sum(q^2)/N in FP64 rounded to FP32 (rdf.cuf:272, where
// avq2 is a default-real variable) from the sorting blocks' sums, then gqq += gqq_frame/avq2 (rdf.cuf:273).
// The order is fixed, so avq2 does not depend on scheduling.
__global__ void __launch_bounds__(1024) gqq_finish_kernel(const double* __restrict__ q2, int nparts, int64_t n,
                                                          const double* __restrict__ gqq_frame, int lsmax,
                                                          double* __restrict__ gqq) {
    __shared__ double red[32], total;
    double s = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < nparts; i += 1024) s += q2[i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) total = s;
    __syncthreads();
    const float avq2 = (float)(total / (double)n);
    for (int k = threadIdx.x; k < lsmax; k += 1024) gqq[k] += gqq_frame[k] / (double)avq2;
}

// The squared charge of a one-atom frame, which has no pairs and is not sorted.
__global__ void one_charge_kernel(const float* __restrict__ q, double* __restrict__ q2) {
    q2[0] = (double)q[0] * (double)q[0];
}

// Number fluctuations (s2D3_sh, rdf.cuf:489-553): block b draws one point uniformly in the box with
// the reference's generator and seed (XORWOW, curand_init(b + 12345, 0, 0), b 1-based), counts the
// atoms within each radius r_k = k*deltar (cumulative over nint(r/deltar) bins, the reference's
// gi_s(ind:lsmax) += 1) from the cells around it, and adds N_k and N_k^2 to the int64 sums.
//
// What bounds it: latency of the groups' starts and atoms.  A lane looks at a group of the point's cells (a warp
// at every eighth, so that the warps have equal shares) and drops it where its box is out of reach; the warp then
// has an atom of four groups per lane in flight, and groups of more than 128 atoms (frames of uneven density) go
// to the whole block.  The cumulative counts are a block scan.  4,096 points, every group of the cells read and eight
// consecutive ones to a warp against this: 1e6 atoms (cutoff 8) 0.268 and 0.122 ms, 62,500 atoms 0.334 and 0.131, a
// ball of them in a box of 400 0.432 and 0.077.
constexpr int kS2nThreads = 256, kS2nFlight = 4, kS2nLarge = 128, kS2nList = 64;
__global__ void __launch_bounds__(kS2nThreads, 5)
    s2n_kernel(const float4* __restrict__ sorted, const int32_t* __restrict__ fstart,
               const int32_t* __restrict__ fcount, const int32_t* __restrict__ cflag, const __grid_constant__ RdfParams p,
               unsigned long long* __restrict__ gi, unsigned long long* __restrict__ g2i, float* __restrict__ points,
               int dim) {
    const PairGeom& g = p.g;
    extern __shared__ unsigned s2n_cnt[];  // lsmax + 1
    unsigned* cnt = s2n_cnt;
    __shared__ float pt[3];
    __shared__ unsigned wsum[kS2nThreads / 32];
    __shared__ int2 large[kS2nList];  // groups left to the whole block: start and atoms
    __shared__ int nlarge;
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5), lsmax = g.lsmax;
    for (int k = threadIdx.x; k <= lsmax; k += kS2nThreads) cnt[k] = 0u;
    if (threadIdx.x == 0) {
        nlarge = 0;
        curandStateXORWOW_t h;
        curand_init((unsigned long long)blockIdx.x + 1ull + 12345ull, 0ull, 0ull, &h);
        pt[0] = g.L[0] * curand_uniform(&h);
        pt[1] = g.L[1] * curand_uniform(&h);
        pt[2] = dim == 2 ? 0.f : g.L[2] * curand_uniform(&h);  // s2D2_sh draws x and y only (rdf.cuf:580-581)
        if (points) {
            points[3 * blockIdx.x] = pt[0];
            points[3 * blockIdx.x + 1] = pt[1];
            points[3 * blockIdx.x + 2] = pt[2];
        }
    }
    __syncthreads();
    int pc[3];
    float pw[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {  // the point's cell, as cell_assign_kernel bins an atom
        pw[d] = pt[d] - g.L[d] * floorf(pt[d] / g.L[d]);
        int c = (int)(pw[d] * ((float)p.nc[d] / g.L[d]));
        pc[d] = c < 0 ? 0 : (c >= p.nc[d] ? p.nc[d] - 1 : c);
    }
    const float px = pt[0], py = pt[1], pz = pt[2];
    auto count = [&](const float4& a) {
        // rdf.cuf:533-541: difference point - atom, minimum image, (x^2 + y^2) + z^2, FP32
        const float xd = min_image(__fsub_rn(px, a.x), g.L[0], g.h1[0], g.h2[0]);
        const float yd = min_image(__fsub_rn(py, a.y), g.L[1], g.h1[1], g.h2[1]);
        const float zd = min_image(__fsub_rn(pz, a.z), g.L[2], g.h1[2], g.h2[2]);
        const float rr2 = __fadd_rn(__fadd_rn(__fmul_rn(xd, xd), __fmul_rn(yd, yd)), __fmul_rn(zd, zd));
        if (rr2 < g.side2) {
            const int ind = (int)roundf(__fdiv_rn(__fsqrt_rn(rr2), g.deltar));
            if (ind >= 0 && ind <= lsmax) atomicAdd(&cnt[ind], 1u);
        }
    };
    // an axis that is not split has one cell, a split one three or more
    const int sx = p.nc[0] > 1 ? 3 : 1, sy = p.nc[1] > 1 ? 3 : 1, sz = p.nc[2] > 1 ? 3 : 1;
    const int total = sx * sy * sz * p.nsub;
    for (int base = 0; base < total; base += kS2nThreads) {
        const int t = base + lane * (kS2nThreads / 32) + warp;
        int j0 = 0, na = 0;
        if (t < total) {
            const int e = fast_div(t, p.div_nsub), s = t - e * p.nsub;
            const int cx = wrapc(pc[0] + e / (sy * sz) - (sx >> 1), p.nc[0]);
            const int cy = wrapc(pc[1] + e / sz % sy - (sy >> 1), p.nc[1]);
            const int cz = wrapc(pc[2] + e % sz - (sz >> 1), p.nc[2]);
            const int cell = (cx * p.nc[1] + cy) * p.nc[2] + cz;
            bool near = cflag[cell] & 2;  // coordinates outside [-L, L): anywhere
            if (!near) {
                // nearest image of the group's box, as pair_item culls a neighbour group
                const int q = (int)(((float)s + 0.5f) * p.inv_sub[2]), bz = s - q * p.sub[2];
                const int bx = (int)(((float)q + 0.5f) * p.inv_sub[1]), by = q - bx * p.sub[1];
                const float dx = axis_gap<true>(((float)cx + ((float)bx + 0.5f) * p.inv_sub[0]) * p.edge[0], pw[0],
                                                p.half[0], g.L[0]);
                const float dy = axis_gap<true>(((float)cy + ((float)by + 0.5f) * p.inv_sub[1]) * p.edge[1], pw[1],
                                                p.half[1], g.L[1]);
                const float dz = axis_gap<true>(((float)cz + ((float)bz + 0.5f) * p.inv_sub[2]) * p.edge[2], pw[2],
                                                p.half[2], g.L[2]);
                near = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= p.cull2;
            }
            if (near) {
                const int key = cell * p.nsub + s;
                j0 = fstart[key];
                na = fcount[key];
                if (na > kS2nLarge) {
                    const int k = atomicAdd(&nlarge, 1);
                    if (k < kS2nList) {
                        large[k] = make_int2(j0, na);
                        na = 0;
                    }
                }
            }
        }
        unsigned m = __ballot_sync(0xffffffffu, na > 0);
        while (m) {
            float4 a[kS2nFlight];
            int n[kS2nFlight], j[kS2nFlight];
#pragma unroll
            for (int k = 0; k < kS2nFlight; ++k) {
                const int from = m ? __ffs(m) - 1 : 0;
                j[k] = __shfl_sync(0xffffffffu, j0, from);
                n[k] = __shfl_sync(0xffffffffu, na, from);
                if (!m) n[k] = 0;
                m &= m - 1u;
                if (lane < n[k]) a[k] = sorted[j[k] + lane];
            }
#pragma unroll
            for (int k = 0; k < kS2nFlight; ++k) {
                if (lane < n[k]) count(a[k]);
                for (int q = lane + 32; q < n[k]; q += 32) count(sorted[j[k] + q]);
            }
        }
    }
    __syncthreads();
    for (int k = 0; k < min(nlarge, kS2nList); ++k)
        for (int q = (int)threadIdx.x; q < large[k].y; q += kS2nThreads) count(sorted[large[k].x + q]);
    __syncthreads();
    // cumulative counts N_k = sum_{j <= k} cnt[j] (at most the frame's atoms): a thread's run, then the runs before it
    const int run = (lsmax + kS2nThreads) / kS2nThreads, k0 = (int)threadIdx.x * run, k1 = min(k0 + run, lsmax + 1);
    unsigned sum = 0;
    for (int k = k0; k < k1; ++k) sum += cnt[k];
    unsigned incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    unsigned at = incl - sum;
    for (int w = 0; w < warp; ++w) at += wsum[w];
    for (int k = k0; k < k1; ++k) {
        at += cnt[k];
        cnt[k] = at;
    }
    __syncthreads();
    for (int k = threadIdx.x; k <= lsmax; k += kS2nThreads) {
        const unsigned long long v = cnt[k];
        if (v) {
            atomicAdd(&gi[k], v);
            atomicAdd(&g2i[k], v * v);
        }
    }
}


// ---- fused multi-request launch: pair histogram of every packed frame --------------------------
//
// The cell sort and the work items of the single-frame path for all frames of the turn at once: keys and counts
// of every atom, group offsets (each item's groups start at its key_begin, a multiple of 32), placing, and one
// pair kernel whose CTAs each work on one frame at a time, merge its counts and move on to the next frame that
// has items left.
__global__ void __launch_bounds__(kBatchThreads) batch_keys_kernel(const BatchHeader* __restrict__ hdr,
                                                                   const BatchItem* __restrict__ items,
                                                                   const float4* __restrict__ packed, BatchSort st) {
    __shared__ RdfParams p;
    const int64_t total = hdr->total_chunk;
    int cur = -1;
    for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {
        const int r = batch_item_of<&BatchItem::chunk_begin>(items, hdr->nitems, u);
        const BatchItem& it = items[r];
        if (!it.hist) continue;  // block-uniform
        if (r != cur) {
            __syncthreads();
            for (int k = threadIdx.x; k < (int)(sizeof(RdfParams) / 4); k += kBatchThreads)
                reinterpret_cast<unsigned*>(&p)[k] = reinterpret_cast<const unsigned*>(&it.pair)[k];
            __syncthreads();
            cur = r;
        }
        const int64_t c = u - it.chunk_begin;
        for (int k = threadIdx.x; k < kBatchChunk; k += kBatchThreads) {
            const int64_t i = c * kBatchChunk + k;
            unsigned ff = 0;
            if (i < it.n) {
                const float4 v = packed[it.atom_off + i];
                const AtomCell a = place(v, p);
                ff = a.frame;
                const bool ok = __float_as_uint(v.w) < (unsigned)p.g.nsp;  // else flagged as bad data: not placed
                st.akey[it.atom_off + i] = ok ? a.key : -1;
                if (ok) st.aslot[it.atom_off + i] = atomicAdd(&st.fcount[it.key_begin + a.key], 1);
                if (a.flag) atomicOr(&st.cflag[it.key_begin + a.cell], a.flag);
            }
            ff = __reduce_or_sync(0xffffffffu, ff);
            if ((threadIdx.x & 31) == 0 && ff) atomicOr(&st.state[kWorkWords * r + kWorkFlags], ff);
        }
    }
}

__global__ void __launch_bounds__(kBatchThreads) batch_offsets_kernel(const BatchHeader* __restrict__ hdr,
                                                                      const BatchItem* __restrict__ items, BatchSort st) {
    const int lane = threadIdx.x & 31;
    for (int64_t k0 = ((int64_t)blockIdx.x * kBatchThreads + threadIdx.x) & ~31ll; k0 < hdr->total_key;
         k0 += (int64_t)gridDim.x * kBatchThreads) {
        const int r = batch_item_of<&BatchItem::key_begin>(items, hdr->nitems, k0);
        const int v = st.fcount[k0 + lane];
        const u64 x = warp_scan(group_sums(v), lane);
        u64 base = 0;
        if (lane == 31) base = atomicAdd(reinterpret_cast<u64*>(&st.state[kWorkWords * r + kWorkAtoms]), x);
        const u64 at = __shfl_sync(0xffffffffu, base, 31) + x - group_sums(v);
        st.fstart[k0 + lane] = (int)(unsigned)at;
        emit_rounds(st.rounds + batch_rounds_begin(items[r]), (unsigned)(at >> 32), (int)(k0 + lane - items[r].key_begin),
                    (int)(unsigned)at, v);
    }
}

__global__ void __launch_bounds__(kBatchThreads) batch_place_kernel(const BatchHeader* __restrict__ hdr,
                                                                    const BatchItem* __restrict__ items,
                                                                    const float4* __restrict__ packed, BatchSort st) {
    const int64_t total = hdr->total_chunk;
    for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {
        const BatchItem& it = items[batch_item_of<&BatchItem::chunk_begin>(items, hdr->nitems, u)];
        if (!it.hist) continue;
        const unsigned wscale = it.square ? 4u * (unsigned)it.pair.g.row_words : 64u;
        const int64_t c = u - it.chunk_begin;
        for (int k = threadIdx.x; k < kBatchChunk; k += kBatchThreads) {
            const int64_t i = c * kBatchChunk + k;
            if (i >= it.n) break;
            const int key = st.akey[it.atom_off + i];
            if (key < 0) continue;
            float4 v = packed[it.atom_off + i];
            v.w = __uint_as_float(__float_as_uint(v.w) * wscale);
            st.sorted[it.atom_off + st.fstart[it.key_begin + key] + st.aslot[it.atom_off + i]] = v;
        }
    }
}

// What bounds it: instruction issue, as the single-frame kernel.  64 frames of 1,000 to 16,384 atoms: 2.74 ms
// for an all-pairs sweep with a branch per pair, 0.70 ms so (80 registers a thread; 64, at four CTAs per SM: 0.73;
// two blocks of survivors per turn of the loop: 0.76, runs are short in small frames).
constexpr int kBatchPairWarps = 3 * kBatchThreads / 32;  // per SM
__global__ void __launch_bounds__(kBatchThreads, 3) batch_pairs_kernel(const BatchHeader* __restrict__ hdr,
                                                                       const BatchItem* __restrict__ items, BatchSort st,
                                                                       int hist_words) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ RdfParams p;
    __shared__ unsigned rowtab[256];
    __shared__ int next;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* ring = reinterpret_cast<float*>(smem + (size_t)warp * kWarpBytes);
    WarpState* ws = reinterpret_cast<WarpState*>(smem + (size_t)warp * kWarpBytes + 16 * kRing);
    unsigned* hist = reinterpret_cast<unsigned*>(smem + (size_t)(kBatchThreads / 32) * kWarpBytes);
    const unsigned hist_base = trj_smem_addr(hist), rowtab_base = trj_smem_addr(rowtab);
    for (int k = tid; k < batch_hist_smem_words(hist_words); k += kBatchThreads) hist[k] = 0u;
    const int nitems = hdr->nitems;
    if (nitems == 0) return;
    // CTAs start spread over the turn's work; each then moves on cyclically to frames with items left
    int r = batch_item_of<&BatchItem::pair_begin>(items, nitems, hdr->total_pair * blockIdx.x / gridDim.x);
    for (;;) {
        if (tid == 0) next = nitems;
        __syncthreads();
        for (int k = tid; k < nitems; k += kBatchThreads) {
            const int q = r + k < nitems ? r + k : r + k - nitems;
            const volatile unsigned* work = &st.state[kWorkWords * q];
            if (items[q].hist && work[kWorkNext] < work[kWorkRounds] * (unsigned)items[q].pair.nseg) {
                atomicMin(&next, k);
                break;
            }
        }
        __syncthreads();
        const int k = next;
        if (k >= nitems) break;
        r = r + k < nitems ? r + k : r + k - nitems;
        const BatchItem& it = items[r];
        for (int q = tid; q < (int)(sizeof(RdfParams) / 4); q += kBatchThreads)
            reinterpret_cast<unsigned*>(&p)[q] = reinterpret_cast<const unsigned*>(&it.pair)[q];
        __syncthreads();
        const bool square = it.square;
        if (!square)
            for (int q = tid; q < p.g.nsp * p.g.nsp; q += kBatchThreads)
                rowtab[(q / p.g.nsp) * 16 + q % p.g.nsp] =
                    hist_base + (unsigned)(trj_pair_row(q / p.g.nsp, q % p.g.nsp, p.g.nsp) * p.g.row_words * 4) -
                    4u * kBinBias;
        __syncthreads();
        PairCounters pc;
        u64 n_tested = 0;
        const bool frame_ok = frame_within(st.state[kWorkWords * r + kWorkFlags]);
        const unsigned nwork = st.state[kWorkWords * r + kWorkRounds] * (unsigned)p.nseg;
        const int4* rounds = st.rounds + batch_rounds_begin(it);
        const float4* sorted = st.sorted + it.atom_off;
        const int32_t *fstart = st.fstart + it.key_begin, *fcount = st.fcount + it.key_begin,
                      *cflag = st.cflag + it.key_begin;
        if (lane == 0) ws->since = (unsigned)clock();  // here, so that the first item is always taken
        for (;;) {
            const unsigned item = next_item(&st.state[kWorkWords * r + kWorkNext], ws);
            if (item >= nwork) break;
#define TRJ_ITEM(F, S, E)                                                                                       \
    pair_item<F, false, S, E, 1>(p, (int)item, rounds, sorted, fstart, fcount, cflag, frame_ok, nullptr, ring, nullptr, \
                                 ws, hist_base, rowtab_base, nullptr, pc, n_tested)
            if (p.g.floor_bins) TRJ_ITEM(true, false, true);
            else if (!square) TRJ_ITEM(false, false, true);
            else if (p.g.want_edge) TRJ_ITEM(false, true, true);
            else TRJ_ITEM(false, true, false);
#undef TRJ_ITEM
        }
        __syncthreads();
        if (square) merge_rows<true>(p, hist, it.hist, pc);
        else merge_rows<false>(p, hist, it.hist, pc);
        if (it.edge) add_edges(it.edge, pc, n_tested);
        __syncthreads();
        // the words before and after a row's bins as well: the next frame's rows lie elsewhere
        const int rows = square ? p.g.nsp * p.g.nsp : p.nit;
        for (int q = tid; q < rows * p.g.row_words; q += kBatchThreads) hist[q] = 0u;
        r = r + 1 < nitems ? r + 1 : 0;
    }
}

}  // namespace

struct trj_rdf_plan {
    trj_ctx* ctx = nullptr;
    int nsp = 0, nit = 0, lsmax = 0;
    int floor_bins = 0;
    long long wait_clocks = TRJ_WAIT_CLOCKS;  // limit of the stall test's wait
    int stall_test = 0;
    int dim = 3;                // 2: frames in the xy plane (z = 0); z is neither clipped nor split
    float deltar = 0.f, rcrdf_eff = 0.f, side2 = 0.f;
    int64_t n_max = 0;
    int ncell_cap = 0;
    int nc[3] = {1, 1, 1};      // cells per axis of the cutoff
    int64_t key_cap = 0;        // capacity of the per-group arrays
    int32_t* fstart = nullptr;  // key_cap: first atom of every (cell, group) in `sorted`
    // Zeroed per frame by one memset: work state (kWorkWords), cell flags (ncell: bit 0 a coordinate outside
    // [0, L), bit 1 outside [-L, L)), atoms per group (nkey).
    int32_t* zeroed = nullptr;  // kWorkWords + ncell_cap + key_cap
    int4* rounds = nullptr;     // key_cap + n_max / 32: every round of homes (emit_rounds)
    int32_t* akey = nullptr;    // n_max: (cell, group) key per atom
    int32_t* aslot = nullptr;   // n_max
    RdfParams frame_last;       // geometry, cells and groups of the last accumulated frame
    float4* sorted = nullptr;   // n_max
    float* sorted_q = nullptr;  // n_max charges in cell order (first charged call)
    int32_t *cflag_last = nullptr, *fcount_last = nullptr;  // its cell flags and atoms per group (in `zeroed`)
    int cells_valid = 0;        // sorted, fstart and the counts hold the last accumulated frame
    double* gqq_frame = nullptr;  // lsmax: this frame's charge-product sums
    double* q2_part = nullptr;    // one per sorting block: sums of squared charges
    int64_t scratch_bytes = 0;
    trj_kernel_timer timer;
};

// Least float x >= 0 with fl(x / L) >= q in FP32 (host SSE division, correctly rounded like the
// device's __fdiv_rn): the minimum-image thresholds of min_image.
static float nint_threshold(float L, float q) {
    volatile float vl = L;  // keep the division in single precision at run time
    float x = q * L;
    for (int k = 0; k < 256 && x > 0.f && x / vl >= q; ++k) x = nextafterf(x, 0.f);
    for (int k = 0; k < 256 && x / vl < q; ++k) x = nextafterf(x, INFINITY);
    return x;
}

// Most work items a fused frame's neighbour lists are cut into (frames of more rounds have one segment each).
constexpr int64_t kBatchItemsMost = (int64_t)1 << 20;

static int nint_host(float x) {  // Fortran NINT: half away from zero
    double v = (double)x;
    return (int)(v >= 0 ? floor(v + 0.5) : -floor(-v + 0.5));
}

// Smallest box edge of the plan's geometry (the x and y edges in 2D).
static float min_edge(const float box[3], int dim) {
    return dim == 2 ? fminf(box[0], box[1]) : fminf(box[0], fminf(box[1], box[2]));
}

// Cells per axis for cutoff^2 side2 in box L; axes with < 3 cells are not split (nor z in 2D).
static void cells_for(const float L[3], float side2, int nc[3], int dim = 3) {
    double rc = sqrt((double)side2) * (1.0 + 1.0 / 1024.0);
    for (int d = 0; d < 3; ++d) {
        int k = rc > 0 ? (int)floor((double)L[d] / rc) : 1;
        if (k < 3) k = 1;
        if (k > 1024) k = 1024;
        nc[d] = k;
    }
    if (dim == 2) nc[2] = 1;
}

// Shared memory kept back from the largest histogram a plan may have.
constexpr size_t kHistReserve = 20480;

// What a pair's test needs, from the frame's box and the plan's cutoff and bins.
static void fill_geom(PairGeom& g, const float box[3], float side2, float deltar, int lsmax, int nsp, int floor_bins,
                      bool want_edge) {
    for (int d = 0; d < 3; ++d) {
        g.L[d] = box[d];
        g.inv_L[d] = 1.0f / box[d];
        g.h1[d] = nint_threshold(box[d], 0.5f);
        g.h2[d] = nint_threshold(box[d], 1.5f);
    }
    g.side2 = side2;
    g.side2_lo = (float)((double)side2 * (1.0 - 1.0 / 1048576.0));
    g.side2_hi = (float)((double)side2 * (1.0 + 1.0 / 1048576.0));
    g.side2_win = fmaxf(g.side2_hi - side2, side2 - g.side2_lo);
    g.deltar = deltar;
    g.inv_deltar = 1.0f / deltar;
    // Window around a bin edge outside which the approximate q has the reference's bin (test_run): 0.34 (with
    // edge statistics 0.5) x 2^-20 of the largest q of a pair in range, plus 2^-22; floor bins round q + 1/2 once
    // more: 0.41 (0.57).  Cutoffs whose squares leave the normal range (and bins beyond the integer trick) take the
    // exact path throughout.
    const double qmax = sqrt((double)g.side2_hi) / (double)deltar + 1.0;
    const double window = floor_bins ? (want_edge ? 0.57 : 0.41) : (want_edge ? 0.5 : 0.34);
    const double thr = 0.5 - (qmax * window / 1048576.0 + 1.0 / 4194304.0);
    g.edge_thr = (side2 > 1e-30f && thr > 0.0) ? (float)thr : -1.0f;
    g.lsmax = lsmax;
    g.nsp = nsp;
    g.floor_bins = floor_bins;
    g.row_words = lsmax + 2;
    g.want_edge = want_edge;
    g.one = 1.0f;
}

static FastDiv make_fast_div(int d) {
    FastDiv f = {(unsigned)d, 0u, 0};
    if (d > 1) {
        int l = 0;
        while ((1ll << l) < d) ++l;
        f.mul = (unsigned)((((unsigned long long)1 << (31 + l)) + d - 1) / d);
        f.shift = l - 1;
    }
    return f;
}

// Volume (2D: area) of the region within r of a box of edges e: what the homes of one group are tested against.
static double reach(const double e[3], double r, int dim) {
    if (dim == 2) return e[0] * e[1] + 2.0 * r * (e[0] + e[1]) + M_PI * r * r;
    return e[0] * e[1] * e[2] + 2.0 * r * (e[0] * e[1] + e[1] * e[2] + e[2] * e[0]) +
           M_PI * r * r * (e[0] + e[1] + e[2]) + 4.0 / 3.0 * M_PI * r * r * r;
}

// Cells (nc, in: the most the cutoff allows) and groups per cell (sub) of an n-atom frame.  A group wants
// about 28 atoms, one per lane with room for fluctuations: sparse cells are merged (never below 3 per axis)
// and dense ones divided, into the split of lowest cost = groups x volume tested per group.
static void choose_groups(int64_t n, const float box[3], double rc, int dim, int64_t key_cap, int nc[3], int sub[3]) {
    const int nd = dim == 2 ? 2 : 3;
    double m = (double)n / ((double)nc[0] * nc[1] * nc[2]);
    if (m < 0.75 * kGroupFill) {
        const double f = pow(kGroupFill / std::max(m, 1e-3), 1.0 / nd);
        for (int d = 0; d < nd; ++d)
            if (nc[d] >= 3) nc[d] = std::max(3, (int)(nc[d] / f));
        m = (double)n / ((double)nc[0] * nc[1] * nc[2]);
    }
    // room for the cells themselves: coarser ones where there is not (an axis without a split always works)
    while ((int64_t)nc[0] * nc[1] * nc[2] > key_cap) {
        int d = nc[0] >= nc[1] ? (nc[0] >= nc[2] ? 0 : 2) : (nc[1] >= nc[2] ? 1 : 2);
        nc[d] = nc[d] > 3 ? std::max(3, nc[d] / 2) : 1;
    }
    m = (double)n / ((double)nc[0] * nc[1] * nc[2]);
    sub[0] = sub[1] = sub[2] = 1;
    if (m <= kGroupFill) return;
    double e[3], vol = 1.0;
    for (int d = 0; d < 3; ++d) e[d] = (double)box[d] / nc[d];
    for (int d = 0; d < nd; ++d) vol *= e[d];
    const double ideal = pow(vol * kGroupFill / m, 1.0 / nd);
    const int64_t most = std::max<int64_t>(1, key_cap / ((int64_t)nc[0] * nc[1] * nc[2]));
    double best = -1.0;
    int lo[3], hi[3];
    for (int d = 0; d < 3; ++d) {
        lo[d] = d < nd ? std::max(1, (int)(e[d] / ideal) - 1) : 1;
        hi[d] = d < nd ? std::max(1, (int)(e[d] / ideal) + 2) : 1;
    }
    for (int a = lo[0]; a <= hi[0]; ++a)
        for (int b = lo[1]; b <= hi[1]; ++b)
            for (int c = lo[2]; c <= hi[2]; ++c) {
                const double groups = (double)a * b * c;
                if (m / groups > kGroupFill || groups > (double)most) continue;
                const double edge[3] = {e[0] / a, e[1] / b, e[2] / c};
                const double cost = groups * reach(edge, rc, dim);
                if (best < 0.0 || cost < best) {
                    best = cost;
                    sub[0] = a;
                    sub[1] = b;
                    sub[2] = c;
                }
            }
}

// Cells, groups, stencil and cull of an n-atom frame; P.nc holds the most cells the cutoff allows.
static void fill_grid(RdfParams& P, int64_t n, const float box[3], float side2, float rc, int dim, int64_t key_cap) {
    choose_groups(n, box, rc, dim, key_cap, P.nc, P.sub);
    P.nsub = P.sub[0] * P.sub[1] * P.sub[2];
    // Cull radius 2^-10 above the cutoff (the exact test needs rr2 < side2*(1 + 2^-20)); the pad,
    // 2^-16 of the largest edge, exceeds the rounding of the box and gap arithmetic (a few ulps of
    // coordinates below 2L).
    P.cull2 = (float)((double)side2 * (1.0 + 1.0 / 1024.0) * (1.0 + 1.0 / 1024.0));
    P.cull_pad = (float)((double)std::max(box[0], std::max(box[1], box[2])) / 65536.0);
    for (int d = 0; d < 3; ++d) {
        P.inv_sub[d] = 1.0f / (float)P.sub[d];
        P.edge[d] = box[d] / (float)P.nc[d];
        P.half[d] = 0.5f * P.edge[d] / (float)P.sub[d] + P.cull_pad;
    }
    P.split_all = P.nc[0] >= 3 && P.nc[1] >= 3 && (P.nc[2] >= 3 || dim == 2);
    // Half-shell stencil over the split axes: (0,0,0) first, then offsets > 0 lexicographically.
    int no = 0;
    P.off[no][0] = P.off[no][1] = P.off[no][2] = 0;
    ++no;
    for (int dx = -1; dx <= 1; ++dx)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dz = -1; dz <= 1; ++dz) {
                if ((dx && P.nc[0] == 1) || (dy && P.nc[1] == 1) || (dz && P.nc[2] == 1)) continue;
                bool pos = dx > 0 || (dx == 0 && (dy > 0 || (dy == 0 && dz > 0)));
                if (!pos) continue;
                P.off[no][0] = dx;
                P.off[no][1] = dy;
                P.off[no][2] = dz;
                ++no;
            }
    P.nself = P.nsub / 2 + 1;
    P.list = P.nself + (no - 1) * P.nsub;
    P.div_nsub = make_fast_div(P.nsub);
    P.div_nc1 = make_fast_div(P.nc[1]);
    P.div_nc2 = make_fast_div(P.nc[2]);
}

// Neighbour lists cut into about nseg segments, at most so many that the work items of n atoms in nkey groups
// (the groups' rounds: ceil(atoms / 32) each) are below 2^31.
static void set_segments(RdfParams& P, int64_t nseg, int64_t nkey, int64_t n) {
    const int64_t rounds = nkey + n / kGroup;
    nseg = std::max<int64_t>(1, std::min(nseg, ((int64_t)1 << 30) / rounds));
    P.per_seg = (int)((P.list + nseg - 1) / nseg);
    P.nseg = (P.list + P.per_seg - 1) / P.per_seg;
    P.div_nseg = make_fast_div(P.nseg);
    P.nitems = (unsigned)(rounds * P.nseg);
}

constexpr size_t kPairStatic = 1200;  // more than the pair kernel's static shared memory

struct PairShape {
    int ctas, warps;  // per SM, per CTA
    bool square;      // a bin row per ordered species pair
    size_t smem;      // dynamic shared memory of a CTA
};

// Launch shape of the pair kernel: 32 warps per SM (64 registers a thread) in CTAs of 8 while their
// histograms fit, then fewer, larger CTAs that share one, then fewer warps.  The square row layout is
// taken where it does not cost warps.
static bool pair_shape(const trj_ctx* ctx, int nsp, int nit, int row_words, bool charged, PairShape* out) {
    static const int kCtas[] = {4, 2, 1, 1, 1, 1, 1};
    static const int kWarps[] = {8, 16, 32, 24, 16, 8, 4};
    const size_t optin = ctx->smem_optin, per_sm = optin + 1024;
    for (int i = 0; i < 7; ++i)
        for (int square = 1; square >= 0; --square) {
            const size_t rows = square ? (size_t)nsp * nsp : (size_t)nit;
            const size_t smem = (size_t)kWarps[i] * (kWarpBytes + (charged ? 8 * kRing : 0)) +
                                (size_t)row_words * (4 * rows + (charged ? 8 : 0)) + 16;
            // the driver's reserve and the static shared memory of a CTA
            if (smem + kPairStatic > optin || (smem + 1024 + kPairStatic) * kCtas[i] > per_sm) continue;
            out->ctas = kCtas[i];
            out->warps = kWarps[i];
            out->square = square;
            out->smem = smem;
            return true;
        }
    return false;
}

typedef void (*PairKernel)(RdfParams, const float4*, const int32_t*, const int32_t*, const int32_t*, const int4*, unsigned*,
                           u64*, u64*, unsigned*, const float*, double*);
template <bool FLOOR, bool SQUARE>
static PairKernel pair_kernel_of(bool charged, bool edge) {
    return charged ? rdf_pairs_kernel<FLOOR, true, SQUARE, true>
                   : (edge ? rdf_pairs_kernel<FLOOR, false, SQUARE, true> : rdf_pairs_kernel<FLOOR, false, SQUARE, false>);
}
static PairKernel pair_kernel(int floor_bins, bool charged, bool square, bool edge) {
    if (floor_bins) return square ? pair_kernel_of<true, true>(charged, edge) : pair_kernel_of<true, false>(charged, edge);
    return square ? pair_kernel_of<false, true>(charged, edge) : pair_kernel_of<false, false>(charged, edge);
}

static int rdf_plan_create_impl(trj_ctx* ctx, int nsp, float deltar, float rcrdf, const float box[3],
                                int64_t n_max, int dim, trj_rdf_plan** out) {
    if (!ctx || !out || !box) return TRJ_ERR_INVALID;
    *out = nullptr;
    if (nsp < 1 || nsp > 16) return trj_fail(ctx, TRJ_ERR_INVALID, "rdf plan: nsp=%d (1..16)", nsp);
    if (!(deltar > 0.f)) return trj_fail(ctx, TRJ_ERR_INVALID, "rdf plan: deltar must be > 0");
    if (!(box[0] > 0.f && box[1] > 0.f && box[2] > 0.f))
        return trj_fail(ctx, TRJ_ERR_INVALID, "rdf plan: box edges must be positive");
    if (n_max < 0 || n_max > (int64_t)INT32_MAX)
        return trj_fail(ctx, TRJ_ERR_INVALID, "rdf plan: n_max out of range");
    trj_rdf_plan* p = new trj_rdf_plan();
    p->ctx = ctx;
    p->nsp = nsp;
    p->nit = nsp * (nsp + 1) / 2;
    p->deltar = deltar;
    p->dim = dim;
    // select_ncdfinput (netcdf.f90:610-617): side = minval(L(1:ndim)); rcrdf = min(rcrdf, side/2)
    float side = min_edge(box, dim);
    float half = side / 2.0f;
    float rc = fminf(rcrdf, half);
    if (!(rc > 0.f)) rc = half;  // rcrdf <= 0 means half the box (netcdf.f90:613-617)
    p->rcrdf_eff = rc;
    p->side2 = rc * rc;
    // RDF_init (rdf.cuf:55-59)
    p->lsmax = nint_host(rc / deltar) + 1;
    p->n_max = n_max;
    size_t hist_bytes = (size_t)p->nit * p->lsmax * 4;
    size_t budget = ctx->smem_optin - kHistReserve;
    if (hist_bytes > budget) {
        delete p;
        return trj_fail(ctx, TRJ_ERR_UNSUPPORTED,
                        "rdf plan: histogram of %zu bytes exceeds shared memory (%zu); increase deltar "
                        "or reduce rcrdf", hist_bytes, budget);
    }
    cells_for(box, p->side2, p->nc, dim);
    int ncell = p->nc[0] * p->nc[1] * p->nc[2];
    // Room for a box up to 25% smaller per axis (more cells) without re-planning.
    p->ncell_cap = std::max(ncell * 2 + 64, 64);
    trj_device_guard g(ctx->device);
    // Groups: one per cell, or at least 16 atoms per group on average (choose_groups).
    p->key_cap = (int64_t)p->ncell_cap + n_max / 16 + 64;
    const size_t na = (size_t)std::max<int64_t>(n_max, 1);
    size_t bytes = 64 + sizeof(int32_t) * (size_t)(kWorkWords + p->ncell_cap + 2 * p->key_cap) +
                   (sizeof(int32_t) * 2 + sizeof(float4)) * na + sizeof(int4) * ((size_t)p->key_cap + na / kGroup + 1);
    char* base = nullptr;
    if (trj_dev_alloc(ctx, (void**)&base, bytes + 256) != cudaSuccess) {
        delete p;
        return trj_fail(ctx, TRJ_ERR_NOMEM, "rdf plan: %zu bytes of scratch", bytes);
    }
    p->sorted = reinterpret_cast<float4*>(base);
    p->rounds = reinterpret_cast<int4*>(p->sorted + na);
    p->akey = reinterpret_cast<int32_t*>(p->rounds + (size_t)p->key_cap + na / kGroup + 1);
    p->aslot = p->akey + na;
    p->zeroed = reinterpret_cast<int32_t*>((reinterpret_cast<uintptr_t>(p->aslot + na) + 15) & ~(uintptr_t)15);
    p->fstart = p->zeroed + kWorkWords + p->ncell_cap + p->key_cap;
    p->scratch_bytes = (int64_t)bytes;
    *out = p;
    return TRJ_OK;
}

extern "C" int trj_rdf_plan_create(trj_ctx* ctx, int nsp, float deltar, float rcrdf, const float box[3],
                                   int64_t n_max, trj_rdf_plan** out) {
    return rdf_plan_create_impl(ctx, nsp, deltar, rcrdf, box, n_max, 3, out);
}

extern "C" int trj_rdf_plan_create_2d(trj_ctx* ctx, int nsp, float deltar, float rcrdf, const float box[3],
                                      int64_t n_max, trj_rdf_plan** out) {
    return rdf_plan_create_impl(ctx, nsp, deltar, rcrdf, box, n_max, 2, out);
}

extern "C" int trj_rdf_plan_create_floor(trj_ctx* ctx, int nsp, float r_max, int nbins, const float box[3],
                                         int64_t n_max, trj_rdf_plan** out) {
    if (!ctx || !out || !box) return TRJ_ERR_INVALID;
    *out = nullptr;
    if (nbins < 1 || !(r_max > 0.f))
        return trj_fail(ctx, TRJ_ERR_INVALID, "rdf plan (floor bins): nbins=%d r_max=%g", nbins, (double)r_max);
    const float side = fminf(box[0], fminf(box[1], box[2]));
    if (!(r_max < side / 2.0f))
        return trj_fail(ctx, TRJ_ERR_INVALID, "rdf plan (floor bins): r_max=%g must be below half the box (%g)",
                        (double)r_max, (double)(side / 2.0f));
    const float deltar = r_max / (float)nbins;
    int rc = trj_rdf_plan_create(ctx, nsp, deltar, r_max, box, n_max, out);
    if (rc != TRJ_OK) return rc;
    trj_rdf_plan* p = *out;
    p->floor_bins = 1;
    p->lsmax = nbins;
    p->rcrdf_eff = r_max;
    p->side2 = r_max * r_max;
    return TRJ_OK;
}

extern "C" int trj_rdf_plan_info(const trj_rdf_plan* p, int* lsmax, int* nit, int cells[3], float* rcrdf_eff,
                                 float* side2, int64_t* scratch_bytes) {
    if (!p) return TRJ_ERR_INVALID;
    if (lsmax) *lsmax = p->lsmax;
    if (nit) *nit = p->nit;
    if (cells) for (int d = 0; d < 3; ++d) cells[d] = p->nc[d];
    if (rcrdf_eff) *rcrdf_eff = p->rcrdf_eff;
    if (side2) *side2 = p->side2;
    if (scratch_bytes) *scratch_bytes = p->scratch_bytes;
    return TRJ_OK;
}

extern "C" int trj_rdf_kernel_ms(trj_rdf_plan* p, float* ms) {
    if (!p) return TRJ_ERR_INVALID;
    return p->timer.elapsed(p->ctx, ms);
}

extern "C" int trj_rdf_plan_destroy(trj_rdf_plan* p) {
    if (!p) return TRJ_OK;
    {
        trj_device_guard g(p->ctx->device);
        trj_dev_free(p->ctx, p->sorted);
        trj_dev_free(p->ctx, p->sorted_q);
        p->timer.release();
    }
    delete p;
    return TRJ_OK;
}

// Frame accumulation; charge_dev/gqq_dev non-null adds the charge-product histogram.
static int rdf_accumulate_impl(trj_rdf_plan* plan, const float* packed_dev, const float* charge_dev, int64_t n,
                               const float box[3], uint64_t* hist_dev, uint64_t* edge_dev, double* gqq_dev,
                               void* stream) {
    if (!plan) return TRJ_ERR_INVALID;
    trj_ctx* ctx = plan->ctx;
    if (!box || !hist_dev) return trj_fail(ctx, TRJ_ERR_INVALID, "rdf accumulate: null argument");
    const bool charged = gqq_dev != nullptr;
    if (charged && n > 0 && !charge_dev)
        return trj_fail(ctx, TRJ_ERR_INVALID, "rdf accumulate: null charge array");
    if (n < 0 || n > plan->n_max)
        return trj_fail(ctx, TRJ_ERR_CAPACITY, "rdf accumulate: n=%lld exceeds plan n_max=%lld", (long long)n,
                        (long long)plan->n_max);
    if (n > 0 && (!packed_dev || ((uintptr_t)packed_dev) % 16))
        return trj_fail(ctx, TRJ_ERR_INVALID, "rdf accumulate: packed_dev null or not 16-byte aligned");
    if (!(box[0] > 0.f && box[1] > 0.f && box[2] > 0.f))
        return trj_fail(ctx, TRJ_ERR_INVALID, "rdf accumulate: box edges must be positive");
    trj_device_guard g(ctx->device);
    cudaStream_t s = (cudaStream_t)stream;
    if (charged && !plan->sorted_q) {
        const size_t nq = (size_t)std::max<int64_t>(plan->n_max, 1);
        const size_t charges = (nq * sizeof(float) + 255) & ~(size_t)255, blocks = (nq + 255) / 256;
        const size_t qbytes = charges + sizeof(double) * ((size_t)plan->lsmax + blocks);
        char* qb = nullptr;
        if (trj_dev_alloc(ctx, (void**)&qb, qbytes) != cudaSuccess)
            return trj_fail(ctx, TRJ_ERR_NOMEM, "rdf accumulate: %zu bytes of charge scratch", qbytes);
        plan->sorted_q = reinterpret_cast<float*>(qb);
        plan->gqq_frame = reinterpret_cast<double*>(qb + charges);
        plan->q2_part = plan->gqq_frame + plan->lsmax;
        plan->scratch_bytes += (int64_t)qbytes;
    }
    plan->cells_valid = 0;
    if (n < 2) {
        // No pair; gqq still receives 0/avq2 per bin, as the reference adds gqq_d/avq2 every frame.
        if (charged && n == 1) {
            TRJ_CUDA_TRY(ctx, cudaMemsetAsync(plan->gqq_frame, 0, sizeof(double) * plan->lsmax, s));
            one_charge_kernel<<<1, 1, 0, s>>>(charge_dev, plan->q2_part);
            gqq_finish_kernel<<<1, 1024, 0, s>>>(plan->q2_part, 1, n, plan->gqq_frame, plan->lsmax, gqq_dev);
            ctx->launches += 2;
            TRJ_CUDA_TRY(ctx, cudaGetLastError());
        }
        return TRJ_OK;
    }
    // Per-frame clip, as select_ncdfinput does on every frame (netcdf.f90:610-617).
    float side = min_edge(box, plan->dim);
    plan->rcrdf_eff = fminf(plan->rcrdf_eff, side / 2.0f);
    plan->side2 = plan->rcrdf_eff * plan->rcrdf_eff;

    RdfParams P;
    memset(&P, 0, sizeof(P));
    fill_geom(P.g, box, plan->side2, plan->deltar, plan->lsmax, plan->nsp, plan->floor_bins, edge_dev != nullptr);
    P.wait_clocks = plan->wait_clocks;
    P.stall_test = plan->stall_test;
    P.nit = plan->nit;
    cells_for(box, plan->side2, P.nc, plan->dim);
    for (int d = 0; d < 3; ++d) plan->nc[d] = P.nc[d];
    if (P.nc[0] * P.nc[1] * P.nc[2] > plan->ncell_cap)
        return trj_fail(ctx, TRJ_ERR_CAPACITY, "rdf accumulate: %d cells exceed plan capacity %d",
                        P.nc[0] * P.nc[1] * P.nc[2], plan->ncell_cap);
    fill_grid(P, n, box, plan->side2, plan->rcrdf_eff, plan->dim, plan->key_cap);
    const int ncell = P.nc[0] * P.nc[1] * P.nc[2];
    const int nkey = ncell * P.nsub;
    // Launch shape: as many warps per SM as the histogram leaves room for, with a row per ordered species
    // pair where that costs no warps.
    PairShape shape;
    if (!pair_shape(ctx, plan->nsp, plan->nit, P.g.row_words, charged, &shape))
        return trj_fail(ctx, TRJ_ERR_UNSUPPORTED, "rdf accumulate: histogram too large");
    // Segments: about twelve items per resident warp, so that the last ones end together (six: 62,500 atoms
    // 485 us instead of 455; twenty-four: 459), but at least two neighbour groups per item.
    const int64_t warps = (int64_t)ctx->sm_count * shape.ctas * shape.warps;
    set_segments(P, std::min<int64_t>((12 * warps + nkey - 1) / nkey, P.list / 2), nkey, n);

    const PairKernel kern = pair_kernel(plan->floor_bins, charged, shape.square, edge_dev != nullptr);
    // the most pair_shape gives any plan: a limit of this call's own could be lowered by another thread's before the
    // launch
    TRJ_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(ctx->smem_optin - kPairStatic)));

    // Cell binning: count, group offsets, scatter.
    unsigned* work = reinterpret_cast<unsigned*>(plan->zeroed);
    unsigned* fflag = work + kWorkFlags;
    int32_t* cflag = plan->zeroed + kWorkWords;
    int32_t* fcount = cflag + ncell;
    plan->fcount_last = fcount;
    plan->cflag_last = cflag;
    plan->frame_last = P;
    const unsigned wscale = shape.square ? 4u * (unsigned)P.g.row_words : 64u;
    const float* q_dev = charged ? charge_dev : nullptr;
    int q2_parts = 0;  // sums of squared charges, one per sorting block
    if (n <= kSmallAtoms && nkey <= kSmallKeys) {
        cell_sort_small_kernel<<<1, kSmallThreads, 0, s>>>((const float4*)packed_dev, (int)n, P, ncell, nkey, wscale, work,
                                                           cflag, fcount, plan->fstart, plan->rounds, plan->sorted,
                                                           q_dev, plan->sorted_q, plan->q2_part);
        q2_parts = 1;
        ctx->launches += 1;
    } else {
        TRJ_CUDA_TRY(ctx, cudaMemsetAsync(plan->zeroed, 0, sizeof(int32_t) * (size_t)(kWorkWords + ncell + nkey), s));
        const unsigned nb = (unsigned)((n + 255) / 256);
        cell_assign_kernel<<<nb, 256, 0, s>>>((const float4*)packed_dev, n, P, fcount, cflag, fflag, plan->akey,
                                              plan->aslot);
        group_offsets_kernel<<<(unsigned)((nkey + 255) / 256), 256, 0, s>>>(
            fcount, nkey, reinterpret_cast<u64*>(work + kWorkAtoms), plan->fstart, plan->rounds);
        cell_scatter_kernel<<<nb, 256, 0, s>>>((const float4*)packed_dev, n, plan->akey, plan->aslot, plan->fstart,
                                               wscale, plan->sorted, q_dev, plan->sorted_q, plan->q2_part);
        q2_parts = (int)nb;
        ctx->launches += 3;
    }
    if (charged) TRJ_CUDA_TRY(ctx, cudaMemsetAsync(plan->gqq_frame, 0, sizeof(double) * plan->lsmax, s));
    const int64_t grid = std::min<int64_t>((int64_t)ctx->sm_count * shape.ctas,
                                           ((int64_t)P.nitems + shape.warps - 1) / shape.warps);
    plan->timer.begin(ctx, s);
    kern<<<(unsigned)grid, shape.warps * 32, shape.smem, s>>>(P, plan->sorted, plan->fstart, fcount, cflag,
                                                              plan->rounds, work, (u64*)hist_dev, (u64*)edge_dev, ctx->status_dev,
                                                              charged ? plan->sorted_q : nullptr,
                                                              charged ? plan->gqq_frame : nullptr);
    plan->timer.end(ctx, s);
    plan->cells_valid = 1;
    ctx->launches += 1;
    if (charged) {
        gqq_finish_kernel<<<1, 1024, 0, s>>>(plan->q2_part, q2_parts, n, plan->gqq_frame, plan->lsmax, gqq_dev);
        ctx->launches += 1;
    }
    TRJ_CUDA_TRY(ctx, cudaGetLastError());
    return TRJ_OK;
}

extern "C" int trj_rdf_accumulate(trj_rdf_plan* plan, const float* packed_dev, int64_t n, const float box[3],
                                  uint64_t* hist_dev, uint64_t* edge_dev, void* stream) {
    return rdf_accumulate_impl(plan, packed_dev, nullptr, n, box, hist_dev, edge_dev, nullptr, stream);
}

extern "C" int trj_rdf_accumulate_charged(trj_rdf_plan* plan, const float* packed_dev, const float* charge_dev,
                                          int64_t n, const float box[3], uint64_t* hist_dev, uint64_t* edge_dev,
                                          double* gqq_dev, void* stream) {
    if (!plan) return TRJ_ERR_INVALID;
    if (!gqq_dev) return trj_fail(plan->ctx, TRJ_ERR_INVALID, "rdf accumulate (charged): null gqq");
    return rdf_accumulate_impl(plan, packed_dev, charge_dev, n, box, hist_dev, edge_dev, gqq_dev, stream);
}

extern "C" int trj_rdf_s2n(trj_rdf_plan* plan, int nrandom, uint64_t* gi_dev, uint64_t* g2i_dev, float* points_dev,
                           void* stream) {
    if (!plan) return TRJ_ERR_INVALID;
    trj_ctx* ctx = plan->ctx;
    if (nrandom < 0 || !gi_dev || !g2i_dev) return trj_fail(ctx, TRJ_ERR_INVALID, "rdf s2n: bad arguments");
    if (plan->floor_bins)
        return trj_fail(ctx, TRJ_ERR_UNSUPPORTED, "rdf s2n: needs the reference's nint bins (not a floor-bin plan)");
    if (!plan->cells_valid)
        return trj_fail(ctx, TRJ_ERR_INVALID, "rdf s2n: no frame accumulated (call trj_rdf_accumulate first)");
    if (nrandom == 0) return TRJ_OK;
    trj_device_guard g(ctx->device);
    const size_t smem = sizeof(unsigned) * (size_t)(plan->lsmax + 1), most = ((size_t)ctx->smem_optin - 64) / 2;
    if (smem > most) return trj_fail(ctx, TRJ_ERR_UNSUPPORTED, "rdf s2n: lsmax=%d too large", plan->lsmax);
    // Always, and always the same: without it the kernel's static shared memory counts against 48 KB as well, and a
    // value of this call's own could be lowered by another thread's before the launch.
    TRJ_CUDA_TRY(ctx, cudaFuncSetAttribute(s2n_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    s2n_kernel<<<(unsigned)nrandom, kS2nThreads, smem, (cudaStream_t)stream>>>(
        plan->sorted, plan->fstart, plan->fcount_last, plan->cflag_last, plan->frame_last, (unsigned long long*)gi_dev,
        (unsigned long long*)g2i_dev, points_dev, plan->dim);
    ctx->launches += 1;
    TRJ_CUDA_TRY(ctx, cudaGetLastError());
    return TRJ_OK;
}

extern "C" int trj_rdf_plan_set_binning(trj_rdf_plan* plan, int floor_bins) {
    if (!plan) return TRJ_ERR_INVALID;
    plan->floor_bins = floor_bins ? 1 : 0;
    return TRJ_OK;
}

extern "C" int trj_rdf_plan_set_wait(trj_rdf_plan* plan, int64_t clocks, int stall_test) {
    if (!plan) return TRJ_ERR_INVALID;
    if (clocks != 0 && (clocks < 1000 || clocks > TRJ_WAIT_CLOCKS))
        return trj_fail(plan->ctx, TRJ_ERR_INVALID, "trj_rdf_plan_set_wait: clocks %lld outside [1000, %lld] (0: default)",
                        (long long)clocks, (long long)TRJ_WAIT_CLOCKS);
    plan->wait_clocks = clocks ? clocks : TRJ_WAIT_CLOCKS;
    plan->stall_test = stall_test ? 1 : 0;
    return TRJ_OK;
}

// ---- fused multi-request launch: host side of the pair kernel ----------------------------------

size_t trj_batch_pairs_smem(int hist_words) {
    return (size_t)(kBatchThreads / 32) * kWarpBytes + 4 * (size_t)batch_hist_smem_words(hist_words);
}

int trj_batch_pairs_prepare() {
    // for the largest batch: a limit of this batch's own would refuse the launches of a larger one made before
    return cudaFuncSetAttribute(batch_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)trj_batch_pairs_smem(kBatchMaxHistWords)) == cudaSuccess ? 0 : -1;
}

int trj_batch_launch_pairs(BatchHeader* hdr, const BatchItem* items, const float4* packed, const BatchSort& st,
                           size_t zero_bytes, int hist_words, int grid_layout, int grid, cudaStream_t s) {
    if (cudaMemsetAsync(st.state, 0, zero_bytes, s) != cudaSuccess) return -1;
    batch_keys_kernel<<<grid_layout, kBatchThreads, 0, s>>>(hdr, items, packed, st);
    batch_offsets_kernel<<<grid_layout, kBatchThreads, 0, s>>>(hdr, items, st);
    batch_place_kernel<<<grid_layout, kBatchThreads, 0, s>>>(hdr, items, packed, st);
    batch_pairs_kernel<<<grid, kBatchThreads, trj_batch_pairs_smem(hist_words), s>>>(hdr, items, st, hist_words);
    return 0;
}

int trj_batch_pairs_occupancy(int hist_words, int* per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, batch_pairs_kernel, kBatchThreads,
                                                         trj_batch_pairs_smem(hist_words)) == cudaSuccess ? 0 : -1;
}

int trj_batch_fill_rdf(trj_rdf_plan* plan, int64_t n, const float box[3], int hist_words, int max_items, bool want_edge,
                       BatchItem* it, int* nsp, int64_t* nkey) {
    trj_ctx* ctx = plan->ctx;
    if (plan->dim != 3) return trj_fail(ctx, TRJ_ERR_UNSUPPORTED, "batch: two-dimensional pair plans run unfused");
    if (plan->nsp > kBatchMaxSpecies)
        return trj_fail(ctx, TRJ_ERR_UNSUPPORTED, "batch: %d species (1..%d)", plan->nsp, kBatchMaxSpecies);
    if ((int64_t)plan->nit * plan->lsmax > hist_words)
        return trj_fail(ctx, TRJ_ERR_UNSUPPORTED, "batch: a histogram of %d x %d bins exceeds the batch's %d words",
                        plan->nit, plan->lsmax, hist_words);
    // the per-frame clip of trj_rdf_accumulate (netcdf.f90:610-617)
    const float side = min_edge(box, plan->dim);
    plan->rcrdf_eff = fminf(plan->rcrdf_eff, side / 2.0f);
    plan->side2 = plan->rcrdf_eff * plan->rcrdf_eff;
    plan->cells_valid = 0;
    RdfParams& P = it->pair;
    memset(&P, 0, sizeof(P));
    fill_geom(P.g, box, plan->side2, plan->deltar, plan->lsmax, plan->nsp, plan->floor_bins, want_edge);
    P.nit = plan->nit;
    cells_for(box, plan->side2, P.nc);
    fill_grid(P, n, box, plan->side2, plan->rcrdf_eff, 3, batch_keys_most(n));
    *nkey = (int64_t)P.nc[0] * P.nc[1] * P.nc[2] * P.nsub;
    // About ten neighbour groups per item, fewer where a full turn of such frames would have less than two items per
    // warp (at least two groups: one ball of 16,000 atoms in a box of 200 has short lists, 466 -> 350 us), but
    // no more items than keep every warp of the GPU busy some 300 times over: the list grows with the frame, and
    // items are numbered in 31 bits.  One-atom frames have no pairs.
    const int64_t rounds = *nkey + n / kGroup, most = kBatchItemsMost / rounds;
    const int64_t want = 2 * (int64_t)ctx->sm_count * kBatchPairWarps / max_items;
    if (n >= 2)
        set_segments(P, std::min<int64_t>(std::max<int64_t>(P.list / 10, std::min<int64_t>(P.list / 2, want / rounds)), most),
                     *nkey, n);
    // a row per ordered species pair where those fit (floor bins: the general layout only)
    it->square = !plan->floor_bins &&
                 (int64_t)plan->nsp * plan->nsp * P.g.row_words <= (int64_t)batch_hist_smem_words(hist_words);
    *nsp = plan->nsp;
    return TRJ_OK;
}
