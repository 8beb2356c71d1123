// dyn.cu -- time correlations over multiple time origins: coherent and self intermediate
// scattering functions F(Q,t), Fs(Q,t) and the mean-squared displacement.
//
// Restates the device work of rtcorr (reference src/modules/dynamics.cuf:157-276) with the kernels
// FqtnD (:421-507) and rtcal (:510-547).  Each of nbuffer time origins ("buffers") keeps the state of
// its origin frame; every frame adds, for every buffer whose origin has been reached, one lag row:
//   F_b(k, lag)  += Re(rho_b(k, t0) conj(rho_b(k, t))),  rho_b(k, t) = sum_a bsc_a sum_{j in a} e^{i k.r_j(t)}
//   Fs_b(k, lag) += sum_j cos(k.(r_j(t) - r_j(t0)))
//   C_r,b(lag)   += sum_j |rt_j(t) - r_j(t0)|^2 / N     (rt: coordinates unwrapped per buffer)
// summed per output bin (the qw shell of k).  Which buffer takes which lag, and when a finished buffer
// is added to the totals, is the caller's bookkeeping (the origin shifting of rtcorr).
//
// Differences from the reference, by design:
// * rho_b(k, t0) is kept per buffer when the origin frame is seen, instead of being recomputed from
//   the origin positions in every later frame (FqtnD evaluates both sums for every buffer);
// * phases are exact: coordinates become 32-bit fixed-point fractions of the box (FP64, once per
//   atom and frame) and n.u wraps in integer arithmetic, so the FP32 cosine/sine always sees an
//   angle in [-pi, pi) (FqtnD feeds __cosf/__sinf FP32 phases of size |k| L);
// * sums are FP64 in a fixed order (FqtnD adds FP32 atomics);
// * lags beyond the plan's ndyn rows are not accumulated (FqtnD has no such bound and writes the row
//   after the last, i.e. the next buffer's first lag).
// The MSD arithmetic is the reference's FP32 per atom (unwrap, difference, dot product), summed in FP64.
#include <math.h>

#include <algorithm>
#include <vector>

#include "trj_common.cuh"

namespace {

constexpr int kDynThreads = 256;
constexpr int kDynVPT = 4;        // vectors per thread
constexpr int kDynChunk = 1024;   // least atoms of a slice
constexpr int kDynStage = 512;    // atoms staged per pass
constexpr int kDynSub = 64;       // FP32 run length before the FP64 add
constexpr int kDynCtas = 4;       // blocks of 256 threads per SM the launch shapes count on
constexpr float kTwoPiOver2_32 = 1.4629180792671596e-09f;

// Vectors in launch order: a thread's kDynVPT vectors are consecutive slots.  Slots hold the components with
// axis `axis` first; shared: the vectors of a thread have that component in common, so its product is formed
// once per atom.
struct DynSlots {
    const int4* slot;  // components, index of the vector (-1: padding)
    int64_t n;         // slots, a multiple of kDynVPT
    int axis, shared;
};

// Components of an atom's phase with the slots' axis first.
__device__ __forceinline__ uint4 axis_first(const uint4& a, int axis) {
    return axis == 0 ? a : axis == 1 ? make_uint4(a.y, a.x, a.z, a.w) : make_uint4(a.z, a.x, a.y, a.w);
}

// Atoms [s0, s1) of slice sl of nsl; a part of it takes runs [r0, r1) of 64 atoms from the slice's start, which
// fix the FP32 partial sums whatever the launch shape.
struct DynRuns {
    int64_t s0, s1, r0, r1;
};
__device__ __forceinline__ DynRuns dyn_runs(int64_t n, int row, int nsplit, int parts) {
    const int sl = row / parts, part = row - sl * parts;
    DynRuns r;
    r.s0 = n * sl / nsplit;
    r.s1 = n * (sl + 1) / nsplit;
    const int64_t runs = (r.s1 - r.s0 + kDynSub - 1) / kDynSub;
    r.r0 = runs * part / parts;
    r.r1 = runs * (part + 1) / parts;
    return r;
}

struct DynJob {
    int buf;     // buffer index
    int lag;     // 0-based lag row of this frame
    int origin;  // this frame is the buffer's origin
    int pad;
};

__global__ void dyn_phase_kernel(const float4* __restrict__ packed, int64_t n, double Lx, double Ly, double Lz,
                                 uint4* __restrict__ u) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 v = packed[i];
    const double s[3] = {(double)v.x / Lx, (double)v.y / Ly, (double)v.z / Lz};
    unsigned w[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double f = s[d] - floor(s[d]);
        w[d] = (unsigned)(long long)rint(f * 4294967296.0);  // 2^32 wraps to 0
    }
    u[i] = make_uint4(w[0], w[1], w[2], (unsigned)__float_as_int(v.w));
}

// Phases of a thread's vectors for one atom.
template <bool SHARED>
__device__ __forceinline__ void dyn_phases(const unsigned (&n0)[kDynVPT], const unsigned (&n1)[kDynVPT],
                                           const unsigned (&n2)[kDynVPT], const uint4& a, unsigned (&ph)[kDynVPT]) {
    const unsigned p0 = n0[0] * a.x;
#pragma unroll
    for (int q = 0; q < kDynVPT; ++q) ph[q] = (SHARED ? p0 : n0[q] * a.x) + n1[q] * a.y + n2[q] * a.z;
}

__device__ __forceinline__ void dyn_load_slots(const DynSlots& sl, int64_t first, unsigned (&n0)[kDynVPT],
                                               unsigned (&n1)[kDynVPT], unsigned (&n2)[kDynVPT]) {
#pragma unroll
    for (int q = 0; q < kDynVPT; ++q) {
        const int4 v = first < sl.n ? sl.slot[first + q] : make_int4(0, 0, 0, -1);
        n0[q] = (unsigned)v.x;
        n1[q] = (unsigned)v.y;
        n2[q] = (unsigned)v.z;
    }
}

// Partial rho(k) = sum_j bsc[species_j] e^{i k.r_j} over the runs of row blockIdx.y, by slot.
template <bool SHARED>
__global__ void __launch_bounds__(kDynThreads, kDynCtas) dyn_rho_kernel(const uint4* __restrict__ u, int64_t n,
                                                                        const float* __restrict__ bsc, int nsp,
                                                                        DynSlots sl, int nsplit, int parts,
                                                                        double2* __restrict__ part) {
    __shared__ uint4 atoms[kDynStage];  // w: the atom's weight
    const int tid = threadIdx.x;
    const int64_t first = ((int64_t)blockIdx.x * blockDim.x + tid) * kDynVPT;
    unsigned n0[kDynVPT], n1[kDynVPT], n2[kDynVPT];
    dyn_load_slots(sl, first, n0, n1, n2);
    const DynRuns rr = dyn_runs(n, blockIdx.y, nsplit, parts);
    double accr[kDynVPT], acci[kDynVPT];
#pragma unroll
    for (int q = 0; q < kDynVPT; ++q) accr[q] = acci[q] = 0.0;
    for (int64_t r = rr.r0; r < rr.r1; r += kDynStage / kDynSub) {
        const int64_t c0 = rr.s0 + r * kDynSub, c1 = min(rr.s1, rr.s0 + min(r + kDynStage / kDynSub, rr.r1) * kDynSub);
        const int cnt = (int)(c1 - c0);
        __syncthreads();
        for (int k = tid; k < cnt; k += (int)blockDim.x) {
            uint4 a = axis_first(u[c0 + k], sl.axis);
            const int s = (int)a.w;
            a.w = __float_as_uint((s >= 0 && s < nsp) ? bsc[s] : 0.f);
            atoms[k] = a;
        }
        __syncthreads();
        for (int j0 = 0; j0 < cnt; j0 += kDynSub) {
            const int j1 = min(cnt, j0 + kDynSub);
            u64 fr[kDynVPT / 2], fi[kDynVPT / 2];
#pragma unroll
            for (int q = 0; q < kDynVPT / 2; ++q) fr[q] = fi[q] = 0ull;
            for (int j = j0; j < j1; ++j) {
                const uint4 a = atoms[j];
                const u64 w = pack2(__uint_as_float(a.w), __uint_as_float(a.w));
                unsigned ph[kDynVPT];
                dyn_phases<SHARED>(n0, n1, n2, a, ph);
#pragma unroll
                for (int q = 0; q < kDynVPT / 2; ++q) {
                    float x, y, sx, cx, sy, cy;
                    unpack2(mul2(pack2(__int2float_rn((int)ph[2 * q]), __int2float_rn((int)ph[2 * q + 1])),
                                 pack2(kTwoPiOver2_32, kTwoPiOver2_32)),
                            x, y);
                    __sincosf(x, &sx, &cx);
                    __sincosf(y, &sy, &cy);
                    fr[q] = fma2(w, pack2(cx, cy), fr[q]);
                    fi[q] = fma2(w, pack2(sx, sy), fi[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < kDynVPT / 2; ++q) {
                float x, y;
                unpack2(fr[q], x, y);
                accr[2 * q] += (double)x;
                accr[2 * q + 1] += (double)y;
                unpack2(fi[q], x, y);
                acci[2 * q] += (double)x;
                acci[2 * q + 1] += (double)y;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kDynVPT; ++q)
        if (first < sl.n) part[(int64_t)blockIdx.y * sl.n + first + q] = make_double2(accr[q], acci[q]);
}

// rho_t = sum over the rows (fixed order: warp w of eight takes rows w, w + 8, ..., then the warps in order), 32
// slots per block; origin buffers keep a copy as their rho(k, t0).
__global__ void __launch_bounds__(256) dyn_rho_gather_kernel(const double2* __restrict__ part,
                                                             const int4* __restrict__ slot, int64_t nslot,
                                                             int64_t nvec, int rows, const DynJob* __restrict__ jobs,
                                                             int njobs, double2* __restrict__ rho_t,
                                                             double2* __restrict__ rho0) {
    __shared__ double2 red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t s = (int64_t)blockIdx.x * 32 + lane;
    double2 t = make_double2(0.0, 0.0);
    if (s < nslot) {
#pragma unroll 8
        for (int r = warp; r < rows; r += 8) {
            const double2 p = part[(int64_t)r * nslot + s];
            t.x += p.x;
            t.y += p.y;
        }
    }
    red[warp][lane] = t;
    __syncthreads();
    const int k = warp == 0 && s < nslot ? slot[s].w : -1;
    if (k < 0) return;
    for (int w = 1; w < 8; ++w) {
        t.x += red[w][lane].x;
        t.y += red[w][lane].y;
    }
    rho_t[k] = t;
    for (int j = 0; j < njobs; ++j)
        if (jobs[j].origin) rho0[(int64_t)jobs[j].buf * nvec + k] = t;
}

// Origin frames: phases and coordinates of every atom become the buffer's origin state.
__global__ void dyn_origin_kernel(const float4* __restrict__ packed, const uint4* __restrict__ u, int64_t n,
                                  const DynJob* __restrict__ jobs, uint4* __restrict__ u0,
                                  float4* __restrict__ r0, float4* __restrict__ rt) {
    const DynJob jb = jobs[blockIdx.y];
    if (!jb.origin) return;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t o = (int64_t)jb.buf * n + i;
    const float4 v = packed[i];
    u0[o] = u[i];
    r0[o] = v;
    rt[o] = v;
}

// rtcal (dynamics.cuf:510-547): unwrap rt toward the current frame, FP32 |rt - r0|^2 per atom,
// FP64 block sums (written per block, reduced in a fixed order later).
__global__ void dyn_msd_kernel(const float4* __restrict__ packed, int64_t n, float Lx, float Ly, float Lz,
                               const DynJob* __restrict__ jobs, const float4* __restrict__ r0,
                               float4* __restrict__ rt, double* __restrict__ msd_part) {
    __shared__ double red[kDynThreads / 32];
    const DynJob jb = jobs[blockIdx.y];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double s = 0.0;
    if (i < n) {
        const int64_t o = (int64_t)jb.buf * n + i;
        const float4 r = packed[i];
        float4 t = rt[o];
        const float L[3] = {Lx, Ly, Lz};
        float rc[3] = {r.x, r.y, r.z}, tc[3] = {t.x, t.y, t.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            // rt = r + L*nint((rt - r)/L), each FP32 operation rounded once (nint: half away from zero)
            const float m = roundf(__fdiv_rn(__fsub_rn(tc[d], rc[d]), L[d]));
            tc[d] = __fadd_rn(rc[d], __fmul_rn(L[d], m));
        }
        t.x = tc[0];
        t.y = tc[1];
        t.z = tc[2];
        rt[o] = t;
        const float4 z = r0[o];
        const float dx = __fsub_rn(t.x, z.x), dy = __fsub_rn(t.y, z.y), dz = __fsub_rn(t.z, z.z);
        s = (double)__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        msd_part[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = t;
    }
}

// Partial Fs(k) = sum_j cos(k.(r_j(t) - r_j(t0))) over the runs of row blockIdx.y, for job blockIdx.z, by slot.
//
// What bounds it: the special-function unit's cosine (8.4 clocks per warp and scheduler) and, nearly as long, the
// FMA pipe's integer multiply-adds of the phase, one per atom less for vectors that share a component.  62,500
// atoms x 5,319 vectors x 10 origins: 1.33 ms with one wave and a bit of equal blocks, 0.96 ms so (floor of the
// cosines alone 0.76; five blocks per SM or no unrolling: 1.04 to 1.24 at 256 threads, where this took 1.06).
template <bool SHARED>
__global__ void __launch_bounds__(kDynThreads, kDynCtas) dyn_self_kernel(const uint4* __restrict__ u,
                                                                         const uint4* __restrict__ u0, int64_t n,
                                                                         const DynJob* __restrict__ jobs, DynSlots sl,
                                                                         int nsplit, int parts,
                                                                         double* __restrict__ part) {
    __shared__ uint4 dis[kDynStage];
    const int tid = threadIdx.x;
    const DynJob jb = jobs[blockIdx.z];
    const uint4* __restrict__ org = u0 + (int64_t)jb.buf * n;
    const int64_t first = ((int64_t)blockIdx.x * blockDim.x + tid) * kDynVPT;
    unsigned n0[kDynVPT], n1[kDynVPT], n2[kDynVPT];
    dyn_load_slots(sl, first, n0, n1, n2);
    const DynRuns rr = dyn_runs(n, blockIdx.y, nsplit, parts);
    double acc[kDynVPT];
#pragma unroll
    for (int q = 0; q < kDynVPT; ++q) acc[q] = 0.0;
    for (int64_t r = rr.r0; r < rr.r1; r += kDynStage / kDynSub) {
        const int64_t c0 = rr.s0 + r * kDynSub, c1 = min(rr.s1, rr.s0 + min(r + kDynStage / kDynSub, rr.r1) * kDynSub);
        const int cnt = (int)(c1 - c0);
        __syncthreads();
        for (int k = tid; k < cnt; k += (int)blockDim.x) {
            const uint4 a = u[c0 + k], b = org[c0 + k];
            // displacement, exact mod 1 box
            dis[k] = axis_first(make_uint4(a.x - b.x, a.y - b.y, a.z - b.z, 0u), sl.axis);
        }
        __syncthreads();
        for (int j0 = 0; j0 < cnt; j0 += kDynSub) {
            const int j1 = min(cnt, j0 + kDynSub);
            u64 f[kDynVPT / 2];
#pragma unroll
            for (int q = 0; q < kDynVPT / 2; ++q) f[q] = 0ull;
#pragma unroll 2
            for (int j = j0; j < j1; ++j) {
                unsigned ph[kDynVPT];
                dyn_phases<SHARED>(n0, n1, n2, dis[j], ph);
#pragma unroll
                for (int q = 0; q < kDynVPT / 2; ++q) {
                    float x, y;
                    unpack2(mul2(pack2(__int2float_rn((int)ph[2 * q]), __int2float_rn((int)ph[2 * q + 1])),
                                 pack2(kTwoPiOver2_32, kTwoPiOver2_32)),
                            x, y);
                    f[q] = add2(f[q], pack2(__cosf(x), __cosf(y)));
                }
            }
#pragma unroll
            for (int q = 0; q < kDynVPT / 2; ++q) {
                float x, y;
                unpack2(f[q], x, y);
                acc[2 * q] += (double)x;
                acc[2 * q + 1] += (double)y;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kDynVPT; ++q)
        if (first < sl.n) part[((int64_t)blockIdx.z * nsplit * parts + blockIdx.y) * sl.n + first + q] = acc[q];
}

// Per job and vector: the self term's rows added up (fixed order, as for rho).
__global__ void dyn_self_gather_kernel(const double* __restrict__ part, const int4* __restrict__ slot, int64_t nslot,
                                       int64_t nvec, int rows, double* __restrict__ self) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslot) return;
    const int k = slot[s].w;
    if (k < 0) return;
    const double* p = part + (int64_t)blockIdx.y * rows * nslot + s;
    double t[8] = {};
    for (int r = 0; r < rows; r += 8)
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if (r + c < rows) t[c] += p[(int64_t)(r + c) * nslot];
    double sum = 0.0;
#pragma unroll
    for (int c = 0; c < 8; ++c) sum += t[c];
    self[(int64_t)blockIdx.y * nvec + k] = sum;
}

// Block sum of v in a fixed order (warp shuffles, warps in order); thread 0 has it.
__device__ __forceinline__ double dyn_block_sum(double v, double* red) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v += red[w];
    return v;
}

// One block per (bin, job): the bin's vectors in a fixed order; bin 0's block also adds the MSD.
__global__ void __launch_bounds__(kDynThreads) dyn_reduce_kernel(
    const double* __restrict__ self, const double2* __restrict__ rho_t, const double2* __restrict__ rho0,
    const int32_t* __restrict__ bin_start, const int32_t* __restrict__ bin_vec, int64_t nvec, int nbins, int ndyn,
    const DynJob* __restrict__ jobs, const double* __restrict__ msd_part, int msd_blocks, int64_t n,
    double* __restrict__ fc, double* __restrict__ fs, double* __restrict__ msd) {
    __shared__ double red[3][kDynThreads / 32];
    const int bin = blockIdx.x, j = blockIdx.y;
    const DynJob jb = jobs[j];
    const int v0 = bin_start[bin], v1 = bin_start[bin + 1];
    double sc = 0.0, ss = 0.0, m = 0.0;
    for (int t = v0 + threadIdx.x; t < v1; t += kDynThreads) {
        const int k = bin_vec[t];
        const double2 a = rho0[(int64_t)jb.buf * nvec + k], b = rho_t[k];
        sc += a.x * b.x + a.y * b.y;
        ss += self[(int64_t)j * nvec + k];
    }
    if (bin == 0)
        for (int b = threadIdx.x; b < msd_blocks; b += kDynThreads) m += msd_part[(int64_t)j * msd_blocks + b];
    sc = dyn_block_sum(sc, red[0]);
    ss = dyn_block_sum(ss, red[1]);
    m = dyn_block_sum(m, red[2]);
    if (threadIdx.x == 0) {
        const int64_t o = ((int64_t)jb.buf * ndyn + jb.lag) * nbins + bin;
        fc[o] += sc;
        fs[o] += ss;
        if (bin == 0) msd[(int64_t)jb.buf * ndyn + jb.lag] += m / (double)n;
    }
}

// Finished buffers: their rows are added to the totals and cleared (rtcorr, dynamics.cuf:250-268).
__global__ void dyn_flush_kernel(const int32_t* __restrict__ done, int ndone, int ndyn, int nbins,
                                 double* __restrict__ fc, double* __restrict__ fs, double* __restrict__ msd,
                                 double* __restrict__ fkt, double* __restrict__ fskt, double* __restrict__ r2t) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t rows = (int64_t)ndyn * nbins;
    if (e < rows) {
        double c = fkt[e], s = fskt[e];
        for (int d = 0; d < ndone; ++d) {
            const int64_t o = (int64_t)done[d] * rows + e;
            c += fc[o];
            s += fs[o];
            fc[o] = 0.0;
            fs[o] = 0.0;
        }
        fkt[e] = c;
        fskt[e] = s;
    }
    if (e < ndyn) {
        double m = r2t[e];
        for (int d = 0; d < ndone; ++d) {
            const int64_t o = (int64_t)done[d] * ndyn + e;
            m += msd[o];
            msd[o] = 0.0;
        }
        r2t[e] = m;
    }
}

}  // namespace

struct trj_dyn_plan {
    trj_ctx* ctx = nullptr;
    int nsp = 0, nbuf = 0, ndyn = 0, nbins = 0;
    int64_t n = 0, nvec = 0;
    int gx = 1;              // vector blocks the slice counts go by
    int nsplit_rho = 1;      // slices: they fix the FP32 partial sums
    int nsplit_cap = 1;      // slices of the self term: nsplit * jobs <= nsplit_cap
    int parts_rho = 1;       // parts of a slice
    int gslot = 1, tslot = kDynThreads;  // slot blocks of the rho/self kernels, threads of one
    DynSlots slots = {};
    int4* slot_dev = nullptr;
    int32_t* bin_start = nullptr;  // nbins + 1
    int32_t* bin_vec = nullptr;    // vectors of each bin
    float* bsc = nullptr;
    uint4* u = nullptr;            // n
    uint4* u0 = nullptr;           // nbuf * n
    float4* r0 = nullptr;          // nbuf * n
    float4* rt = nullptr;          // nbuf * n
    double2* rho_part = nullptr;   // rows x slots
    double2* rho_t = nullptr;      // nvec
    double2* rho0 = nullptr;       // nbuf * nvec
    double* self_part = nullptr;   // rows x jobs x slots
    double* self = nullptr;        // nbuf * nvec
    double* msd_part = nullptr;    // nbuf * msd_blocks
    double* fc = nullptr;          // nbuf * ndyn * nbins
    double* fs = nullptr;          // nbuf * ndyn * nbins
    double* msd = nullptr;         // nbuf * ndyn
    DynJob* jobs_dev = nullptr;    // nbuf
    int32_t* done_dev = nullptr;   // nbuf
    std::vector<std::pair<void**, size_t>> arrays;  // the arrays above: where their address goes, their offset
    void* block = nullptr;         // one allocation of them all: each of its own took up to 0.3 ms
    int64_t scratch_bytes = 0;
    trj_kernel_timer timer;        // around the self kernel
};

static void dyn_free(trj_dyn_plan* p) {
    trj_device_guard g(p->ctx->device);
    trj_dev_free(p->ctx, p->block);
    p->block = nullptr;
    p->timer.release();
}

// Room for an array in the plan's allocation; dyn_alloc_all sets the arrays' addresses.
template <class T>
static void dyn_want(trj_dyn_plan* p, T** out, size_t count) {
    p->arrays.emplace_back(reinterpret_cast<void**>(out), (size_t)p->scratch_bytes);
    p->scratch_bytes += (int64_t)((std::max<size_t>(1, count) * sizeof(T) + 255) & ~(size_t)255);
}

static bool dyn_alloc_all(trj_dyn_plan* p) {
    if (trj_dev_alloc(p->ctx, &p->block, (size_t)p->scratch_bytes) != cudaSuccess) return false;
    for (const auto& a : p->arrays) *a.first = static_cast<char*>(p->block) + a.second;
    return true;
}

// Slices of the self term for nj jobs.
static int self_split(const trj_dyn_plan* p, int nj) {
    const int64_t target = (int64_t)p->ctx->sm_count * 8;
    const int64_t by_atoms = std::max<int64_t>(1, p->n / kDynChunk);
    const int64_t blocks = (int64_t)p->gx * nj;
    const int nsplit = (int)std::min<int64_t>(by_atoms, std::max<int64_t>(1, (target + blocks - 1) / blocks));
    return std::max(1, std::min(nsplit, p->nsplit_cap / nj));
}

// Parts of a slice: the number that wastes least of the last wave of equal blocks (up to six waves), within the
// slice's runs and 256 MB of partials.
static int dyn_parts(const trj_dyn_plan* p, int64_t blocks, int nsplit, int64_t row_bytes) {
    const double slots = (double)p->ctx->sm_count * (kDynCtas * kDynThreads / p->tslot);
    const int64_t runs = std::max<int64_t>(1, p->n / ((int64_t)nsplit * kDynSub));
    const int64_t room = std::max<int64_t>(1, ((int64_t)256 << 20) / std::max<int64_t>(1, row_bytes));
    const int64_t most = std::max<int64_t>(1, std::min(std::min(runs, room), (int64_t)(6.0 * slots / (double)blocks)));
    double best = 0.0;
    int parts = 1;
    for (int64_t k = 1; k <= most; ++k) {
        const double waves = (double)(blocks * k) / slots, use = waves / ceil(waves);
        if (use > best + 0.01) {
            best = use;
            parts = (int)k;
        }
    }
    return parts;
}

// Vectors by their component on an axis: how many there are of each of the values lo, lo + 1, ...  Empty where
// the values are too far apart to count.
struct DynAxis {
    int64_t lo = 0;
    std::vector<int64_t> count;
    DynAxis(const int32_t* vec, int64_t nvec, int ax) {
        if (!nvec) return;
        int64_t hi = lo = vec[ax];
        for (int64_t v = 1; v < nvec; ++v) {
            lo = std::min<int64_t>(lo, vec[3 * v + ax]);
            hi = std::max<int64_t>(hi, vec[3 * v + ax]);
        }
        if (hi - lo > 4 * nvec + 1024) return;
        count.assign((size_t)(hi - lo + 1), 0);
        for (int64_t v = 0; v < nvec; ++v) ++count[(size_t)(vec[3 * v + ax] - lo)];
    }
};

// Slots of the vectors when each component's are padded to whole threads; components too far apart: as if each
// vector had one of its own.
static int64_t dyn_axis_slots(const int32_t* vec, int64_t nvec, int ax) {
    const DynAxis a(vec, nvec, ax);
    if (a.count.empty()) return nvec * kDynVPT;
    int64_t total = 0;
    for (int64_t c : a.count) total += (c + kDynVPT - 1) / kDynVPT * kDynVPT;
    return total;
}

// The vectors by their component on axis ax, in the caller's order where it is the same (ax < 0: throughout).
// Counting, not sorting: 5,319 vectors took 1.1 ms to sort for the three axes, 200,000 took 50.
static std::vector<int64_t> dyn_axis_order(const int32_t* vec, int64_t nvec, int ax) {
    std::vector<int64_t> order(nvec);
    if (ax < 0) {
        for (int64_t v = 0; v < nvec; ++v) order[v] = v;
        return order;
    }
    DynAxis a(vec, nvec, ax);
    int64_t at = 0;
    for (int64_t& c : a.count) {
        const int64_t n = c;
        c = at;
        at += n;
    }
    for (int64_t v = 0; v < nvec; ++v) order[(size_t)a.count[(size_t)(vec[3 * v + ax] - a.lo)]++] = v;
    return order;
}

extern "C" int trj_dyn_plan_create(trj_ctx* ctx, int nsp, int64_t n, int nbuffer, int ndyn, int64_t nvec,
                                   const int32_t* vec_host, const int32_t* bin_host, int nbins,
                                   const float* bsc_host, trj_dyn_plan** out) {
    if (!ctx || !out) return TRJ_ERR_INVALID;
    *out = nullptr;
    if (nsp < 1 || nsp > 16) return trj_fail(ctx, TRJ_ERR_INVALID, "dyn plan: nsp=%d (1..16)", nsp);
    if (n < 1 || n > (int64_t)INT32_MAX) return trj_fail(ctx, TRJ_ERR_INVALID, "dyn plan: n=%lld", (long long)n);
    if (nbuffer < 1 || nbuffer > 65535 || ndyn < 1 || nbins < 1)
        return trj_fail(ctx, TRJ_ERR_INVALID, "dyn plan: nbuffer=%d ndyn=%d nbins=%d", nbuffer, ndyn, nbins);
    if (nvec < 0 || nvec > (int64_t)INT32_MAX / 2 || (nvec > 0 && (!vec_host || !bin_host)) || !bsc_host)
        return trj_fail(ctx, TRJ_ERR_INVALID, "dyn plan: vectors");
    for (int64_t v = 0; v < nvec; ++v)
        if (bin_host[v] < 0 || bin_host[v] >= nbins)
            return trj_fail(ctx, TRJ_ERR_INVALID, "dyn plan: vector %lld has bin %d outside 0..%d", (long long)v,
                            bin_host[v], nbins - 1);
    trj_dyn_plan* p = new trj_dyn_plan();
    p->ctx = ctx;
    p->nsp = nsp;
    p->n = n;
    p->nbuf = nbuffer;
    p->ndyn = ndyn;
    p->nbins = nbins;
    p->nvec = nvec;
    p->gx = (int)std::max<int64_t>(1, (nvec + kDynThreads * kDynVPT - 1) / (kDynThreads * kDynVPT));
    const int64_t target = (int64_t)ctx->sm_count * 8;
    const int64_t by_atoms = std::max<int64_t>(1, n / kDynChunk);
    p->nsplit_rho = (int)std::min<int64_t>(by_atoms, std::max<int64_t>(1, (target + p->gx - 1) / p->gx));
    // self-term partial rows (splits x buffers): enough for every buffer to split as far as the atoms
    // allow, within 256 MB of partials
    const int64_t split_max = std::min<int64_t>(by_atoms, target);
    const int64_t rows_budget = std::max<int64_t>(nbuffer, ((int64_t)256 << 20) / (8 * std::max<int64_t>(nvec, 1)));
    p->nsplit_cap = (int)std::min<int64_t>((int64_t)nbuffer * split_max, std::max<int64_t>(rows_budget, nbuffer));
    std::vector<int32_t> start(nbins + 1, 0), bv(nvec);
    for (int64_t v = 0; v < nvec; ++v) start[bin_host[v] + 1] += 1;
    // Slots: vectors by the component of one axis, padded so that no thread's vectors differ in it, for the axis
    // that needs the least padding; in the caller's order where that is more than 6 % (the phase's first product
    // is then formed per vector).
    std::vector<int4> slots;
    {
        int best = -1;
        int64_t best_n = nvec + nvec / 16 + kDynVPT;
        for (int ax = 0; ax < 3; ++ax) {
            const int64_t total = dyn_axis_slots(vec_host, nvec, ax);
            if (total < best_n) {
                best_n = total;
                best = ax;
            }
        }
        const int ax = best >= 0 ? best : 0, a1 = ax == 0 ? 1 : 0, a2 = ax == 2 ? 1 : 2;
        p->slots.axis = ax;
        p->slots.shared = best >= 0;
        const std::vector<int64_t> order = dyn_axis_order(vec_host, nvec, best);
        slots.reserve((size_t)best_n);
        auto pad = [&](int c) {
            while (slots.size() % kDynVPT) slots.push_back(make_int4(c, 0, 0, -1));
        };
        for (int64_t i = 0; i < nvec; ++i) {
            const int32_t* v = vec_host + 3 * order[i];
            if (best >= 0 && !slots.empty() && slots.back().x != v[ax]) pad(slots.back().x);
            slots.push_back(make_int4(v[ax], v[a1], v[a2], (int)order[i]));
        }
        if (!slots.empty()) pad(slots.back().x);
    }
    p->slots.n = (int64_t)slots.size();
    // block size with the fewest idle threads
    for (int t = kDynThreads; t >= kDynThreads / 2; t -= 32) {
        const int64_t quads = p->slots.n / kDynVPT, blocks = std::max<int64_t>(1, (quads + t - 1) / t);
        if (t == kDynThreads || blocks * t < (int64_t)p->gslot * p->tslot) {
            p->gslot = (int)blocks;
            p->tslot = t;
        }
    }
    p->parts_rho = dyn_parts(p, (int64_t)p->gslot * p->nsplit_rho, p->nsplit_rho, 16 * p->slots.n * p->nsplit_rho);
    int64_t self_rows = 0;  // of every job together, the most for any number of jobs
    for (int nj = 1; nj <= nbuffer; ++nj) {
        const int ns = self_split(p, nj);
        self_rows = std::max<int64_t>(self_rows, (int64_t)nj * ns * dyn_parts(p, (int64_t)p->gslot * ns * nj, ns,
                                                                              8 * p->slots.n * ns * nj));
    }
    for (int b = 0; b < nbins; ++b) start[b + 1] += start[b];
    {
        std::vector<int32_t> fill(start.begin(), start.end() - 1);
        for (int64_t v = 0; v < nvec; ++v) bv[fill[bin_host[v]]++] = (int32_t)v;
    }
    trj_device_guard g(ctx->device);
    const int msd_blocks = (int)((n + kDynThreads - 1) / kDynThreads);
    const int64_t rows = (int64_t)nbuffer * ndyn;
    dyn_want(p, &p->slot_dev, slots.size());
    dyn_want(p, &p->bin_start, nbins + 1);
    dyn_want(p, &p->bin_vec, nvec);
    dyn_want(p, &p->bsc, nsp);
    dyn_want(p, &p->u, n);
    dyn_want(p, &p->u0, (size_t)nbuffer * n);
    dyn_want(p, &p->r0, (size_t)nbuffer * n);
    dyn_want(p, &p->rt, (size_t)nbuffer * n);
    dyn_want(p, &p->rho_part, (size_t)p->nsplit_rho * p->parts_rho * slots.size());
    dyn_want(p, &p->rho_t, nvec);
    dyn_want(p, &p->rho0, (size_t)nbuffer * nvec);
    dyn_want(p, &p->self_part, (size_t)self_rows * slots.size());
    dyn_want(p, &p->self, (size_t)nbuffer * nvec);
    dyn_want(p, &p->msd_part, (size_t)nbuffer * msd_blocks);
    dyn_want(p, &p->fc, (size_t)rows * nbins);
    dyn_want(p, &p->fs, (size_t)rows * nbins);
    dyn_want(p, &p->msd, rows);
    dyn_want(p, &p->jobs_dev, nbuffer);
    dyn_want(p, &p->done_dev, nbuffer);
    if (!dyn_alloc_all(p)) {
        dyn_free(p);
        delete p;
        return trj_fail(ctx, TRJ_ERR_NOMEM, "dyn plan: device allocation failed (nbuffer=%d, n=%lld)", nbuffer,
                        (long long)n);
    }
    cudaError_t e = cudaSuccess;
    if (nvec) {
        e = cudaMemcpy(p->slot_dev, slots.data(), sizeof(int4) * slots.size(), cudaMemcpyHostToDevice);
        p->slots.slot = p->slot_dev;
        if (e == cudaSuccess) e = cudaMemcpy(p->bin_vec, bv.data(), sizeof(int32_t) * nvec, cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess)
        e = cudaMemcpy(p->bin_start, start.data(), sizeof(int32_t) * (nbins + 1), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p->bsc, bsc_host, sizeof(float) * nsp, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(p->fc, 0, sizeof(double) * rows * nbins);
    if (e == cudaSuccess) e = cudaMemset(p->fs, 0, sizeof(double) * rows * nbins);
    if (e == cudaSuccess) e = cudaMemset(p->msd, 0, sizeof(double) * rows);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        dyn_free(p);
        delete p;
        return trj_fail(ctx, TRJ_ERR_CUDA, "dyn plan: %s", cudaGetErrorString(e));
    }
    *out = p;
    return TRJ_OK;
}

extern "C" int trj_dyn_plan_info(const trj_dyn_plan* p, int64_t* scratch_bytes) {
    if (!p) return TRJ_ERR_INVALID;
    if (scratch_bytes) *scratch_bytes = p->scratch_bytes;
    return TRJ_OK;
}

extern "C" int trj_dyn_accumulate(trj_dyn_plan* p, const float* packed_dev, int64_t n, const float box[3],
                                  const int32_t* lag_host, const uint8_t* origin_host, void* stream) {
    if (!p) return TRJ_ERR_INVALID;
    trj_ctx* ctx = p->ctx;
    if (!box || !lag_host || !origin_host) return trj_fail(ctx, TRJ_ERR_INVALID, "dyn accumulate: null argument");
    if (n != p->n)
        return trj_fail(ctx, TRJ_ERR_INVALID, "dyn accumulate: n=%lld, plan made for %lld atoms", (long long)n,
                        (long long)p->n);
    if (!packed_dev || ((uintptr_t)packed_dev) % 16)
        return trj_fail(ctx, TRJ_ERR_INVALID, "dyn accumulate: packed_dev null or not 16-byte aligned");
    if (!(box[0] > 0.f && box[1] > 0.f && box[2] > 0.f))
        return trj_fail(ctx, TRJ_ERR_INVALID, "dyn accumulate: box edges must be positive");
    std::vector<DynJob> jobs;
    for (int b = 0; b < p->nbuf; ++b) {
        const int lag = lag_host[b];
        if (lag < 0) continue;
        if (lag >= p->ndyn)
            return trj_fail(ctx, TRJ_ERR_INVALID, "dyn accumulate: buffer %d lag %d outside 0..%d", b, lag,
                            p->ndyn - 1);
        if (origin_host[b] && lag != 0)
            return trj_fail(ctx, TRJ_ERR_INVALID, "dyn accumulate: buffer %d starts at lag %d (must be 0)", b, lag);
        jobs.push_back(DynJob{b, lag, origin_host[b] ? 1 : 0, 0});
    }
    if (jobs.empty()) return TRJ_OK;
    trj_device_guard g(ctx->device);
    cudaStream_t s = (cudaStream_t)stream;
    const int nj = (int)jobs.size();
    // pageable source: the call returns after the bytes are staged, so the vector may go out of scope
    TRJ_CUDA_TRY(ctx, cudaMemcpyAsync(p->jobs_dev, jobs.data(), sizeof(DynJob) * nj, cudaMemcpyHostToDevice, s));
    const unsigned nb = (unsigned)((n + kDynThreads - 1) / kDynThreads);
    dyn_phase_kernel<<<nb, kDynThreads, 0, s>>>((const float4*)packed_dev, n, (double)box[0], (double)box[1],
                                                 (double)box[2], p->u);
    int launches = 1;
    if (p->nvec > 0) {
        const int rows = p->nsplit_rho * p->parts_rho;
        (p->slots.shared ? dyn_rho_kernel<true> : dyn_rho_kernel<false>)<<<dim3(p->gslot, rows), p->tslot, 0, s>>>(
            p->u, n, p->bsc, p->nsp, p->slots, p->nsplit_rho, p->parts_rho, p->rho_part);
        dyn_rho_gather_kernel<<<(unsigned)((p->slots.n + 31) / 32), 256, 0, s>>>(p->rho_part, p->slot_dev, p->slots.n, p->nvec, rows, p->jobs_dev, nj,
                                                 p->rho_t, p->rho0);
        launches += 2;
    }
    dyn_origin_kernel<<<dim3(nb, nj), kDynThreads, 0, s>>>((const float4*)packed_dev, p->u, n, p->jobs_dev, p->u0,
                                                          p->r0, p->rt);
    dyn_msd_kernel<<<dim3(nb, nj), kDynThreads, 0, s>>>((const float4*)packed_dev, n, box[0], box[1], box[2],
                                                       p->jobs_dev, p->r0, p->rt, p->msd_part);
    launches += 2;
    if (p->nvec > 0) {
        const int nsplit = self_split(p, nj);
        const int parts = dyn_parts(p, (int64_t)p->gslot * nsplit * nj, nsplit, 8 * p->slots.n * nsplit * nj);
        const int rows = nsplit * parts;
        p->timer.begin(ctx, s);
        (p->slots.shared ? dyn_self_kernel<true> : dyn_self_kernel<false>)<<<dim3(p->gslot, rows, nj), p->tslot, 0, s>>>(
            p->u, p->u0, n, p->jobs_dev, p->slots, nsplit, parts, p->self_part);
        p->timer.end(ctx, s);
        dyn_self_gather_kernel<<<dim3((unsigned)((p->slots.n + 255) / 256), nj), 256, 0, s>>>(
            p->self_part, p->slot_dev, p->slots.n, p->nvec, rows, p->self);
        launches += 2;
    }
    dyn_reduce_kernel<<<dim3(p->nbins, nj), kDynThreads, 0, s>>>(p->self, p->rho_t, p->rho0, p->bin_start, p->bin_vec,
                                                                 p->nvec, p->nbins, p->ndyn, p->jobs_dev, p->msd_part,
                                                                 (int)nb, n, p->fc, p->fs, p->msd);
    launches += 1;
    ctx->launches += launches;
    TRJ_CUDA_TRY(ctx, cudaGetLastError());
    return TRJ_OK;
}

extern "C" int trj_dyn_flush(trj_dyn_plan* p, const uint8_t* done_host, double* fkt_dev, double* fskt_dev,
                             double* r2t_dev, void* stream) {
    if (!p) return TRJ_ERR_INVALID;
    trj_ctx* ctx = p->ctx;
    if (!done_host || !fkt_dev || !fskt_dev || !r2t_dev)
        return trj_fail(ctx, TRJ_ERR_INVALID, "dyn flush: null argument");
    std::vector<int32_t> done;
    for (int b = 0; b < p->nbuf; ++b)
        if (done_host[b]) done.push_back(b);
    if (done.empty()) return TRJ_OK;
    trj_device_guard g(ctx->device);
    cudaStream_t s = (cudaStream_t)stream;
    TRJ_CUDA_TRY(ctx, cudaMemcpyAsync(p->done_dev, done.data(), sizeof(int32_t) * done.size(), cudaMemcpyHostToDevice,
                                      s));
    const int64_t rows = std::max<int64_t>((int64_t)p->ndyn * p->nbins, p->ndyn);
    dyn_flush_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, s>>>(p->done_dev, (int)done.size(), p->ndyn, p->nbins,
                                                                   p->fc, p->fs, p->msd, fkt_dev, fskt_dev, r2t_dev);
    ctx->launches += 1;
    TRJ_CUDA_TRY(ctx, cudaGetLastError());
    return TRJ_OK;
}

extern "C" int trj_dyn_kernel_ms(trj_dyn_plan* p, float* ms) {
    if (!p) return TRJ_ERR_INVALID;
    return p->timer.elapsed(p->ctx, ms);
}

extern "C" int trj_dyn_plan_destroy(trj_dyn_plan* p) {
    if (!p) return TRJ_OK;
    dyn_free(p);
    delete p;
    return TRJ_OK;
}
