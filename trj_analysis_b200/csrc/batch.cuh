// batch.cuh -- descriptors of the fused multi-request launches (trj_batch_*).
//
// A turn packs one frame of each of up to max_items small requests.  The host writes the frames'
// positions and species ids back to back into mapped pinned staging and one BatchItem per frame into
// a pinned table; the launch sequence (table copy, layout count, layout scatter, pair histogram,
// direct sum, shell reduction) is the same for every turn, so one CUDA graph per staging buffer
// replays any mix of requests.  Every kernel walks a global list of work units; an item's units
// start at its *_begin offset (exclusive prefix over the items before it).
#pragma once

#include "pairs.cuh"
#include "trj_common.cuh"

constexpr int kBatchChunk = 1024;        // atoms per layout unit
constexpr int kBatchThreads = 256;
constexpr int kBatchMaxSpecies = 16;
constexpr int kBatchMaxHistWords = 24576;  // largest pair histogram of a batch
constexpr int kBatchCounters = 2;        // dynamic work counters: direct sum, reduction

struct __align__(16) BatchItem {
    // frame: atoms [atom_off, atom_off + n) of the staging and device arrays
    int64_t atom_off;
    int32_t n, nsp;
    float L[3];
    int32_t nchunk;                      // layout units: ceil(n / kBatchChunk)
    int32_t square;                      // pair rows by ordered species pair (else by ind_ij through a table)
    int64_t sp_off[kBatchMaxSpecies + 1];  // species offsets of the S(Q) plan within the frame
    // pair histogram (the rdf plan's geometry after the per-frame clip); pair.nitems work items
    RdfParams pair;
    unsigned long long* hist;            // [nit][lsmax] accumulator, null: no pair plan
    unsigned long long* edge;            // edge counters (ulp, fma, counted) or null
    // S(Q) direct sum over the plan's vectors (the plain method of trj_sq_accumulate)
    const int4* vecs;
    const int32_t* subset;
    const double* w;
    const int32_t* bin_start;
    const int64_t* sp_off_dev;
    double2* part;                       // [nsplit * parts][nsp][nvec]
    double2* rho;                        // [nsp][nvec]
    double* out;                         // [nbins][nit] accumulator
    int32_t nvec, nsplit, vpt, nbins;
    int32_t nvblk;                       // vector blocks of the direct sum
    int32_t parts, tv, tg;               // rest of its shape (sq.cu PlainShape)
    // first work unit of the item in each kernel's list
    int64_t chunk_begin, pair_begin, sq_begin, red_begin;
    int64_t key_begin;                   // first group of the item in the sort's arrays: a multiple of 32
};

struct __align__(16) BatchHeader {
    unsigned long long counter[kBatchCounters];  // zero in every turn's copy of the table
    int32_t nitems, pad0;
    int64_t total_chunk, total_pair, total_sq, total_red, total_atoms, total_key;
    int64_t pad1[1];
};
static_assert(sizeof(BatchHeader) % 16 == 0, "table alignment");
static_assert(sizeof(BatchItem) % 16 == 0, "table alignment");

// Item of work unit u: the last item whose begin offset (member `field` of BatchItem) is <= u.  Called by whole
// warps: every lane looks at one of 32 items an equal step apart, so that a table of 4,096 items takes three loads
// that wait for one another instead of twelve (1,000 frames of 50 atoms: 142 -> 131 us).
template <int64_t BatchItem::*field>
__device__ __forceinline__ int batch_item_of(const BatchItem* __restrict__ items, int nitems, int64_t u) {
    const int lane = (int)(threadIdx.x & 31u);
    int lo = 0, n = nitems;
    while (n > 1) {
        const int step = (n + 31) / 32, at = lane * step;
        const unsigned le = __ballot_sync(0xffffffffu, lane == 0 || (at < n && items[lo + at].*field <= u));
        const int k = 31 - __clz(le);
        lo += k * step;
        n = min(step, n - k * step);
    }
    return lo;
}

// Device arrays of the turn's cell sort.  Zeroed together at the start of a turn's pair work: state (per item:
// pair work counter, frame flags, atoms placed, rounds of homes), fcount and cflag.
struct BatchSort {
    unsigned* state;
    int32_t *fcount, *cflag, *fstart;    // per group (cflag: per cell), an item's at its key_begin
    int4* rounds;                        // per round of homes, an item's at batch_rounds_begin
    int32_t *akey, *aslot;               // per atom
    float4* sorted;                      // per atom: an item's atoms by group
};

// First round of homes of an item: its groups' ceil(atoms / 32) add up to at most its groups + n / 32.
__host__ __device__ inline int64_t batch_rounds_begin(const BatchItem& it) { return it.key_begin + it.atom_off / 32; }

// Most groups of an item of n atoms (choose_groups keeps to it), and the shared-memory words of the pair kernel's
// bin rows: triangular rows always fit (hist_words plus two words for each of up to 136 rows), square rows are
// taken where they do.
inline int64_t batch_keys_most(int64_t n) { return n / 8 + 64; }
__host__ __device__ inline int batch_hist_smem_words(int hist_words) { return 2 * hist_words + 272; }

// Kernel launchers of the fused turn, each defined beside the single-request kernels whose
// arithmetic it shares.  grid: CTAs of the fixed-size launch.
void trj_batch_launch_layout(const BatchHeader* hdr, const BatchItem* items, const float* xyz_staged,
                             const int32_t* sp_staged, float4* raw, int32_t* chunk_counts, float4* packed,
                             uint4* phase, unsigned* status, int grid, cudaStream_t s);        // ctx.cu
int trj_batch_launch_pairs(BatchHeader* hdr, const BatchItem* items, const float4* packed, const BatchSort& st,
                           size_t zero_bytes, int hist_words, int grid_layout, int grid, cudaStream_t s);  // rdf.cu
size_t trj_batch_pairs_smem(int hist_words);                                                  // rdf.cu
int trj_batch_pairs_prepare();                                                                // rdf.cu
int trj_batch_pairs_occupancy(int hist_words, int* per_sm);                                   // rdf.cu
void trj_batch_launch_sq(BatchHeader* hdr, const BatchItem* items, const uint4* phase, const float2* turn, int grid_sq,
                         int grid_red, cudaStream_t s);                                       // sq.cu
int trj_batch_sq_occupancy(int* per_sm_sq, int* per_sm_red);                                   // sq.cu
struct trj_rdf_plan;
struct trj_sq_plan;
// Fill the pair part of an item from a plan after the per-frame clip (rdf.cu), and the S(Q) part
// (sq.cu); non-zero: the plan cannot run in a fused launch (the message is on the context).
int trj_batch_fill_rdf(trj_rdf_plan* plan, int64_t n, const float box[3], int hist_words, int max_items, bool want_edge,
                       BatchItem* it, int* nsp, int64_t* nkey);
int trj_batch_fill_sq(trj_sq_plan* plan, int64_t n, BatchItem* it);
