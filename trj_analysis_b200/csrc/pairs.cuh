// pairs.cuh -- geometry of one frame's pair histogram, filled on the host (rdf.cu) for the cell-pair kernel and
// for the items of a fused launch.
#pragma once
#include <stdint.h>

constexpr int kMaxOffsets = 14;  // half-shell stencil with the cell itself

// What one pair's test and bin need.
struct PairGeom {
    float L[3];
    float inv_L[3];
    float h1[3], h2[3];         // |dx| < h1: nint(dx/L) = 0; h1 <= |dx| < h2: +-1; else the division
    float side2, side2_lo, side2_hi;
    float side2_win;            // side2_hi - side2, the larger half of that window
    float deltar, inv_deltar;
    float edge_thr;             // distance of q from the nearest integer above which a bin edge may be near
    int lsmax, nsp;
    int floor_bins;             // 0: bin nint(r/deltar) (reference); 1: bin floor(r/deltar)+1
    int row_words;              // words of a shared histogram row: lsmax + 2 (first and last: not counted)
    int want_edge;              // edge statistics are collected
    float one;                  // 1.0f, from the host: not a constant the assembler could fold
};

// Division of n < 2^31 by a launch constant: n * ceil(2^(31+l) / d) >> (31+l), l = ceil(log2 d).
struct FastDiv {
    unsigned d, mul;
    int shift;
};
struct RdfParams {
    PairGeom g;
    int nit;
    int nc[3];                  // cells per axis (1: the axis is not split)
    int sub[3], nsub;           // groups per cell: sub[0] x sub[1] x sub[2] boxes, z fastest
    float inv_sub[3];           // 1 / sub
    float edge[3];              // cell edge
    float half[3];              // half edge of a group's box, with the cull pad
    FastDiv div_nsub, div_nc1, div_nc2, div_nseg;
    // A home group's neighbour list: its own cell's groups at distance 0 .. nsub / 2 after it (cyclically, so
    // that every group has the same share), then all groups of each further stencil cell.
    int nself, list;            // entries of the own cell, of the list
    int nseg, per_seg;          // segments of the list (one work item each); their length
    int split_all;              // every axis of the geometry is split (in two dimensions: x and y)
    float cull2;                // (cutoff * (1 + 2^-10))^2: neighbours farther from the homes' box are skipped
    float cull_pad;             // added to half-widths: covers the FP32 rounding of the cull test
    long long wait_clocks;      // limit of the stall test's wait
    int stall_test;             // 1: every warp waits on a barrier nothing arrives on (timeout test)
    int off[kMaxOffsets][3];
    unsigned nitems;
};
