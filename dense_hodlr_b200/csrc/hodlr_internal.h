// Internal structures shared by the kernels and the host orchestration.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "kfun.h"

// Where a matrix entry comes from: a kernel of point coordinates, or a
// dense column-major matrix resident in HBM.
struct EntrySrc {
  const double* pts;  // SoA coordinates, pts[d * ld + i]
  const double* A;    // dense input, A[i + j * ld]
  int64_t ld;         // = n
  hx_kparams kp;
  int dense;
  // forest of independent systems: kernel of system psys[i] (null for one system)
  const hx_kparams* kps;
  const int* psys;
};

// ----------------------------------------------------------------- ACA
enum {
  ACA_RUNNING = 0,   // loop in progress (or not started)
  ACA_POST = 1,      // loop finished, post-processing pending
  ACA_DONE = 2,      // W, V and rank final
  ACA_NEED_CAP = 3,  // loop paused: more columns of W/V are needed
  ACA_ERROR = 4,
  ACA_NEED_CAP_POST = 5,  // loop done; the full-rank form needs more columns
  ACA_PAUSED = 6,         // loop paused for another share of the CTAs
};

// One off-diagonal block.  W and V point at the block's first row inside the
// level arenas (leading dimension = N), so W(i,l) = W[i + l*N] for the block's
// local row i, and V(j,l) = V[j + l*N] for its local column j.
struct AcaState;

struct AcaBlock {
  AcaState* st;       // loop state of this block
  double* W;
  double* V;
  unsigned char* cR;  // chosen rows, local index
  unsigned char* cC;  // chosen columns, local index
  int* prow;          // pivot row of step t, local index
  int* pcol;          // pivot column of step t
  int r0, c0, m, n;
  int kcap;           // columns available in W and V
  int kstop;          // aca_group_kernel: columns at which the block pauses
  int level;
  int g0, G;          // with a CTA table: first CTA of this block's group, group size
  // aca_group_kernel: the block's slices of W and V in the launch's working
  // layout, doubles from one CTA's to the next
  double *sW, *sV;
  int64_t strW, strV;
  int minRank, maxRank;  // the node's rank bounds for this block (-1: none)
};

// Loop state of one block; lets a paused block resume where it stopped.
struct AcaState {
  double frob2, eps, margin;
  double swp, svp;  // |w_{k-1}|^2, |v_{k-1}|^2 while epsilon_{k-1} is pending
  int k, cur, status, iters, rank, near;
  int pending;      // 1: epsilon of step k-1 not evaluated yet
  int pad;
};

struct AcaLaunch {
  const AcaBlock* blocks;
  int nblocks;
  int G;                 // CTAs per block
  int64_t ld;            // N
  double tol, minPivot;
  int kcap_max;          // largest kcap among the launch's blocks (shared memory rows)
  double* part;          // per-CTA partials, part_stride doubles each
  int64_t part_stride;
  unsigned* bar;         // per-block barrier counters (zeroed before launch)
  unsigned* err;         // device error word
  EntrySrc src;
  const int* cta_block;  // CTA -> block (groups of uneven size, AcaBlock::g0/G), or null
  int ncta;              // CTAs of the launch when cta_block is set
  double* dotg;          // per-CTA per-warp dot partials in global memory (large ranks), or null
  int64_t dotg_stride;   // doubles per CTA in dotg (NT/32 * kcap_max)
  int narrow;            // 1 (aca_kernel with 256 threads): 2 elements per thread, 512-row chunks
  unsigned spin_limit;   // polls of a group barrier before it gives up (DEV_ERR_TIMEOUT)
  unsigned bar_extra;    // arrivals a group barrier waits for beyond its G CTAs (0; 1 makes
                         // every barrier unreachable, to exercise the timeout path)
  // aca_group_kernel: ring stages, doubles of a stage (a tile's columns of the
  // largest chunk), and the exchange slots (128 bytes a CTA, zeroed before launch)
  int ring_stages, stage_elems;
  unsigned char* slots;
  // rows published for the next pass: two per CTA of pub_stride bytes (16 a
  // column), tagged with this launch's number and the exchange's
  unsigned char* pub;
  int64_t pub_stride;
  unsigned launch_tag;
  // CTAs of the launch that ran out of work so far (zeroed before launch); once
  // there are yield_at (0: never) the blocks still running pause
  unsigned* idle;
  int yield_at;
};
