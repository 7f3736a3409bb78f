// Resident step forms: LPs whose matrix fits in the shared memory of one
// thread-block cluster, or of all SMs (see resident.cu).
#pragma once

#include <vector>

#include "gridsync.cuh"
#include "mixed.h"

namespace sihg {

// Passes of one side held by one block (32 / L segments of L lanes each) and
// where its share of the layout lies.
struct ResSide {
    int pass_begin, passes;  // in the pass table
    int row_begin, rows;     // pairs of entries of 32 lanes
    int locals;              // segments of the side this block owns
};

struct ResBlock {
    ResSide side[2];  // 0 rows of A (A x), 1 columns (A^T y)
};

// Where a block keeps what, in bytes of dynamic shared memory; the same in
// every block of a launch.
struct ResSmem {
    int pass[2], rows[2], xs, ys, col, row, seg, red, eval, locals[2], total;
};

struct ResArgs {
    const ResBlock* blocks;  // [instances x cluster]
    const int4* inst;        // {first column, columns, first row, rows} of each instance
    // pass: {first pair in its block, width | log2 L << 24, first segment in the
    // instance, first local segment | segments << 24}; a pass of width w holds
    // (w + 1) / 2 pairs per lane
    const int4* passes;
    const char* rows;        // the pairs (Compact or Wide, see resident.cu), indices in the instance
    ResSmem sm;
    int cluster;
};

struct PlainVecs;   // plain.h
struct PlainState;

class ResidentPlan {
  public:
    // kCluster: a cluster per instance; kGrid: one LP over every SM; kPlain: the
    // plain algorithm of one LP on a cluster.
    enum Kind { kCluster, kGrid, kPlain };
    // Plans the form for these instances (segment pointers of the batch, lanes
    // per segment of both sides); ready() says whether they fit.  most_us > 0: a
    // batch whose clusters take turns is left out where a step is estimated to
    // take longer.
    int build(const std::vector<int>& csr_ptr, const std::vector<int>& csc_ptr, const std::vector<int>& roff,
              const std::vector<int>& coff, const std::vector<uint8_t>& row_lanes,
              const std::vector<uint8_t>& col_lanes, int sm_count, cudaStream_t s, Kind kind, double most_us = 0.0);
    // Copies the scaled entries into the layout.
    int fill(const SegMatrix& rows_A, const SegMatrix& cols_A, cudaStream_t s);
    // `periods` times nsteps steps and an evaluation of every running instance.
    int launch(int nsteps, int periods, const Vecs& V, Inst* st, unsigned* done_count, cudaStream_t s) const;
    // Start of a run: the grid form's barriers count from zero.
    int reset(cudaStream_t s);
    // The same for kGrid (cooperative launch; `records`: 2 N column records; gb:
    // status word and limit of the barrier waits).  SIH_PDHG_ERR_UNSUPPORTED:
    // the grid does not fit on the device now, nothing was launched.
    int launch_grid(int nsteps, int periods, const Vecs& V, Inst* st, unsigned* done_count, float4* records, int N,
                    const GridBar& gb, cudaStream_t s) const;
    // `checks` times `iterations` iterations and a check of the plain algorithm.
    int launch_plain(int iterations, int checks, const PlainVecs& v, PlainState* st, cudaStream_t s) const;
    bool ready() const { return ready_; }
    Kind kind() const { return kind_; }
    int grid() const { return args_.cluster * instances_; }
    void release();

  private:
    cudaLaunchConfig_t config(cudaLaunchAttribute* at, cudaStream_t s) const;
    bool ready_ = false;
    Kind kind_ = kCluster;
    int instances_ = 0, threads_ = 0, npass_ = 0;
    ResArgs args_{};
    DevMem tab_, rows_, slots_, esums_;
};

}  // namespace sihg
