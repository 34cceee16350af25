// batch_tile.cuh — complex64 batches as tile programs (batch_tile.cu).
#pragma once

#include <vector>

#include "plk_internal.cuh"

namespace plk {

struct XOp;
struct ETerm;

// a circuit of a batch, as batch.cu keeps it
struct BatchCircuit {
    int nq;
    const std::vector<XOp> *ops;
    int jac0, ntp;
    const std::vector<ETerm> *terms;
};

struct BatchTiles; // compiled circuits, their device buffers and launch lists

// nullptr (and PLK_OK) when an op is not of this path (dense matrices) or the
// device has no room for the states and programs
int batch_tiles_create(const std::vector<BatchCircuit> &circs, int device, cudaStream_t st, BatchTiles **out);
void batch_tiles_destroy(BatchTiles *t);
// Queues one evaluation: parameters and results on the device; no allocation,
// no host synchronisation, capturable.
int batch_tiles_enqueue(BatchTiles *t, const double *d_params, double *d_expval, double *d_jac, cudaStream_t st);
int batch_tiles_launches(const BatchTiles *t);

} // namespace plk
