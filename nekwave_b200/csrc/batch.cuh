// batch.cuh -- device-side types of the multi-cavity pool (pool.cpp, batch.cu).
#pragma once

#include "nwb_internal.h"

namespace nwb {

constexpr int kBatchThreads = 128;  // block size of the persistent batch kernel
constexpr int kMaxProbes = 8;

// One resident cavity ("slot") as the device sees it.  All pointers are
// sub-allocations of the pool's HBM arena.
struct SlotDev {
    double* u[2];           // ping-pong state [6][stride]
    double* k;              // LSRK register [6][stride]
    const double* D;        // [N*N]
    const double* w3;       // [N^3]
    const ElemGeo* geo;     // [nelt]
    const int* conn;        // [6*nelt]
    double* partial;        // [ntiles] energy partial sums
    double* energy;         // [nsteps+1] energy history (index 0 = initial state)
    double* probes;         // [(nsteps+1) * nprobes * 6] probe history
    const int* probe_elem;  // [nprobes]
    const double* probe_w;  // [nprobes][3][N] tensor-product Lagrange weights
    long long stride;
    double c0, dt;
    double zl[10];          // line coordinates of D (nwb::line_coords)
    int N, nelt, ntiles, epb;
    int nprobes, energy_every;
    int nsteps;             // steps this cavity must take
    int done;               // steps taken
    int par;                // ping-pong parity at the start of the next step
    int active;             // 1 while done < nsteps
    int snel[3], spmask;    // structured box: elements per axis and periodic axes, or 0
    unsigned sdiv[2];       // StageParams::sdiv, sshift
    int sshift[2];
    int oblique;            // diagonal metrics with normals off the axes: launch_batch_oblique's
};

// One tile of work: EPB consecutive elements of one slot.
struct WorkItem {
    int slot;
    int e0;
    int N;
    int tile;  // index of the tile within its slot (energy partial slot)
};

struct BatchShape {
    int ks, epb;
};

// Batch launchers (batch.cu).
// stage: 0..4.  counters[stage] is the dynamic tile counter of that stage.
// dry = 1 runs the stage with a = b = dt = 0 (timing only: u_out = u_in).
cudaError_t launch_batch_stage(int f32, int stage, const SlotDev* slots, const WorkItem* work,
                               const int* ntiles, int* counters, int grid, int smem, int dry,
                               cudaStream_t st);
// Per-N mode: one block per tile of the given N (work points at that N's tiles,
// which must have been cut with batch_epb_n(N, f32) elements each).  Dh: that N's D on
// the host when every resident cavity of that N shares it (lets the kernel take D
// from its parameters), else null.
// form: batch_form_n of that N's resident elements, also when the tiles were cut.
// err: device pointer of the word in which an expired bounded wait is recorded.
cudaError_t launch_batch_stage_n(int N, int f32, int form, int stage, const SlotDev* slots,
                                 const WorkItem* work, int ntiles, int dry, const double* Dh, int* err,
                                 cudaStream_t st);
// The same stage of the oblique slots among the work items [work, work + ntiles) of one N,
// cut with batch_shape(N) elements (those of the other launches leave them out).  A plain
// launch, not an overlapped one: the next stage of that N may overlap it.
cudaError_t launch_batch_oblique(int N, int stage, const SlotDev* slots, const WorkItem* work, int ntiles, int dry,
                                 cudaStream_t st);
// Kernel form of a per-N launch over nelt elements in all (0: the large one), as the
// single solver's default follows its mesh's size; elements per block of a form.
constexpr int kBatchForms = 3;
int batch_form_n(int N, int f32, long long nelt);
int batch_epb_n(int N, int f32, int form);
// Diagnostics after a step (post = 1) or of the initial state (post = 0): energy
// partials per tile of the work items [work, work + ntiles) (ntiles_p, when given: their
// number on the device).  overlap: see launch_overlapped.
cudaError_t launch_batch_diag(SlotDev* slots, const WorkItem* work, int ntiles, const int* ntiles_p, int post,
                              int grid, bool overlap, cudaStream_t st);
// End of step of nslots slots (slot_list[0..nslots), or first_slot..): per-slot energy sum
// (fixed order), probe values, parity flip, step count, completion; resets the stage
// counters (when given).
cudaError_t launch_batch_epilogue(SlotDev* slots, const int* slot_list, int first_slot, int nslots, int post,
                                  int* counters, bool overlap, cudaStream_t st);

// Shape per N used by the batch kernel and its dynamic shared memory need.
BatchShape batch_shape(int N, int f32);
int batch_smem(int N, int f32);
cudaError_t batch_prepare(int f32, int smem);

}  // namespace nwb
