// What the PCG's kernels share: the preconditioner as they read it, and the
// one-launch loop of small systems.
#pragma once
#include "b2s_internal.cuh"

namespace b2s
{
struct MasView
{
    int            active;  // MAS present
    int            off, vn;
    int            abd_off, abd_n;  // affine-body range: block rows abd_off .. abd_off + 4 abd_n
    const double*  abd_inv;         // [abd_n * 144]
    const int32_t* r2p;
    const int32_t* node1;  // [vn] level-1 node of each vertex (global slot)
    const int4*    anc;    // per level-1 node: its ancestors' slots (-1: none)
    int            begin1;  // first level-1 slot
    int            T;      // coarse levels (L-1)
    const float*   Z;      // node values by slot
    // rows in PCG order (null: the matrix's own order)
    const int32_t* row_of;
    const int32_t* pos;  // its inverse
    const int32_t* slot_node1;  // [slots]
    int            slots;
};

MasView mas_view(b2s_solver* s);

// One launch for up to `iterations` PCG iterations (b2s_pcg_small.cu): A and
// the vectors in PCG order with the MAS (`ord`), r, p and x set by the caller,
// Ap zero, the scalars in s->pcg.sc (read and written back). The launch returns
// false, with nothing done, when the device refuses it (fewer SMs than the
// device has: a shared or partitioned GPU) or has no room for its sums: the
// caller launches step by step.
bool pcg_small_fits(b2s_solver* s, const Matrix& A, int kind, bool ord, bool f32);
bool pcg_small_launch(b2s_solver* s, const Matrix& A, int kind, long long iterations, double* x);
bool pcg_small_launch_f32(b2s_solver* s, const Matrix& A, int kind, long long iterations, double* x);
}  // namespace b2s
