// CG and BiCGStab iterations of systems that fit on chip, as one cooperative
// kernel (resident.cu).
#pragma once

#include "krylov_kernels.cuh"

namespace b2s {

template< typename Real >
struct ResidentVecs
{
   Real *x, *r, *p, *Ap, *z, *r_ast;
   Real *p2, *Ap2;  // scratch: the second copies of p and Ap
   Real *r0, *p0;   // scratch: r and p as they were before the launch
};

// Whether the kernel takes this matrix and solver with values of `es` bytes.
bool resident_fits( const b2s_matrix_t* A, int solver, size_t es );

// The kernel's exchange slots, allocated and emptied.
b2s_status resident_scratch_init( DevBuf& scratch, cudaStream_t s );

// At most `iterations` iterations of `solver` (B2S_CG or B2S_BICGSTAB) from the
// state in `v` and `ctl`, which are left as the kernels of krylov.cu leave
// them: p is the next direction unless ctl->done. BiCGStab ends early with
// ctl->restart_flag set, before the direction update, when r has become too
// orthogonal to r_ast (eps2: its threshold). ctl->gave_up: a wait of `looks`
// polls (0: the default) ran out, as when another kernel keeps some of the
// blocks off the device; then x and *ctl are as before the launch, r0 and p0
// hold r and p, and the slots have to be initialised again.
template< typename Real >
b2s_status resident_iterate( const b2s_matrix_t* A, int solver, const Real* vals, const Real* diag,
                             const ResidentVecs< Real >& v, Ctl* ctl, DevBuf& scratch, int iterations, int looks,
                             double eps2, cudaStream_t s );

}  // namespace b2s
