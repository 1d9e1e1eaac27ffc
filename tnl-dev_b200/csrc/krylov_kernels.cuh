// Device side of the Krylov solvers: the control block (TNL's IterativeSolver
// state, Solvers/IterativeSolver.hpp:98-146, kept in device memory), the
// SpMV sinks that fuse each solver's dot products into the SpMV epilogue, and
// the fused vector kernels.
#pragma once

#include "spmv_kernels.cuh"

#include <type_traits>
#include <utility>

namespace b2s {

// Control block of one solve. Every kernel of an iteration first reads
// `done`; the deciding scalar work runs in the last block of the kernel that
// completes a reduction ("finisher").
struct Ctl
{
   // IterativeSolver
   double residue, tol, div_tol;
   long long it, maxit, minit;
   int done;       // no more work in this solve
   int reason;     // 0 running, 1 converged/stopped by check, 2 zero curvature, 3 breakdown
   int gave_up;    // a bounded wait between the resident kernel's blocks ran out
   // shared scalars
   double normb;
   // CG
   double s1, s2, alpha, beta;
   // BiCGStab
   double rho, rho_old, r_ast_sqnorm, omega, bi_alpha, bi_beta;
   int restart_flag;
   // GMRES
   double gm_beta, normw, beta_old;
   int cycle_stop;     // Arnoldi loop of the current cycle ended early
   int o_steps;        // steps of the current cycle that completed
   int m;              // restart length of the current cycle
   // TFQMR
   double tf_tau, tf_theta, tf_eta, tf_alpha, tf_rho, tf_beta;
   // BiCGStab(ell)
   double bl_rho0, bl_rho1, bl_alpha, bl_beta, bl_omega, bl_sigma0;
   // refinement (mixed precision)
   double outer_norm, outer_res;
   // reliable updates (mixed precision): (r, z) of the iteration before the last one
   double s1_prev;
};

// checkNextIteration (IterativeSolver.hpp:108-118)
__device__ __forceinline__ bool
check_next( const Ctl& c )
{
   if( isnan( c.residue ) || c.it > c.maxit || ( c.residue > c.div_tol && c.it >= c.minit )
       || ( c.residue < c.tol && c.it >= c.minit ) )
      return false;
   return true;
}

// nextIteration (IterativeSolver.hpp:98-106): check, then count the iteration.
__device__ __forceinline__ void
next_iteration( Ctl& c )
{
   const bool go = check_next( c );
   c.it++;
   if( ! go ) {
      c.done = 1;
      c.reason = 1;
   }
}

// ---------------------------------------------------------------------------
// Four consecutive vector elements as one 16-byte (FP32) or one 32-byte (FP64,
// sm_100's 256-bit global access) access; solver vectors live in global memory
// and start on 256-byte boundaries, so every access of four elements at an
// index that is a multiple of 4 is aligned.
template< typename Real >
struct V4
{
   Real v[ 4 ];
};
__device__ __forceinline__ V4< float >
ld4( const float* p )
{
   const float4 a = *reinterpret_cast< const float4* >( p );
   return { { a.x, a.y, a.z, a.w } };
}
__device__ __forceinline__ V4< double >
ld4( const double* p )
{
   V4< double > r;
   asm volatile( "ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"( r.v[ 0 ] ), "=d"( r.v[ 1 ] ), "=d"( r.v[ 2 ] ), "=d"( r.v[ 3 ] )
                 : "l"( p )
                 : "memory" );
   return r;
}
__device__ __forceinline__ void
st4( float* p, const V4< float >& a )
{
   *reinterpret_cast< float4* >( p ) = make_float4( a.v[ 0 ], a.v[ 1 ], a.v[ 2 ], a.v[ 3 ] );
}
__device__ __forceinline__ void
st4( double* p, const V4< double >& a )
{
   asm volatile( "st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"( p ), "d"( a.v[ 0 ] ), "d"( a.v[ 1 ] ), "d"( a.v[ 2 ] ),
                 "d"( a.v[ 3 ] )
                 : "memory" );
}

// Ops that provide apply4( i, acc ) (i a multiple of 4) run four elements per
// thread step: all loads of the step are issued before any store.
template< class Op, class = void >
struct HasApply4 : std::false_type
{};
template< class Op >
struct HasApply4< Op, decltype( std::declval< const Op& >().apply4( int64_t(), (double*) nullptr ), void() ) >
   : std::true_type
{};

// ---------------------------------------------------------------------------
// Reductions over plain vectors with a finisher functor.
template< typename Real, class Op, class Fin >
__global__ void __launch_bounds__( kReduceBlock )
vec_kernel( int64_t n, Ctl* ctl, Op op, Fin fin, RedScratch rs )
{
   if( ctl->done )
      return;
   op.load( *ctl );
   double acc[ Op::NR ];
#pragma unroll
   for( int k = 0; k < Op::NR; k++ )
      acc[ k ] = 0.0;
   const int64_t t0 = blockIdx.x * (int64_t) kReduceBlock + threadIdx.x, step = (int64_t) gridDim.x * kReduceBlock;
   int64_t tail = 0;
   if constexpr( HasApply4< Op >::value ) {
      const int64_t n4 = n / 4;
      for( int64_t q = t0; q < n4; q += step )
         op.apply4( 4 * q, acc );
      tail = 4 * n4;
   }
   for( int64_t i = tail + t0; i < n; i += step )
      op( i, acc );
   if constexpr( Fin::active ) {
      double tot[ Op::NR ];
      if( grid_reduce< Op::NR, kReduceBlock >( acc, rs, tot ) && threadIdx.x == 0 )
         fin( *ctl, tot );
   }
}

struct NoFin
{
   static constexpr bool active = false;
   __device__ void operator()( Ctl&, const double* ) const {}
};

// ---------------------------------------------------------------------------
// SpMV sinks (y = A x row results) with solver-specific epilogues.
// All of them skip their kernel when ctl->done (checked by the SpMV wrapper).

// r = b - s ; [z = r / diag] ; p = z or r ; acc += (r, z) or (r, r)
// CG initialisation (CG.hpp:37-58).
template< typename Real >
struct CgInitSink
{
   static constexpr int NR = 1;
   const Real* b;
   Real *r, *z, *p;
   const Real* diag;
   Ctl* ctl;
   __device__ __forceinline__ void
   put( int row, Real s, double* acc ) const
   {
      const Real rr = b[ row ] - s;
      r[ row ] = rr;
      Real zz = rr;
      if( diag ) {
         zz = rr / diag[ row ];
         z[ row ] = zz;
      }
      p[ row ] = zz;
      acc[ 0 ] += (double) rr * (double) zz;
   }
   __device__ void
   finish( const double* t ) const
   {
      Ctl& c = *ctl;
      c.s1 = t[ 0 ];
      c.it = 0;
      c.residue = sqrt( c.s1 ) / c.normb;
      next_iteration( c );
   }
};

// Ap = A p ; acc += (Ap, p)  ->  alpha = s1 / s2 (CG.hpp:60-73)
template< typename Real >
struct CgApSink
{
   static constexpr int NR = 1;
   Real* Ap;
   const Real* p;
   Ctl* ctl;
   __device__ __forceinline__ void
   put( int row, Real s, double* acc ) const
   {
      Ap[ row ] = s;
      acc[ 0 ] += (double) s * (double) p[ row ];
   }
   __device__ void
   finish( const double* t ) const
   {
      Ctl& c = *ctl;
      c.s2 = t[ 0 ];
      if( c.s2 == 0.0 ) {
         // p = 0 => r = 0: the solution has been reached (CG.hpp:64-67)
         c.residue = 0.0;
         c.done = 1;
         c.reason = 2;
         return;
      }
      c.alpha = c.s1 / c.s2;
   }
};

// x += alpha p ; r -= alpha Ap ; [z = r/diag] ; acc += (r,z) or (r,r)
// -> beta, residue, next iteration (CG.hpp:75-101)
template< typename Real >
struct CgUpdateOp
{
   static constexpr int NR = 1;
   Real *x, *r, *z;
   const Real *p, *Ap, *diag;
   Real alpha;
   __device__ __forceinline__ void load( const Ctl& c ) { alpha = (Real) c.alpha; }
   __device__ __forceinline__ void
   operator()( int64_t i, double* acc ) const
   {
      x[ i ] += alpha * p[ i ];
      const Real rr = r[ i ] - alpha * Ap[ i ];
      r[ i ] = rr;
      Real zz = rr;
      if( diag ) {
         zz = rr / diag[ i ];
         z[ i ] = zz;
      }
      acc[ 0 ] += (double) rr * (double) zz;
   }
   __device__ __forceinline__ void
   apply4( int64_t i, double* acc ) const
   {
      V4< Real > X = ld4( x + i ), P = ld4( p + i ), R = ld4( r + i ), AP = ld4( Ap + i ), D, Z;
      if( diag )
         D = ld4( diag + i );
#pragma unroll
      for( int u = 0; u < 4; u++ ) {
         X.v[ u ] += alpha * P.v[ u ];
         const Real rr = R.v[ u ] - alpha * AP.v[ u ];
         R.v[ u ] = rr;
         const Real zz = diag ? rr / D.v[ u ] : rr;
         Z.v[ u ] = zz;
         acc[ 0 ] += (double) rr * (double) zz;
      }
      st4( x + i, X );
      st4( r + i, R );
      if( diag )
         st4( z + i, Z );
   }
};

struct CgUpdateFin
{
   static constexpr bool active = true;
   __device__ void
   operator()( Ctl& c, const double* t ) const
   {
      const double s2 = c.s1;
      c.s1_prev = s2;
      c.s1 = t[ 0 ];
      c.beta = ( s2 == 0.0 ) ? 0.0 : c.s1 / s2;
      c.residue = sqrt( c.s1 ) / c.normb;
      next_iteration( c );
   }
};

// ---------------------------------------------------------------------------
// Pieces for a preconditioner applied between kernels (ILU(0)).

// out = b - s (b != NULL) or out = s: the SpMV half of a sink whose
// preconditioned half runs after the preconditioner; skipped with the gate
template< typename Real, class Gate >
struct StoreSink
{
   static constexpr int NR = 0;
   Real* out;
   const Real* b;
   Gate gate;
   __device__ bool skip() const { return gate.skip(); }
   __device__ __forceinline__ void put( int row, Real s, double* ) const { out[ row ] = b ? b[ row ] - s : s; }
   __device__ void finish( const double* ) const {}
};

// gate: the solve is finished
struct DoneGate
{
   const Ctl* ctl;
   __device__ bool skip() const { return ctl->done != 0; }
};

// the preconditioned half of a sink: sink.put( i, val[ i ] ) for every row,
// then the sink's reduction and finisher
template< typename Real, class Sink >
__global__ void __launch_bounds__( kReduceBlock )
sink_post_kernel( int64_t n, const Real* __restrict__ val, Sink sink, RedScratch rs )
{
   if( sink.skip() )
      return;
   AccOf< Sink > acc{};
   for( int64_t i = blockIdx.x * (int64_t) kReduceBlock + threadIdx.x; i < n; i += (int64_t) gridDim.x * kReduceBlock )
      sink.put( (int) i, val[ i ], acc.v );
   spmv_epilogue< Sink, kReduceBlock >( sink, acc.v, rs );
}

// CG with ILU(0): p = z ; acc = (r, z) (CG.hpp:37-58 after the preconditioner)
template< typename Real >
struct CgPrecInitOp
{
   static constexpr int NR = 1;
   const Real *r, *z;
   Real* p;
   __device__ __forceinline__ void load( const Ctl& ) {}
   __device__ __forceinline__ void
   operator()( int64_t i, double* acc ) const
   {
      const Real zz = z[ i ];
      p[ i ] = zz;
      acc[ 0 ] += (double) r[ i ] * (double) zz;
   }
};
struct CgInitFin
{
   static constexpr bool active = true;
   __device__ void
   operator()( Ctl& c, const double* t ) const
   {
      c.s1 = t[ 0 ];
      c.it = 0;
      c.residue = sqrt( c.s1 ) / c.normb;
      next_iteration( c );
   }
};

// CG with ILU(0): acc = (r, z) -> beta, residue (CgUpdateFin)
template< typename Real >
struct DotOp
{
   static constexpr int NR = 1;
   const Real *a, *b;
   __device__ __forceinline__ void load( const Ctl& ) {}
   __device__ __forceinline__ void operator()( int64_t i, double* acc ) const { acc[ 0 ] += (double) a[ i ] * (double) b[ i ]; }
};

// ---------------------------------------------------------------------------
// Reliable updates (mixed precision). The FP32 recurrence runs until its
// residue has dropped by the phase's factor; then x (FP64) takes the FP32
// correction, the residual is recomputed in FP64 from the FP64 matrix and
// replaces the recursive one, and the recurrence continues with its search
// direction: van der Vorst & Ye, "Residual replacement strategies for Krylov
// subspace iterative methods", SIAM J. Sci. Comput. 22 (2000), in the form
// used by mixed-precision lattice-QCD solvers (Clark et al., Comput. Phys.
// Commun. 181, 2010).

// z = M^-1 r ; [p = z] ; acc = (r, z)
template< typename Real >
struct CgReplaceOp
{
   static constexpr int NR = 1;
   const Real* r;
   Real *z, *p;
   const Real* diag;
   int restart;  // 1: p = z (first phase, or after a breakdown)
   __device__ __forceinline__ void load( const Ctl& ) {}
   __device__ __forceinline__ void
   operator()( int64_t i, double* acc ) const
   {
      const Real rr = r[ i ];
      Real zz = rr;
      if( diag ) {
         zz = rr / diag[ i ];
         z[ i ] = zz;
      }
      if( restart )
         p[ i ] = zz;
      acc[ 0 ] += (double) rr * (double) zz;
   }
};

// s1 = (r, z) of the replaced residual; beta against the iteration before
// (the phase ended after the x, r update and before the direction update)
struct CgReplaceFin
{
   static constexpr bool active = true;
   int restart;
   __device__ void
   operator()( Ctl& c, const double* t ) const
   {
      c.s1 = t[ 0 ];
      c.beta = ( restart || c.s1_prev == 0.0 ) ? 0.0 : c.s1 / c.s1_prev;
      c.residue = sqrt( c.s1 ) / c.normb;
      c.done = 0;
      c.reason = 0;
   }
};

// BiCGStab: r = M^-1 b (the correction restarts from 0) ; acc = {(r, r_ast), (r, r)}
template< typename Real >
struct BiReplaceOp
{
   static constexpr int NR = 2;
   const Real* b;
   Real* r;
   const Real *r_ast, *diag;
   __device__ __forceinline__ void load( const Ctl& ) {}
   __device__ __forceinline__ void
   operator()( int64_t i, double* acc ) const
   {
      Real rr = b[ i ];
      if( diag )
         rr = rr / diag[ i ];
      r[ i ] = rr;
      acc[ 0 ] += (double) rr * (double) r_ast[ i ];
      acc[ 1 ] += (double) rr * (double) rr;
   }
};

struct BiReplaceFin
{
   static constexpr bool active = true;
   __device__ void
   operator()( Ctl& c, const double* t ) const
   {
      c.rho = t[ 0 ];
      c.bi_beta = ( c.rho / c.rho_old ) * ( c.bi_alpha / c.omega );
      c.residue = sqrt( t[ 1 ] ) / c.normb;
      c.restart_flag = 0;
      c.done = 0;
      c.reason = 0;
   }
};

// p = (z or r) + beta p
template< typename Real >
struct CgDirOp
{
   static constexpr int NR = 1;
   Real* p;
   const Real* zr;
   Real beta;
   __device__ __forceinline__ void load( const Ctl& c ) { beta = (Real) c.beta; }
   __device__ __forceinline__ void operator()( int64_t i, double* ) const { p[ i ] = zr[ i ] + beta * p[ i ]; }
   __device__ __forceinline__ void
   apply4( int64_t i, double* ) const
   {
      V4< Real > P = ld4( p + i );
      const V4< Real > Z = ld4( zr + i );
#pragma unroll
      for( int u = 0; u < 4; u++ )
         P.v[ u ] = Z.v[ u ] + beta * P.v[ u ];
      st4( p + i, P );
   }
};

// ---------------------------------------------------------------------------
// BiCGStab (BICGStab.hpp:33-145)

// r = M^-1 (b - A x) with acc[0] += r*r ; used at start, on restart and for
// the exact residue. mode 0: init (p = r_ast = r, s = 0, rho), 1: restart
// (r_ast = r, rho = r_ast_sqnorm), 2: exact residue into `r` (the s vector).
template< typename Real >
struct BiResSink
{
   static constexpr int NR = 1;
   const Real* b;
   Real *r, *r_ast, *p, *s;
   const Real* diag;
   Ctl* ctl;
   int mode;
   int pre = 0;  // 1: sv is already M^-1 (b - A x) (ILU(0), applied between the SpMV and this pass)
   __device__ __forceinline__ void
   put( int row, Real sv, double* acc ) const
   {
      Real rr = pre ? sv : b[ row ] - sv;
      if( diag && ! pre )
         rr = rr / diag[ row ];
      r[ row ] = rr;
      if( mode <= 1 )
         r_ast[ row ] = rr;
      if( mode == 0 ) {
         p[ row ] = rr;
         s[ row ] = 0;
      }
      acc[ 0 ] += (double) rr * (double) rr;
   }
   __device__ void
   finish( const double* t ) const
   {
      Ctl& c = *ctl;
      if( mode == 0 ) {
         c.rho = c.r_ast_sqnorm = t[ 0 ];
         c.it = 0;
         c.residue = sqrt( c.rho ) / c.normb;
         next_iteration( c );
      }
      else if( mode == 1 ) {
         c.rho = c.r_ast_sqnorm = t[ 0 ];
         c.bi_beta = ( c.rho / c.rho_old ) * ( c.bi_alpha / c.omega );
         c.restart_flag = 0;
      }
      else {
         c.residue = sqrt( t[ 0 ] ) / c.normb;
         next_iteration( c );
      }
   }
};

// dst = M^-1 A src ; acc[0] += (dst, w0) ; acc[1] += (dst, w1) (w1 optional)
template< typename Real >
struct BiMatvecSink
{
   static constexpr int NR = 2;
   Real* dst;
   const Real* w0;
   const Real* diag;
   Ctl* ctl;
   int which;    // 0: alpha = rho / (Ap, r_ast) ; 1: omega = (As, s) / (As, As)
   int pre = 0;  // 1: sv is already M^-1 A src
   __device__ __forceinline__ void
   put( int row, Real sv, double* acc ) const
   {
      if( diag && ! pre )
         sv = sv / diag[ row ];
      dst[ row ] = sv;
      acc[ 0 ] += (double) sv * (double) w0[ row ];
      acc[ 1 ] += (double) sv * (double) sv;
   }
   __device__ void
   finish( const double* t ) const
   {
      Ctl& c = *ctl;
      if( which == 0 )
         c.bi_alpha = c.rho / t[ 0 ];
      else
         c.omega = t[ 0 ] / t[ 1 ];
   }
};

// s = r - alpha Ap
template< typename Real >
struct BiSOp
{
   static constexpr int NR = 1;
   Real* s;
   const Real *r, *Ap;
   Real alpha;
   __device__ __forceinline__ void load( const Ctl& c ) { alpha = (Real) c.bi_alpha; }
   __device__ __forceinline__ void operator()( int64_t i, double* ) const { s[ i ] = r[ i ] - alpha * Ap[ i ]; }
   __device__ __forceinline__ void
   apply4( int64_t i, double* ) const
   {
      const V4< Real > R = ld4( r + i ), AP = ld4( Ap + i );
      V4< Real > S;
#pragma unroll
      for( int u = 0; u < 4; u++ )
         S.v[ u ] = R.v[ u ] - alpha * AP.v[ u ];
      st4( s + i, S );
   }
};

// x += alpha p + omega s ; r = s - omega As ; acc = {(r, r_ast), (r, r)}
template< typename Real >
struct BiXrOp
{
   static constexpr int NR = 2;
   Real *x, *r;
   const Real *p, *s, *As, *r_ast;
   Real alpha, omega;
   __device__ __forceinline__ void
   load( const Ctl& c )
   {
      alpha = (Real) c.bi_alpha;
      omega = (Real) c.omega;
   }
   __device__ __forceinline__ void
   operator()( int64_t i, double* acc ) const
   {
      const Real si = s[ i ];
      x[ i ] += alpha * p[ i ] + omega * si;
      const Real rr = si - omega * As[ i ];
      r[ i ] = rr;
      acc[ 0 ] += (double) rr * (double) r_ast[ i ];
      acc[ 1 ] += (double) rr * (double) rr;
   }
   __device__ __forceinline__ void
   apply4( int64_t i, double* acc ) const
   {
      V4< Real > X = ld4( x + i );
      const V4< Real > S = ld4( s + i ), P = ld4( p + i ), AS = ld4( As + i ), RA = ld4( r_ast + i );
      V4< Real > R;
#pragma unroll
      for( int u = 0; u < 4; u++ ) {
         X.v[ u ] += alpha * P.v[ u ] + omega * S.v[ u ];
         const Real rr = S.v[ u ] - omega * AS.v[ u ];
         R.v[ u ] = rr;
         acc[ 0 ] += (double) rr * (double) RA.v[ u ];
         acc[ 1 ] += (double) rr * (double) rr;
      }
      st4( x + i, X );
      st4( r + i, R );
   }
};

struct BiXrFin
{
   static constexpr bool active = true;
   double eps2;
   int exact;
   __device__ void
   operator()( Ctl& c, const double* t ) const
   {
      c.rho_old = c.rho;
      c.rho = t[ 0 ];
      if( fabs( c.rho ) < eps2 * c.r_ast_sqnorm ) {
         // r has become too orthogonal to r_ast: restart with a new r0 (BICGStab.hpp:86-92)
         c.restart_flag = 1;
         return;
      }
      c.bi_beta = ( c.rho / c.rho_old ) * ( c.bi_alpha / c.omega );
      if( ! exact ) {
         c.residue = sqrt( t[ 1 ] ) / c.normb;
         next_iteration( c );
      }
   }
};

// p = r + beta p - (beta*omega) Ap
template< typename Real >
struct BiPOp
{
   static constexpr int NR = 1;
   Real* p;
   const Real *r, *Ap;
   Real beta, bo;
   __device__ __forceinline__ void
   load( const Ctl& c )
   {
      beta = (Real) c.bi_beta;
      bo = (Real) ( c.bi_beta * c.omega );
   }
   __device__ __forceinline__ void operator()( int64_t i, double* ) const
   {
      p[ i ] = r[ i ] + beta * p[ i ] - bo * Ap[ i ];
   }
   __device__ __forceinline__ void
   apply4( int64_t i, double* ) const
   {
      V4< Real > P = ld4( p + i );
      const V4< Real > R = ld4( r + i ), AP = ld4( Ap + i );
#pragma unroll
      for( int u = 0; u < 4; u++ )
         P.v[ u ] = R.v[ u ] + beta * P.v[ u ] - bo * AP.v[ u ];
      st4( p + i, P );
   }
};

// ---------------------------------------------------------------------------
// SpMV wrapper that skips the launch's work when the solve is done or a
// conditional step is not requested. The flag is read inside the kernel so
// that captured graphs stay valid.
template< typename Real, class Sink >
struct GatedSink
{
   static constexpr int NR = Sink::NR;
   Sink inner;
   __device__ __forceinline__ void put( int row, Real s, double* acc ) const { inner.put( row, s, acc ); }
   __device__ void finish( const double* t ) const { inner.finish( t ); }
};

}  // namespace b2s
