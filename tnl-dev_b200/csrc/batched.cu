// Batched solves in one persistent launch: many independent SPD systems,
// each with 1..8 right-hand sides, solved by TNL's CG recurrence
// (Solvers/Linear/CG.hpp:17-104) with the Jacobi preconditioner
// (Preconditioners/Diagonal.hpp:13-47), one thread-block cluster per system.
//
// The kernel is persistent: clusters take systems from a device work queue
// (largest first, so the long ones do not end up in the tail) until it is
// empty. A cluster of C CTAs (one per SM) splits a system's rows; its
// reductions go through distributed shared memory and every CTA sums the C
// partials in rank order, so all of them take the same decisions and the
// result does not depend on timing. Between the three phases of an iteration
// the cluster synchronizes with barrier.cluster (no global memory flags, no
// spin waits). C is chosen by the autotuner from timed samples of the batch.
//
// What bounds it is L2 traffic: per row, right-hand side and iteration the
// direction P is gathered once per nonzero and X, R and AP are read and
// written. Where a CTA's rows of P fit its shared memory (and then R, then AP)
// they stay there, P gathered from it and, at the edge of a CTA's rows, from
// the other CTAs' (solve_system). 512 systems of 1k to 65k rows, 1 to 8
// right-hand sides: 324 -> 188 ms; 60 systems of up to 10k rows: 13.2 -> 4.7 ms.
//
// Right-hand sides of one system are interleaved (element (i, j) at
// i*k + j), so one pass over a matrix row serves all k of them.
//
// TNL solves one system per call (and one right-hand side per solve); this
// batched form has no counterpart there.
#include "b2s_internal.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>
#include <numeric>
#include <vector>

namespace cg = cooperative_groups;

namespace b2s {

constexpr int kBatchBlock = 1024;
constexpr int kBatchMaxRhs = 8;
constexpr int kBatchWarps = kBatchBlock / 32;
constexpr size_t kBatchSmem = 208 * 1024;  // per CTA (one CTA per SM), beside the static state

struct BatchArgs
{
   const int32_t* off;
   const int32_t* col;
   const double* val;
   const double* diag;     // Jacobi diagonal; nullptr: no preconditioner
   const int64_t* row_ptr;  // nsys + 1
   const int32_t* nrhs;     // nsys
   const int64_t* vec_off;  // nsys: first element of the system's interleaved vectors
   const int64_t* rhs_off;  // nsys: first right-hand side of the system (report slots)
   const int32_t* order;    // work queue: systems, largest first
   int32_t nsys;
   const double* B;
   double* X;
   double *R, *P, *AP;
   int64_t* it_out;
   double* res_out;
   int32_t* status_out;
   unsigned int* counter;
   double tol, div_tol;
   int64_t maxit, minit;
   int smem_elems;  // doubles of dynamic shared memory per CTA
   int64_t* t_sys;  // optional (autotuner): global-timer ns at start and end of each system
};

__device__ __forceinline__ int64_t
global_ns()
{
   int64_t t;
   asm volatile( "mov.u64 %0, %%globaltimer;" : "=l"( t ) );
   return t;
}

// Per-CTA shared state of the system being solved.
template< int K >
struct SysState
{
   double part[ 2 ][ K ];  // this CTA's partial sums (double buffered)
   double red[ K ][ kBatchWarps ];
   double normb[ K ], s1[ K ], alpha[ K ], beta[ K ], residue[ K ];
   long long it[ K ];
   int done[ K ], reason[ K ];
};

// IterativeSolver::checkNextIteration / nextIteration for one right-hand side
__device__ __forceinline__ void
next_iteration_rhs( double residue, long long& it, int& done, int& reason, const BatchArgs& a )
{
   const bool go = ! ( isnan( residue ) || it > a.maxit || ( residue > a.div_tol && it >= a.minit )
                       || ( residue < a.tol && it >= a.minit ) );
   it++;
   if( ! go ) {
      done = 1;
      reason = 1;
   }
}

// Cluster-wide sums of K values in a fixed order: lanes, then warps (warp j
// sums value j), then the C CTAs in rank order. Thread j < K hands the total
// of value j to `fn( j, total )`, so the right-hand sides' scalar work runs
// side by side; what it writes is visible to the CTA on return.
template< int K, class F >
__device__ __forceinline__ void
cluster_sum( cg::cluster_group& cl, SysState< K >& st, int& buf, double ( &v )[ K ], F&& fn )
{
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
   for( int j = 0; j < K; j++ ) {
      const double s = warp_sum( v[ j ] );
      if( lane == 0 )
         st.red[ j ][ warp ] = s;
   }
   __syncthreads();
   if( warp < K ) {
      const double s = warp_sum( lane < kBatchWarps ? st.red[ warp ][ lane ] : 0.0 );
      if( lane == 0 )
         st.part[ buf ][ warp ] = s;
   }
   cl.sync();
   if( threadIdx.x < K ) {
      const int j = threadIdx.x, C = (int) cl.num_blocks();
      double t = 0.0;
      for( int q = 0; q < C; q++ )
         t += cl.map_shared_rank( &st.part[ buf ][ 0 ], q )[ j ];
      fn( j, t );
   }
   __syncthreads();
   buf ^= 1;
}

// y(rows) = A p over the CTA's rows of the system, K columns at once:
// `gather( c, xs )` gives the K entries at column c (local to the system),
// `fn( i, acc )` receives each row's K sums (i counted from r_begin).
template< int K, class G, class F >
__device__ __forceinline__ void
spmm_rows( const BatchArgs& a, int64_t row0, int r_begin, int rows, G&& gather, F&& fn )
{
   for( int i = threadIdx.x; i < rows; i += kBatchBlock ) {
      const int64_t gr = row0 + r_begin + i;
      const int b = __ldg( a.off + gr ), e = __ldg( a.off + gr + 1 );
      double acc[ K ];
#pragma unroll
      for( int j = 0; j < K; j++ )
         acc[ j ] = 0.0;
      // the row's columns and values four at a time, then their gathers, so a
      // stencil row costs two round trips instead of one per nonzero
      for( int t0 = b; t0 < e; t0 += 4 ) {
         int lc[ 4 ];
         double v[ 4 ];
#pragma unroll
         for( int u = 0; u < 4; u++ ) {
            lc[ u ] = t0 + u < e ? __ldg( a.col + t0 + u ) - (int) row0 : 0;
            v[ u ] = t0 + u < e ? __ldg( a.val + t0 + u ) : 0.0;
         }
#pragma unroll
         for( int u = 0; u < 4; u++ ) {
            if( t0 + u < e ) {
               double xs[ K ];
               gather( lc[ u ], xs );
#pragma unroll
               for( int j = 0; j < K; j++ )
                  acc[ j ] += v[ u ] * xs[ j ];
            }
         }
      }
      fn( i, acc );
   }
}

// One system on one cluster. PS: the direction P sits in the CTAs' shared
// memory (`smem`, a.smem_elems doubles each), where the product gathers it
// (other CTAs' rows through distributed shared memory), and R and AP too as
// far as they fit; otherwise P goes through L2. The vectors are kept by
// right-hand side (element (i, j) at j * ld + i), so a warp's accesses to one
// right-hand side are consecutive in either memory; with PS, X is worked on
// in that order too, in the buffer that P would take.
template< int K, bool PS >
__device__ void
solve_system( const BatchArgs& a, int sys, cg::cluster_group& cl, SysState< K >& st, double* smem )
{
   const int C = (int) cl.num_blocks(), q = (int) cl.block_rank();
   const int64_t row0 = a.row_ptr[ sys ];
   const int n = (int) ( a.row_ptr[ sys + 1 ] - row0 );
   const int per = ( n + C - 1 ) / C;  // rows per CTA
   const int r_begin = min( n, q * per ), rows = min( n, r_begin + per ) - r_begin;
   const int64_t vo = a.vec_off[ sys ];
   const double* B = a.B + vo + (int64_t) r_begin * K;
   double* X = a.X + vo;
   const double* dg = a.diag ? a.diag + row0 + r_begin : nullptr;
   int buf = 0;
   // where the vectors live: pointer to this CTA's first row, distance between right-hand sides
   const int fit = PS ? a.smem_elems / max( 1, per * K ) : 0;  // vectors that fit (P, then R, then AP)
   double *P, *R, *AP;
   const int64_t ldP = PS ? per : n;
   const int64_t ldR = fit >= 2 ? per : n, ldA = fit >= 3 ? per : n;
   P = PS ? smem : a.P + vo + r_begin;
   R = fit >= 2 ? smem + per * K : a.R + vo + r_begin;
   AP = fit >= 3 ? smem + 2 * per * K : a.AP + vo + r_begin;
   double* xw = PS ? a.P + vo + r_begin : X + (int64_t) r_begin * K;
   const int xi = PS ? 1 : K, xj = PS ? n : 1;

   // ||M^-1 b|| per right-hand side (CG.hpp:24-32)
   {
      double v[ K ];
#pragma unroll
      for( int j = 0; j < K; j++ )
         v[ j ] = 0.0;
      for( int i = threadIdx.x; i < rows; i += kBatchBlock ) {
         const double d = dg ? dg[ i ] : 1.0;
#pragma unroll
         for( int j = 0; j < K; j++ ) {
            const double t = dg ? B[ (int64_t) i * K + j ] / d : B[ (int64_t) i * K + j ];
            v[ j ] += t * t;
         }
      }
      cluster_sum< K >( cl, st, buf, v, [ & ]( int j, double t ) {
         st.normb[ j ] = t == 0.0 ? 1.0 : sqrt( t );
      } );
   }
   // r = b - A x ; z = M^-1 r ; p = z ; s1 = (r, z) (CG.hpp:37-58)
   {
      double v[ K ];
#pragma unroll
      for( int j = 0; j < K; j++ )
         v[ j ] = 0.0;
      spmm_rows< K >(
         a, row0, r_begin, rows,
         [ & ]( int c, double( &xs )[ K ] ) {
#pragma unroll
            for( int j = 0; j < K; j++ )
               xs[ j ] = X[ (int64_t) c * K + j ];
         },
         [ & ]( int i, const double( &acc )[ K ] ) {
            const double d = dg ? dg[ i ] : 1.0;
#pragma unroll
            for( int j = 0; j < K; j++ ) {
               const double r = B[ (int64_t) i * K + j ] - acc[ j ];
               const double z = dg ? r / d : r;
               R[ j * ldR + i ] = r;
               P[ j * ldP + i ] = z;
               if( PS )
                  xw[ j * xj + i ] = X[ (int64_t) ( r_begin + i ) * K + j ];
               v[ j ] += r * z;
            }
         } );
      cluster_sum< K >( cl, st, buf, v, [ & ]( int j, double t ) {
         st.s1[ j ] = t;
         st.it[ j ] = 0;
         st.done[ j ] = 0;
         st.reason[ j ] = 0;
         st.residue[ j ] = sqrt( t ) / st.normb[ j ];
         next_iteration_rhs( st.residue[ j ], st.it[ j ], st.done[ j ], st.reason[ j ], a );
      } );
   }
   for( ;; ) {
      bool any = false;
#pragma unroll
      for( int j = 0; j < K; j++ )
         any |= ! st.done[ j ];
      if( ! any )
         break;
      // P of every row is complete before anyone gathers it
      cl.sync();
      // s2 = (A p, p)
      {
         double v[ K ];
#pragma unroll
         for( int j = 0; j < K; j++ )
            v[ j ] = 0.0;
         spmm_rows< K >(
            a, row0, r_begin, rows,
            [ & ]( int c, double( &xs )[ K ] ) {
               const double* p;
               if constexpr( PS ) {
                  const int i = c - r_begin;
                  if( i >= 0 && i < rows ) {
#pragma unroll
                     for( int j = 0; j < K; j++ )
                        xs[ j ] = smem[ j * per + i ];
                     return;
                  }
                  const int owner = c / per;
                  p = cl.map_shared_rank( smem, owner ) + ( c - owner * per );
#pragma unroll
                  for( int j = 0; j < K; j++ )
                     xs[ j ] = p[ j * per ];
               }
               else {
                  p = a.P + vo + c;
#pragma unroll
                  for( int j = 0; j < K; j++ )
                     xs[ j ] = __ldcg( p + (int64_t) j * n );  // written by other CTAs: read through L2
               }
            },
            [ & ]( int i, const double( &acc )[ K ] ) {
#pragma unroll
               for( int j = 0; j < K; j++ ) {
                  AP[ j * ldA + i ] = acc[ j ];
                  v[ j ] += acc[ j ] * P[ j * ldP + i ];
               }
            } );
         cluster_sum< K >( cl, st, buf, v, [ & ]( int j, double t ) {
            if( st.done[ j ] )
               return;
            if( t == 0.0 ) {
               // p = 0 => r = 0: solved (CG.hpp:64-67)
               st.residue[ j ] = 0.0;
               st.done[ j ] = 1;
               st.reason[ j ] = 2;
               st.alpha[ j ] = 0.0;
            }
            else
               st.alpha[ j ] = st.s1[ j ] / t;
         } );
      }
      // x += alpha p ; r -= alpha Ap ; z = M^-1 r ; s1 = (r, z)
      {
         double al[ K ], v[ K ];
         bool act[ K ];
#pragma unroll
         for( int j = 0; j < K; j++ ) {
            al[ j ] = st.alpha[ j ];
            act[ j ] = ! st.done[ j ];
            v[ j ] = 0.0;
         }
         for( int i = threadIdx.x; i < rows; i += kBatchBlock ) {
            const double d = dg ? dg[ i ] : 1.0;
#pragma unroll
            for( int j = 0; j < K; j++ ) {
               if( ! act[ j ] )
                  continue;
               double* x = xw + (int64_t) i * xi + (int64_t) j * xj;
               *x += al[ j ] * P[ j * ldP + i ];
               const double r = R[ j * ldR + i ] - al[ j ] * AP[ j * ldA + i ];
               R[ j * ldR + i ] = r;
               v[ j ] += dg ? r * ( r / d ) : r * r;
            }
         }
         cluster_sum< K >( cl, st, buf, v, [ & ]( int j, double t ) {
            if( st.done[ j ] )
               return;
            const double s2 = st.s1[ j ];
            st.s1[ j ] = t;
            st.beta[ j ] = s2 == 0.0 ? 0.0 : t / s2;
            st.residue[ j ] = sqrt( t ) / st.normb[ j ];
            next_iteration_rhs( st.residue[ j ], st.it[ j ], st.done[ j ], st.reason[ j ], a );
         } );
      }
      // p = z + beta p
      {
         double be[ K ];
         bool act[ K ];
#pragma unroll
         for( int j = 0; j < K; j++ ) {
            be[ j ] = st.beta[ j ];
            act[ j ] = ! st.done[ j ];
         }
         for( int i = threadIdx.x; i < rows; i += kBatchBlock ) {
            const double d = dg ? dg[ i ] : 1.0;
#pragma unroll
            for( int j = 0; j < K; j++ ) {
               if( ! act[ j ] )
                  continue;
               const double r = R[ j * ldR + i ];
               P[ j * ldP + i ] = ( dg ? r / d : r ) + be[ j ] * P[ j * ldP + i ];
            }
         }
      }
   }
   if( PS )
      for( int i = threadIdx.x; i < rows; i += kBatchBlock )
#pragma unroll
         for( int j = 0; j < K; j++ )
            X[ (int64_t) ( r_begin + i ) * K + j ] = xw[ j * xj + i ];
   // report (rank 0)
   if( q == 0 && threadIdx.x < K ) {
      const int j = threadIdx.x;
      const int64_t slot = a.rhs_off[ sys ] + j;
      a.it_out[ slot ] = st.it[ j ];
      a.res_out[ slot ] = st.residue[ j ];
      const double r = st.residue[ j ];
      int s = B2S_OK;
      if( isnan( r ) )
         s = B2S_NAN;
      else if( r > a.div_tol && st.it[ j ] > a.minit )
         s = B2S_DIVERGED;
      else if( st.it[ j ] >= a.maxit || r > a.tol )
         s = st.reason[ j ] == 2 ? B2S_OK : B2S_NOT_CONVERGED;
      a.status_out[ slot ] = s;
   }
}

__global__ void __launch_bounds__( kBatchBlock, 1 )
batch_cg_kernel( BatchArgs a )
{
   cg::cluster_group cl = cg::this_cluster();
   __shared__ __align__( 16 ) unsigned char smem_raw[ sizeof( SysState< kBatchMaxRhs > ) ];
   __shared__ int next_sys;
   extern __shared__ __align__( 16 ) double batch_smem[];
   for( ;; ) {
      if( cl.block_rank() == 0 && threadIdx.x == 0 )
         next_sys = (int) atomicAdd( a.counter, 1u );
      cl.sync();
      const int idx = *cl.map_shared_rank( &next_sys, 0 );
      // every CTA has read rank 0's ticket before it can be overwritten
      cl.sync();
      if( idx >= a.nsys )
         break;
      const int sys = a.order[ idx ];
      const bool stamp = a.t_sys && cl.block_rank() == 0 && threadIdx.x == 0;
      if( stamp )
         a.t_sys[ 2 * sys ] = global_ns();
      // the direction of the largest CTA's rows in shared memory
      const int64_t C = cl.num_blocks(), rows = a.row_ptr[ sys + 1 ] - a.row_ptr[ sys ];
      const bool in_smem = ( rows + C - 1 ) / C * a.nrhs[ sys ] <= a.smem_elems;
      switch( a.nrhs[ sys ] ) {
#define B2S_BATCH_K( KK )                                                                            \
   case KK:                                                                                          \
      if( in_smem )                                                                                  \
         solve_system< KK, true >( a, sys, cl, *reinterpret_cast< SysState< KK >* >( smem_raw ), batch_smem );  \
      else                                                                                           \
         solve_system< KK, false >( a, sys, cl, *reinterpret_cast< SysState< KK >* >( smem_raw ), batch_smem ); \
      break;
         B2S_BATCH_K( 1 )
         B2S_BATCH_K( 2 )
         B2S_BATCH_K( 3 )
         B2S_BATCH_K( 4 )
         B2S_BATCH_K( 5 )
         B2S_BATCH_K( 6 )
         B2S_BATCH_K( 7 )
         B2S_BATCH_K( 8 )
#undef B2S_BATCH_K
         default:
            break;
      }
      // the shared state of this system is dead before the next one starts
      cl.sync();
      if( stamp )
         a.t_sys[ 2 * sys + 1 ] = global_ns();
   }
}

__global__ void
batch_diag_kernel( int64_t rows, const int32_t* __restrict__ off, const int32_t* __restrict__ col,
                   const double* __restrict__ val, double* diag )
{
   for( int64_t r = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; r < rows; r += (int64_t) gridDim.x * blockDim.x ) {
      double d = 0.0;
      for( int t = off[ r ]; t < off[ r + 1 ]; t++ )
         if( col[ t ] == r ) {
            d = val[ t ];
            break;
         }
      diag[ r ] = d;  // Diagonal::update takes A_ii (Diagonal.hpp:24-36); solve divides by it
   }
}

// The first row whose offsets do not lie in [0, nnz] in order or that has a
// column outside its system's diagonal block: solve_system turns columns into
// places of the system's vectors, in another CTA's shared memory among others.
__global__ void
batch_check_kernel( int64_t rows, int64_t nnz, int nsys, const int64_t* __restrict__ row_ptr,
                    const int32_t* __restrict__ off, const int32_t* __restrict__ col, int* bad )
{
   for( int64_t r = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; r < rows; r += (int64_t) gridDim.x * blockDim.x ) {
      const int b = off[ r ], e = off[ r + 1 ];
      if( b < 0 || e < b || e > nnz ) {
         atomicMin( bad, (int) r );
         continue;
      }
      int lo = 0, hi = nsys;  // the last system that starts at or before r (empty ones start there too)
      while( hi - lo > 1 ) {
         const int mid = ( lo + hi ) / 2;
         if( row_ptr[ mid ] <= r )
            lo = mid;
         else
            hi = mid;
      }
      const int64_t c0 = row_ptr[ lo ], c1 = row_ptr[ lo + 1 ];
      for( int t = b; t < e; t++ )
         if( col[ t ] < c0 || col[ t ] >= c1 ) {
            atomicMin( bad, (int) r );
            break;
         }
   }
}

}  // namespace b2s

using namespace b2s;

struct b2s_batch_t
{
   int32_t nsys = 0;
   int64_t rows = 0, nnz = 0, nvec = 0, nslots = 0;
   std::vector< int64_t > row_ptr_h, vec_off_h, rhs_off_h;
   std::vector< int32_t > nrhs_h;
   DevBuf off, col, val, diag, row_ptr, nrhs, vec_off, rhs_off, order;
   DevBuf R, P, AP, counter, it_out, res_out, status_out;
   b2s_batch_opts o{};
   int cluster = 0;  // chosen cluster size
};

namespace b2s {

static b2s_status
launch_batch( b2s_batch_t* bt, const double* B, double* X, int cluster, int nsys_limit, int64_t maxit,
              cudaStream_t s, const int32_t* order = nullptr, int64_t* t_sys = nullptr, int* clusters_out = nullptr )
{
   BatchArgs a{};
   a.off = bt->off.as< int32_t >();
   a.col = bt->col.as< int32_t >();
   a.val = bt->val.as< double >();
   a.diag = bt->o.preconditioner ? bt->diag.as< double >() : nullptr;
   a.row_ptr = bt->row_ptr.as< int64_t >();
   a.nrhs = bt->nrhs.as< int32_t >();
   a.vec_off = bt->vec_off.as< int64_t >();
   a.rhs_off = bt->rhs_off.as< int64_t >();
   a.order = order ? order : bt->order.as< int32_t >();
   a.nsys = nsys_limit;
   a.B = B;
   a.X = X;
   a.R = bt->R.as< double >();
   a.P = bt->P.as< double >();
   a.AP = bt->AP.as< double >();
   a.it_out = bt->it_out.as< int64_t >();
   a.res_out = bt->res_out.as< double >();
   a.status_out = bt->status_out.as< int32_t >();
   a.counter = bt->counter.as< unsigned int >();
   a.tol = bt->o.convergence_residue;
   a.div_tol = bt->o.divergence_residue;
   a.maxit = maxit;
   a.minit = bt->o.min_iterations;
   a.smem_elems = (int) ( kBatchSmem / sizeof( double ) );
   a.t_sys = t_sys;
   B2S_TRY_CUDA( cudaMemsetAsync( bt->counter.p, 0, sizeof( unsigned int ), s ) );
   cudaLaunchConfig_t cfg{};
   cudaLaunchAttribute attr[ 1 ];
   attr[ 0 ].id = cudaLaunchAttributeClusterDimension;
   attr[ 0 ].val.clusterDim.x = cluster;
   attr[ 0 ].val.clusterDim.y = 1;
   attr[ 0 ].val.clusterDim.z = 1;
   cfg.blockDim = dim3( kBatchBlock );
   cfg.dynamicSmemBytes = kBatchSmem;
   B2S_TRY( allow_smem( reinterpret_cast< const void* >( batch_cg_kernel ), kBatchSmem ) );
   cfg.stream = s;
   cfg.attrs = attr;
   cfg.numAttrs = 1;
   cfg.gridDim = dim3( cluster );
   int nclusters = 0;
   B2S_TRY_CUDA( cudaOccupancyMaxActiveClusters( &nclusters, batch_cg_kernel, &cfg ) );
   if( nclusters < 1 ) {
      set_error( "batched solver: a cluster of %d CTAs does not fit on the device", cluster );
      return B2S_UNSUPPORTED;
   }
   if( clusters_out )
      *clusters_out = nclusters;
   nclusters = std::min( nclusters, std::max( 1, nsys_limit ) );
   cfg.gridDim = dim3( nclusters * cluster );
   B2S_TRY_CUDA( cudaLaunchKernelEx( &cfg, batch_cg_kernel, a ) );
   return B2S_OK;
}

// Autotuner of the cluster size. A sample of systems (even strides through
// the size-sorted queue) is solved from X under every candidate C while the
// kernel stamps each system's start and end: to convergence under the first C,
// which tells the systems' iterations, under the others for kTuneIterations,
// scaled to them. Every system of the queue is then taken to last as long as
// its neighbour in the sample, and the queue is played through on the resident
// clusters of C; the C whose last system ends first wins. (The systems' total
// time spread over the device, or the longest of them, leaves out the tail
// where a few long systems run alone.)
// W: the sample's solutions.
constexpr int64_t kTuneIterations = 32;

static b2s_status
autotune_cluster( b2s_batch_t* bt, const double* B, const double* X, double* W, cudaStream_t s, int& best )
{
   best = 1;
   const int cands[] = { 8, 4, 2, 1 };
   const int sample = std::min( bt->nsys, 2 * num_sms() );
   std::vector< int32_t > order_h( bt->nsys );
   B2S_TRY( copy_d2h( order_h.data(), bt->order.p, bt->nsys * sizeof( int32_t ), s ) );
   std::vector< int32_t > pick( sample );
   for( int k = 0; k < sample; k++ )
      pick[ k ] = order_h[ (int64_t) k * bt->nsys / sample ];
   DevBuf sample_order, stamps;
   B2S_TRY( sample_order.alloc( sample * sizeof( int32_t ) ) );
   B2S_TRY( copy_h2d( sample_order.p, pick.data(), sample * sizeof( int32_t ), s ) );
   B2S_TRY( stamps.alloc( (size_t) 2 * bt->nsys * sizeof( int64_t ) ) );
   std::vector< int64_t > t( 2 * bt->nsys ), its( bt->nslots );
   std::vector< double > scale;  // a system's iterations over the timed ones
   double best_est = 1e300;
   for( int c : cands ) {
      int nclusters = 0;
      B2S_TRY_CUDA( cudaMemcpyAsync( W, X, bt->nvec * sizeof( double ), cudaMemcpyDeviceToDevice, s ) );
      const bool all = scale.empty();
      const b2s_status st = launch_batch( bt, B, W, c, sample, all ? bt->o.max_iterations : std::min< int64_t >( bt->o.max_iterations, kTuneIterations ), s,
                                          sample_order.as< int32_t >(), stamps.as< int64_t >(), &nclusters );
      if( st != B2S_OK ) {
         cudaGetLastError();
         clear_error();
         continue;
      }
      B2S_TRY( copy_d2h( t.data(), stamps.p, t.size() * sizeof( int64_t ), s ) );
      if( all ) {
         B2S_TRY( copy_d2h( its.data(), bt->it_out.p, bt->nslots * sizeof( int64_t ), s ) );
         for( const int sys : pick ) {
            int64_t most = 1;
            for( int j = 0; j < bt->nrhs_h[ sys ]; j++ )
               most = std::max( most, its[ bt->rhs_off_h[ sys ] + j ] );
            scale.push_back( std::max( 1.0, (double) most / (double) ( kTuneIterations + 1 ) ) );
         }
      }
      std::vector< double > ends( (size_t) std::max( nclusters, 1 ), 0.0 );  // a heap, the earliest first
      double est = 0;
      for( int k = 0; k < bt->nsys; k++ ) {
         const int q = (int) ( (int64_t) k * sample / bt->nsys ), sys = pick[ q ];
         std::pop_heap( ends.begin(), ends.end(), std::greater< double >() );
         ends.back() += (double) ( t[ 2 * sys + 1 ] - t[ 2 * sys ] ) * ( all ? 1.0 : scale[ q ] );
         est = std::max( est, ends.back() );
         std::push_heap( ends.begin(), ends.end(), std::greater< double >() );
      }
      if( est < best_est ) {
         best_est = est;
         best = c;
      }
   }
   return B2S_OK;
}

}  // namespace b2s

extern "C" {

void
b2s_batch_opts_default( b2s_batch_opts* o )
{
   if( ! o )
      return;
   std::memset( o, 0, sizeof( *o ) );
   o->preconditioner = B2S_PRECOND_JACOBI;
   o->convergence_residue = 1e-8;
   o->divergence_residue = 1e300;
   o->max_iterations = 1000000;
   o->min_iterations = 0;
   o->cluster_size = 0;
}

b2s_status
b2s_batch_create( int32_t nsys, const int64_t* row_ptr, const int32_t* nrhs, const int32_t* offsets,
                  const int32_t* columns, const double* values, b2s_memory where, const b2s_batch_opts* opts,
                  b2s_stream stream, b2s_batch* out )
{
   clear_error();
   B2S_CHECK_ARG( out && row_ptr && nrhs && offsets && nsys >= 0, "NULL argument" );
   *out = nullptr;
   B2S_CHECK_ARG( where == B2S_HOST || where == B2S_DEVICE, "where" );
   cudaStream_t s = as_stream( stream );
   std::unique_ptr< b2s_batch_t > bt( new b2s_batch_t() );
   b2s_batch_opts_default( &bt->o );
   if( opts )
      bt->o = *opts;
   B2S_CHECK_ARG( bt->o.preconditioner == B2S_PRECOND_NONE || bt->o.preconditioner == B2S_PRECOND_JACOBI,
                  "batched solves take no preconditioner or Jacobi" );
   B2S_CHECK_ARG( bt->o.cluster_size == 0 || bt->o.cluster_size == 1 || bt->o.cluster_size == 2
                     || bt->o.cluster_size == 4 || bt->o.cluster_size == 8,
                  "cluster_size in {0 (autotune), 1, 2, 4, 8}" );
   bt->nsys = nsys;
   bt->row_ptr_h.assign( row_ptr, row_ptr + nsys + 1 );
   bt->nrhs_h.assign( nrhs, nrhs + nsys );
   B2S_CHECK_ARG( bt->row_ptr_h[ 0 ] == 0, "row_ptr[0] must be 0" );
   for( int i = 0; i < nsys; i++ ) {
      B2S_CHECK_ARG( bt->row_ptr_h[ i + 1 ] >= bt->row_ptr_h[ i ], "row_ptr must be non-decreasing" );
      B2S_CHECK_ARG( bt->nrhs_h[ i ] >= 1 && bt->nrhs_h[ i ] <= kBatchMaxRhs, "right-hand sides per system in [1, 8]" );
   }
   bt->rows = bt->row_ptr_h[ nsys ];
   B2S_CHECK_ARG( bt->rows < INT32_MAX, "total rows must fit in int32" );
   int32_t nnz32 = 0;
   if( where == B2S_HOST )
      nnz32 = offsets[ bt->rows ];
   else
      B2S_TRY( copy_d2h( &nnz32, offsets + bt->rows, sizeof( int32_t ), s ) );
   bt->nnz = nnz32;
   B2S_CHECK_ARG( bt->nnz >= 0 && ( bt->nnz == 0 || ( columns && values ) ), "columns / values" );
   bt->vec_off_h.resize( nsys );
   bt->rhs_off_h.resize( nsys );
   int64_t v = 0, k = 0;
   for( int i = 0; i < nsys; i++ ) {
      bt->vec_off_h[ i ] = v;
      bt->rhs_off_h[ i ] = k;
      v += ( bt->row_ptr_h[ i + 1 ] - bt->row_ptr_h[ i ] ) * bt->nrhs_h[ i ];
      k += bt->nrhs_h[ i ];
   }
   bt->nvec = v;
   bt->nslots = k;
   // work queue: largest systems first (rows x right-hand sides)
   std::vector< int32_t > order( nsys );
   std::iota( order.begin(), order.end(), 0 );
   std::stable_sort( order.begin(), order.end(), [ & ]( int a, int b ) {
      const int64_t wa = ( bt->row_ptr_h[ a + 1 ] - bt->row_ptr_h[ a ] ) * ( 4 + bt->nrhs_h[ a ] );
      const int64_t wb = ( bt->row_ptr_h[ b + 1 ] - bt->row_ptr_h[ b ] ) * ( 4 + bt->nrhs_h[ b ] );
      return wa > wb;
   } );
   const cudaMemcpyKind kin = where == B2S_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
   B2S_TRY( bt->off.alloc( ( bt->rows + 1 ) * sizeof( int32_t ) ) );
   B2S_TRY( bt->col.alloc( std::max< int64_t >( bt->nnz, 1 ) * sizeof( int32_t ) ) );
   B2S_TRY( bt->val.alloc( std::max< int64_t >( bt->nnz, 1 ) * sizeof( double ) ) );
   B2S_TRY_CUDA( cudaMemcpyAsync( bt->off.p, offsets, ( bt->rows + 1 ) * sizeof( int32_t ), kin, s ) );
   if( bt->nnz > 0 ) {
      B2S_TRY_CUDA( cudaMemcpyAsync( bt->col.p, columns, bt->nnz * sizeof( int32_t ), kin, s ) );
      B2S_TRY_CUDA( cudaMemcpyAsync( bt->val.p, values, bt->nnz * sizeof( double ), kin, s ) );
   }
   B2S_TRY( bt->row_ptr.alloc( ( nsys + 1 ) * sizeof( int64_t ) ) );
   B2S_TRY( copy_h2d( bt->row_ptr.p, bt->row_ptr_h.data(), ( nsys + 1 ) * sizeof( int64_t ), s ) );
   if( bt->rows > 0 ) {
      B2S_TRY( bt->counter.alloc( 64 ) );
      const int none = INT32_MAX;
      B2S_TRY( copy_h2d( bt->counter.p, &none, sizeof( int ), s ) );
      batch_check_kernel<<< (int) std::min< int64_t >( ( bt->rows + 255 ) / 256, (int64_t) num_sms() * 16 ), 256, 0,
                               s >>>( bt->rows, bt->nnz, nsys, bt->row_ptr.as< int64_t >(), bt->off.as< int32_t >(),
                                      bt->col.as< int32_t >(), bt->counter.as< int >() );
      B2S_TRY_CUDA( cudaGetLastError() );
      int bad = none;
      B2S_TRY( copy_d2h( &bad, bt->counter.p, sizeof( int ), s ) );
      if( bad != none ) {
         set_error( "batch: row %d has offsets out of order or a column outside its system's block", bad );
         return B2S_INVALID_ARG;
      }
   }
   B2S_TRY( bt->diag.alloc( std::max< int64_t >( bt->rows, 1 ) * sizeof( double ) ) );
   if( bt->rows > 0 ) {
      batch_diag_kernel<<< (int) std::min< int64_t >( ( bt->rows + 255 ) / 256, (int64_t) num_sms() * 16 ), 256, 0,
                              s >>>( bt->rows, bt->off.as< int32_t >(), bt->col.as< int32_t >(), bt->val.as< double >(),
                                     bt->diag.as< double >() );
      B2S_TRY_CUDA( cudaGetLastError() );
   }
   B2S_TRY( bt->nrhs.alloc( std::max( nsys, 1 ) * sizeof( int32_t ) ) );
   B2S_TRY( bt->vec_off.alloc( std::max( nsys, 1 ) * sizeof( int64_t ) ) );
   B2S_TRY( bt->rhs_off.alloc( std::max( nsys, 1 ) * sizeof( int64_t ) ) );
   B2S_TRY( bt->order.alloc( std::max( nsys, 1 ) * sizeof( int32_t ) ) );
   if( nsys > 0 ) {
      B2S_TRY( copy_h2d( bt->nrhs.p, bt->nrhs_h.data(), nsys * sizeof( int32_t ), s ) );
      B2S_TRY( copy_h2d( bt->vec_off.p, bt->vec_off_h.data(), nsys * sizeof( int64_t ), s ) );
      B2S_TRY( copy_h2d( bt->rhs_off.p, bt->rhs_off_h.data(), nsys * sizeof( int64_t ), s ) );
      B2S_TRY( copy_h2d( bt->order.p, order.data(), nsys * sizeof( int32_t ), s ) );
   }
   const size_t vb = (size_t) std::max< int64_t >( bt->nvec, 1 ) * sizeof( double );
   B2S_TRY( bt->R.alloc( vb ) );
   B2S_TRY( bt->P.alloc( vb ) );
   B2S_TRY( bt->AP.alloc( vb ) );
   if( ! bt->counter.p )
      B2S_TRY( bt->counter.alloc( 64 ) );
   B2S_TRY( bt->it_out.alloc( std::max< int64_t >( bt->nslots, 1 ) * sizeof( int64_t ) ) );
   B2S_TRY( bt->res_out.alloc( std::max< int64_t >( bt->nslots, 1 ) * sizeof( double ) ) );
   B2S_TRY( bt->status_out.alloc( std::max< int64_t >( bt->nslots, 1 ) * sizeof( int32_t ) ) );
   B2S_TRY_CUDA( cudaStreamSynchronize( s ) );
   bt->cluster = bt->o.cluster_size;
   *out = bt.release();
   return B2S_OK;
}

b2s_status
b2s_batch_destroy( b2s_batch b )
{
   clear_error();
   delete b;
   return B2S_OK;
}

b2s_status
b2s_batch_solve( b2s_batch bt, const double* B, double* X, b2s_stream stream, b2s_batch_report* report )
{
   clear_error();
   B2S_CHECK_ARG( bt && ( bt->nvec == 0 || ( B && X ) ), "NULL argument" );
   cudaStream_t s = as_stream( stream );
   b2s_batch_report rep{};
   if( bt->nsys == 0 ) {
      if( report )
         *report = rep;
      return B2S_OK;
   }
   if( bt->cluster == 0 ) {
      // autotune on copies of the initial guess so X is untouched
      DevBuf xs;
      B2S_TRY( xs.alloc( bt->nvec * sizeof( double ) ) );
      int best = 1;
      B2S_TRY( autotune_cluster( bt, B, X, xs.as< double >(), s, best ) );
      B2S_TRY_CUDA( cudaStreamSynchronize( s ) );
      bt->cluster = best;
   }
   cudaEvent_t e0, e1;
   B2S_TRY_CUDA( cudaEventCreate( &e0 ) );
   B2S_TRY_CUDA( cudaEventCreate( &e1 ) );
   cudaEventRecord( e0, s );
   b2s_status st = launch_batch( bt, B, X, bt->cluster, bt->nsys, bt->o.max_iterations, s );
   cudaEventRecord( e1, s );
   if( st == B2S_OK ) {
      cudaError_t e = cudaEventSynchronize( e1 );
      if( e != cudaSuccess ) {
         set_error( "batched solve: %s", cudaGetErrorString( e ) );
         st = B2S_CUDA_ERROR;
      }
   }
   float ms = 0;
   if( st == B2S_OK )
      cudaEventElapsedTime( &ms, e0, e1 );
   cudaEventDestroy( e0 );
   cudaEventDestroy( e1 );
   if( st != B2S_OK )
      return st;
   std::vector< int64_t > its( bt->nslots );
   std::vector< double > res( bt->nslots );
   std::vector< int32_t > sts( bt->nslots );
   B2S_TRY( copy_d2h( its.data(), bt->it_out.p, bt->nslots * sizeof( int64_t ), s ) );
   B2S_TRY( copy_d2h( res.data(), bt->res_out.p, bt->nslots * sizeof( double ), s ) );
   B2S_TRY( copy_d2h( sts.data(), bt->status_out.p, bt->nslots * sizeof( int32_t ), s ) );
   rep.device_ms = ms;
   rep.cluster_size = bt->cluster;
   rep.solves = bt->nslots;
   for( int64_t i = 0; i < bt->nslots; i++ ) {
      rep.total_iterations += its[ i ];
      rep.max_iterations = std::max< int64_t >( rep.max_iterations, its[ i ] );
      rep.max_residue = std::max( rep.max_residue, res[ i ] );
      if( sts[ i ] == B2S_OK )
         rep.converged++;
   }
   if( report )
      *report = rep;
   return rep.converged == bt->nslots ? B2S_OK : B2S_NOT_CONVERGED;
}

b2s_status
b2s_batch_results( b2s_batch bt, int64_t* iterations, double* residues, int32_t* statuses )
{
   clear_error();
   B2S_CHECK_ARG( bt, "NULL batch" );
   if( iterations )
      B2S_TRY( copy_d2h( iterations, bt->it_out.p, bt->nslots * sizeof( int64_t ), nullptr ) );
   if( residues )
      B2S_TRY( copy_d2h( residues, bt->res_out.p, bt->nslots * sizeof( double ), nullptr ) );
   if( statuses )
      B2S_TRY( copy_d2h( statuses, bt->status_out.p, bt->nslots * sizeof( int32_t ), nullptr ) );
   return B2S_OK;
}

}  // extern "C"
