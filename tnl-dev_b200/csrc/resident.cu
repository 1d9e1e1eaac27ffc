// CG (CG.hpp:60-101) and BiCGStab (BICGStab.hpp:58-116) iterations of systems
// that fit on chip, as one cooperative kernel over one block per SM.
//
// Small systems are bound by latency: the graph of krylov.cu runs three
// (CG) to five (BiCGStab) kernels per iteration, each of which starts, waits
// for its last block's reduction and drains, about 5 us apiece whatever the
// size. Here a block owns a contiguous range of rows for the whole run of
// iterations: their matrix elements sit in its shared memory, their vector
// elements in its registers, and blocks meet only where a dot product needs
// all of them.
//   * A meeting: each block stores its partial sums, counts itself in, waits
//     for the count and adds all blocks' sums in block order, so every block
//     takes the same decisions. It measures 2.7 us with 148 blocks (polling
//     every block's sum in place of one count: 5.6 us, 148 readers to a line).
//     Up to kClusterRows rows the blocks are one thread-block cluster that
//     meets in distributed shared memory.
//   * The gathers form the direction at each column from vectors that are
//     complete (CG: z + beta p, BiCGStab: r + beta p - beta omega Ap and
//     r - alpha Ap), with p and Ap in two copies used in turn, so the
//     direction and s updates need no meeting of their own: two meetings per
//     CG iteration, three per BiCGStab iteration. Every element is the same
//     expression wherever it is formed, so results do not depend on it.
// Every wait is bounded: after kMeetSpin polls a block marks the count and
// leaves, as do the others when they see the mark. The mark is set only while
// the count is short of the meeting, so at the last meeting either every block
// goes on and writes its part of the result or none does, and the host goes
// on from the state before the launch with the graph of kernels.
// Measured per iteration, graph of kernels before: CG in FP64 32^2 11.5 -> 3.4
// us, 256^2 12.2 -> 7.1 us, 500^2 18.4 -> 12.7 us; BiCGStab 10^3 19.7 -> 7.8 us.
#include "resident.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace b2s {

constexpr int kResBlock = 512;
// Rows of a block: eight per thread, four for BiCGStab in FP64, whose vectors
// no longer fit the registers with eight (70^3 rows: 47 us per iteration
// against 41 us of the graph of kernels).
constexpr int kResMaxRows = 8 * kResBlock;
constexpr int kResMaxRowsBicg64 = 4 * kResBlock;
constexpr int kResMaxBlocks = 256;             // slots per set and value
constexpr int kResSmemMax = 200 * 1024;
constexpr int kMeetSpin = 1 << 22;             // polls of L2, 290 cycles or more each: 0.6 s or more
constexpr unsigned long long kMeetOff = 1ull << 63;  // in the count: a block gave up
constexpr int kClusterBlocks = 8;
// Rows up to which one cluster takes the system, four to a thread of its eight
// blocks (CG, 1,024 rows: 3.4 us per iteration)
constexpr int kClusterRows = 16384;
static_assert( kClusterRows <= 4 * kClusterBlocks * kResBlock, "four rows per thread" );
// Beyond one cluster, blocks take at most this many rows while there are SMs
// for more blocks, then equal shares.
constexpr int kResBlockRows = 256;
struct MeetSlots
{
   double v[ 2 ][ 2 ][ kResMaxBlocks ];  // [meeting's parity][value][block]
   unsigned long long count;             // blocks counted in, over all meetings of all launches
   unsigned long long base;              // `count` before this launch
};

__device__ __forceinline__ void
meet_fence()
{
   asm volatile( "fence.acq_rel.gpu;" ::: "memory" );
}

// element k of row r at base + stride * k, k < cap; column -1: none
struct RowCursor
{
   int32_t format, alignedSize, segmentSize, shift;
   const int32_t* offsets;
   __device__ __forceinline__ void
   row( int r, int64_t& base, int& stride, int& cap ) const
   {
      if( format == B2S_CSR ) {
         base = offsets[ r ];
         stride = 1;
         cap = offsets[ r + 1 ] - offsets[ r ];
      }
      else if( format == B2S_ELLPACK ) {
         base = r;
         stride = alignedSize;
         cap = segmentSize;
      }
      else {
         const int s = r >> shift;
         base = (int64_t) offsets[ s ] + ( r & ( ( 1 << shift ) - 1 ) );
         stride = 1 << shift;
         cap = ( offsets[ s + 1 ] - offsets[ s ] ) >> shift;
      }
   }
};

template< typename Real >
struct ResidentArgs
{
   int32_t n, rows_per_block, width;
   RowCursor rows;
   const int32_t* col;
   const Real* val;
   const Real* diag;
   ResidentVecs< Real > v;
   Ctl* ctl;
   MeetSlots* slots;
   int iterations, looks;
   double eps2;
};

// All blocks' sums of NV values, the same in every thread of every block;
// everything a block wrote before is visible to all after. false: gave up.
// `meeting` counts the launch's meetings; *due, thread 0's, is the slots' count
// after the last one (in shared memory: as 64 bits in registers it cost BiCGStab
// 2 %).
// `fin( totals )` runs in one thread of every block before the others go on:
// the scalar work, which every block does alike (a double division or root in
// all 16 warps takes longer than in one).
template< int NV, bool CLUSTER, class Fin >
__device__ __forceinline__ bool
meet( double ( &v )[ NV ], MeetSlots* S, int looks, unsigned& meeting, unsigned long long* due, Fin&& fin )
{
   __shared__ double sh[ NV ][ kResBlock / 32 ];
   __shared__ double part[ 2 ][ NV ];
   __shared__ int gave_up;
   const int G = (int) gridDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
   const unsigned set = meeting & 1;
#pragma unroll
   for( int k = 0; k < NV; k++ ) {
      const double s = warp_sum( v[ k ] );
      if( lane == 0 )
         sh[ k ][ warp ] = s;
   }
   __syncthreads();  // the block's stores are behind thread 0's fence (or the cluster's barrier)
   meeting++;
   if( warp == 0 ) {
#pragma unroll
      for( int k = 0; k < NV; k++ )
         v[ k ] = warp_sum( lane < kResBlock / 32 ? sh[ k ][ lane ] : 0.0 );
   }
   bool ok = true;
   if constexpr( CLUSTER ) {
      cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
      if( tid == 0 )
#pragma unroll
         for( int k = 0; k < NV; k++ )
            part[ set ][ k ] = v[ k ];
      cl.sync();
      if( warp == 0 ) {
#pragma unroll
         for( int k = 0; k < NV; k++ )
            v[ k ] = warp_sum( lane < G ? cl.map_shared_rank( &part[ 0 ][ 0 ], lane )[ set * NV + k ] : 0.0 );
      }
   }
   else {
      if( tid == 0 ) {
#pragma unroll
         for( int k = 0; k < NV; k++ )
            S->v[ set ][ k ][ blockIdx.x ] = v[ k ];
         meet_fence();
         atomicAdd( &S->count, 1ull );
         const unsigned long long want = *due += (unsigned) G;
         unsigned long long c;
         for( int it = 0; ( c = *(volatile unsigned long long*) &S->count ) < want; it++ )
            if( it >= looks && atomicCAS( &S->count, c, c | kMeetOff ) == c ) {
               c |= kMeetOff;
               break;
            }
         ok = ( c & kMeetOff ) == 0;
         meet_fence();  // what the others wrote before they counted in is read after this
         gave_up = ok ? 0 : 1;
      }
      __syncthreads();
      ok = gave_up == 0;
      if( warp == 0 ) {
#pragma unroll
         for( int k = 0; k < NV; k++ ) {
            double s = 0;
            for( int b = lane; b < G; b += 32 )
               s += __ldcg( &S->v[ set ][ k ][ b ] );
            v[ k ] = warp_sum( s );
         }
      }
   }
   if( tid == 0 )
      fin( v );
   __syncthreads();
   return ok;
}

// the block's rows in shared memory: element k of local row t at k * rows + t
template< typename Real >
__device__ __forceinline__ void
load_rows( const ResidentArgs< Real >& a, int c0, int c1, Real* sval, int32_t* scol, int* slen )
{
   for( int t = threadIdx.x; t < c1 - c0; t += kResBlock ) {
      int64_t base;
      int stride, cap, len = 0;
      a.rows.row( c0 + t, base, stride, cap );
      for( int k = 0; k < cap; k++ ) {
         const int64_t g = base + (int64_t) stride * k;
         const int c = __ldg( a.col + g );
         if( c >= 0 ) {
            scol[ len * a.rows_per_block + t ] = c;
            sval[ len * a.rows_per_block + t ] = __ldg( a.val + g );
            len++;
         }
      }
      slen[ t ] = len;
   }
}

// sum of A(row, c) * at( c ) in the row's order, W gathers in flight
template< typename Real, int W, class At >
__device__ __forceinline__ Real
row_times( const Real* sval, const int32_t* scol, int rows, int t, int len, At&& at )
{
   Real s = 0;
   for( int k0 = 0; k0 < len; k0 += W ) {
      Real xv[ W ];
#pragma unroll
      for( int i = 0; i < W; i++ )
         if( k0 + i < len )
            xv[ i ] = at( scol[ ( k0 + i ) * rows + t ] );
#pragma unroll
      for( int i = 0; i < W; i++ )
         if( k0 + i < len )
            s += sval[ ( k0 + i ) * rows + t ] * xv[ i ];
   }
   return s;
}

template< typename Real, int RPT, bool BICG, bool CLUSTER >
__global__ void __launch_bounds__( kResBlock, 1 )
resident_kernel( ResidentArgs< Real > a )
{
   extern __shared__ __align__( 16 ) unsigned char res_smem[];
   if( a.ctl->done )
      return;  // the same word for every block: only the last launch's end wrote it
   constexpr int W = RPT <= 2 ? 8 : 4;
   const int R = a.rows_per_block;
   Real* sval = reinterpret_cast< Real* >( res_smem );
   int32_t* scol = reinterpret_cast< int32_t* >( sval + (size_t) R * a.width );
   int32_t* slen = scol + (size_t) R * a.width;
   const int tid = threadIdx.x;
   const int c0 = blockIdx.x * R, c1 = min( a.n, c0 + R );
   load_rows< Real >( a, c0, c1, sval, scol, slen );
   Real x[ RPT ], r[ RPT ], p[ RPT ], Ap[ RPT ], d[ RPT ];
   int len[ RPT ];
#pragma unroll
   for( int j = 0; j < RPT; j++ ) {
      const int t = tid + j * kResBlock, i = c0 + t;
      const bool own = i < c1;
      x[ j ] = own ? a.v.x[ i ] : Real( 0 );
      r[ j ] = own ? a.v.r[ i ] : Real( 0 );
      p[ j ] = own ? a.v.p[ i ] : Real( 0 );
      Ap[ j ] = 0;
      d[ j ] = own && a.diag ? a.diag[ i ] : Real( 1 );
      len[ j ] = own ? slen[ t ] : 0;
      if( ! CLUSTER && own ) {
         a.v.r0[ i ] = r[ j ];
         a.v.p0[ i ] = p[ j ];
      }
   }
   // the iterations' scalars, the same in every block
   __shared__ Ctl c;
   if( tid == 0 )
      c = *a.ctl;
   auto give_up = [ & ]() {
      if( tid == 0 )
         a.ctl->gave_up = 1;
   };
   unsigned meeting = 0;
   __shared__ unsigned long long due;  // thread 0's: the count that the last meeting waited for
   if( tid == 0 )
      due = *(volatile unsigned long long*) &a.slots->base;
   // every block's start (its copy of ctl included) precedes any end
   {
      double one[ 1 ] = { 0.0 };
      if( ! meet< 1, CLUSTER >( one, a.slots, a.looks, meeting, &due, []( const double* ) {} ) )
         return give_up();
   }
   Real *pa = a.v.p, *pb = a.v.p2;      // p of the last direction, and the one being formed
   Real *aa = a.v.Ap, *ab = a.v.Ap2;    // BiCGStab: A p of the last direction, and the one being formed
   bool first = true, live = true;
   for( int iter = 0; iter < a.iterations && live; iter++ ) {
      if constexpr( ! BICG ) {
         // p = z + beta p (formed at the end of the last iteration in `p`, here at the columns)
         const Real beta = (Real) c.beta;
         const Real* z = a.diag ? a.v.z : a.v.r;
         double acc[ 1 ] = { 0.0 };
#pragma unroll
         for( int j = 0; j < RPT; j++ ) {
            const int t = tid + j * kResBlock, i = c0 + t;
            if( i >= c1 )
               continue;
            Real s;
            if( first )
               s = row_times< Real, W >( sval, scol, R, t, len[ j ], [ & ]( int q ) { return __ldcg( pa + q ); } );
            else {
               s = row_times< Real, W >( sval, scol, R, t, len[ j ],
                                      [ & ]( int q ) { return __ldcg( z + q ) + beta * __ldcg( pa + q ); } );
               pb[ i ] = p[ j ];
            }
            Ap[ j ] = s;
            acc[ 0 ] += (double) s * (double) p[ j ];
         }
         if( ! meet< 1, CLUSTER >( acc, a.slots, a.looks, meeting, &due, [ & ]( const double* t ) {
                // CgApSink::finish
                c.s2 = t[ 0 ];
                if( c.s2 == 0.0 ) {
                   c.residue = 0.0;
                   c.done = 1;
                   c.reason = 2;
                }
                else
                   c.alpha = c.s1 / c.s2;
             } ) )
            return give_up();
         if( ! first ) {
            Real* q = pa;
            pa = pb;
            pb = q;
         }
         first = false;
         if( c.done )
            break;
         const Real alpha = (Real) c.alpha;
         Real zz[ RPT ];
         acc[ 0 ] = 0.0;
#pragma unroll
         for( int j = 0; j < RPT; j++ ) {
            const int i = c0 + tid + j * kResBlock;
            zz[ j ] = 0;
            if( i >= c1 )
               continue;
            x[ j ] += alpha * p[ j ];
            r[ j ] = r[ j ] - alpha * Ap[ j ];
            a.v.r[ i ] = r[ j ];
            zz[ j ] = r[ j ];
            if( a.diag ) {
               zz[ j ] = r[ j ] / d[ j ];
               a.v.z[ i ] = zz[ j ];
            }
            acc[ 0 ] += (double) r[ j ] * (double) zz[ j ];
         }
         if( ! meet< 1, CLUSTER >( acc, a.slots, a.looks, meeting, &due, [ & ]( const double* t ) { CgUpdateFin{}( c, t ); } ) )
            return give_up();
         live = ! c.done;
         if( live ) {
            const Real be = (Real) c.beta;
#pragma unroll
            for( int j = 0; j < RPT; j++ )
               p[ j ] = zz[ j ] + be * p[ j ];
         }
      }
      else {
         const Real beta = (Real) c.bi_beta, bo = (Real) ( c.bi_beta * c.omega );
         double acc[ 2 ] = { 0.0, 0.0 };
#pragma unroll
         for( int j = 0; j < RPT; j++ ) {
            const int t = tid + j * kResBlock, i = c0 + t;
            if( i >= c1 )
               continue;
            Real s;
            if( first )
               s = row_times< Real, W >( sval, scol, R, t, len[ j ], [ & ]( int q ) { return __ldcg( pa + q ); } );
            else {
               s = row_times< Real, W >( sval, scol, R, t, len[ j ], [ & ]( int q ) {
                  return __ldcg( a.v.r + q ) + beta * __ldcg( pa + q ) - bo * __ldcg( aa + q );
               } );
               pb[ i ] = p[ j ];
            }
            if( a.diag )
               s = s / d[ j ];
            Ap[ j ] = s;
            ab[ i ] = s;
            acc[ 0 ] += (double) s * (double) __ldg( a.v.r_ast + i );
         }
         double a1[ 1 ] = { acc[ 0 ] };
         if( ! meet< 1, CLUSTER >( a1, a.slots, a.looks, meeting, &due,
                                   [ & ]( const double* t ) { c.bi_alpha = c.rho / t[ 0 ]; } ) )
            return give_up();
         if( ! first ) {
            Real* q = pa;
            pa = pb;
            pb = q;
         }
         first = false;
         {
            Real* q = aa;
            aa = ab;
            ab = q;
         }
         // aa: A p of this direction
         const Real alpha = (Real) c.bi_alpha;
         Real s_[ RPT ], As[ RPT ];
         acc[ 0 ] = acc[ 1 ] = 0.0;
#pragma unroll
         for( int j = 0; j < RPT; j++ ) {
            const int t = tid + j * kResBlock, i = c0 + t;
            s_[ j ] = As[ j ] = 0;
            if( i >= c1 )
               continue;
            s_[ j ] = r[ j ] - alpha * Ap[ j ];
            Real s = row_times< Real, W >( sval, scol, R, t, len[ j ],
                                        [ & ]( int q ) { return __ldcg( a.v.r + q ) - alpha * __ldcg( aa + q ); } );
            if( a.diag )
               s = s / d[ j ];
            As[ j ] = s;
            acc[ 0 ] += (double) s * (double) s_[ j ];
            acc[ 1 ] += (double) s * (double) s;
         }
         if( ! meet< 2, CLUSTER >( acc, a.slots, a.looks, meeting, &due,
                                   [ & ]( const double* t ) { c.omega = t[ 0 ] / t[ 1 ]; } ) )
            return give_up();
         const Real omega = (Real) c.omega;
         acc[ 0 ] = acc[ 1 ] = 0.0;
#pragma unroll
         for( int j = 0; j < RPT; j++ ) {
            const int i = c0 + tid + j * kResBlock;
            if( i >= c1 )
               continue;
            x[ j ] += alpha * p[ j ] + omega * s_[ j ];
            r[ j ] = s_[ j ] - omega * As[ j ];
            a.v.r[ i ] = r[ j ];
            acc[ 0 ] += (double) r[ j ] * (double) __ldg( a.v.r_ast + i );
            acc[ 1 ] += (double) r[ j ] * (double) r[ j ];
         }
         if( ! meet< 2, CLUSTER >( acc, a.slots, a.looks, meeting, &due, [ & ]( const double* t ) { BiXrFin{ a.eps2, 0 }( c, t ); } ) )
            return give_up();
         if( c.restart_flag )
            break;
         live = ! c.done;
         if( live ) {
            const Real be = (Real) c.bi_beta, bw = (Real) ( c.bi_beta * c.omega );
#pragma unroll
            for( int j = 0; j < RPT; j++ )
               p[ j ] = r[ j ] + be * p[ j ] - bw * Ap[ j ];
         }
      }
   }
   // every block has left the gathers of its last direction: the vectors may be put back
   {
      double one[ 1 ] = { 0.0 };
      if( ! meet< 1, CLUSTER >( one, a.slots, a.looks, meeting, &due, []( const double* ) {} ) )
         return give_up();
   }
#pragma unroll
   for( int j = 0; j < RPT; j++ ) {
      const int i = c0 + tid + j * kResBlock;
      if( i >= c1 )
         continue;
      a.v.x[ i ] = x[ j ];
      a.v.p[ i ] = p[ j ];
      if( BICG )
         a.v.Ap[ i ] = Ap[ j ];
   }
   if( blockIdx.x == 0 && tid == 0 ) {
      Ctl& o = *a.ctl;  // only what the iterations changed: the rest need not stay in registers
      o.residue = c.residue;
      o.it = c.it;
      o.done = c.done;
      o.reason = c.reason;
      if( BICG ) {
         o.rho = c.rho;
         o.rho_old = c.rho_old;
         o.omega = c.omega;
         o.bi_alpha = c.bi_alpha;
         o.bi_beta = c.bi_beta;
         o.restart_flag = c.restart_flag;
      }
      else {
         o.s1 = c.s1;
         o.s1_prev = c.s1_prev;
         o.s2 = c.s2;
         o.alpha = c.alpha;
         o.beta = c.beta;
      }
      a.slots->base = due;
   }
   if constexpr( CLUSTER )
      cooperative_groups::this_cluster().sync();  // the others may still read this block's sums
}

struct ResidentShape
{
   int blocks = 0, rows = 0;
   bool cluster = false;
};

// Blocks and rows per block, or blocks == 0: the matrix does not fit.
static ResidentShape
resident_shape( const b2s_matrix_t* A, int solver, size_t es )
{
   ResidentShape S;
   if( A->format != B2S_CSR && A->format != B2S_SLICED_ELLPACK && A->format != B2S_ELLPACK )
      return S;
   if( A->rows == 0 || A->max_row < 1 )
      return S;
   const int n = A->rows;
   auto fits = [ & ]( int rows ) {
      return rows <= ( solver == B2S_BICGSTAB && es == 8 ? kResMaxRowsBicg64 : kResMaxRows ) && (int64_t) rows * ( A->max_row * ( (int64_t) es + 4 ) + 4 ) <= kResSmemMax;
   };
   if( n <= kClusterRows ) {
      int blocks = 1;
      while( blocks < kClusterBlocks && blocks * kResBlock < n )
         blocks *= 2;
      const int rows = ( n + blocks - 1 ) / blocks;
      if( fits( rows ) )
         return ResidentShape{ blocks, rows, true };
   }
   const int want = std::max( 1, std::min( num_sms(), ( n + kResBlockRows - 1 ) / kResBlockRows ) );
   const int rows = ( n + want - 1 ) / want;
   if( fits( rows ) )
      return ResidentShape{ ( n + rows - 1 ) / rows, rows, false };
   return S;
}

bool
resident_fits( const b2s_matrix_t* A, int solver, size_t es )
{
   return resident_shape( A, solver, es ).blocks > 0;
}

__global__ void
slots_clear_kernel( MeetSlots* S )
{
   S->count = 0;
   S->base = 0;
}

b2s_status
resident_scratch_init( DevBuf& scratch, cudaStream_t s )
{
   if( scratch.bytes < sizeof( MeetSlots ) )
      B2S_TRY( scratch.alloc( sizeof( MeetSlots ) ) );
   slots_clear_kernel<<< 1, 1, 0, s >>>( scratch.as< MeetSlots >() );
   B2S_TRY_CUDA( cudaGetLastError() );
   return B2S_OK;
}

template< typename Real, int RPT, bool BICG, bool CLUSTER >
static b2s_status
launch_resident( const ResidentArgs< Real >& a, int blocks, cudaStream_t s )
{
   auto kern = resident_kernel< Real, RPT, BICG, CLUSTER >;
   const size_t smem = (size_t) a.rows_per_block * ( a.width * ( sizeof( Real ) + sizeof( int32_t ) ) + sizeof( int32_t ) );
   B2S_TRY( allow_smem( reinterpret_cast< const void* >( kern ), smem ) );
   cudaLaunchConfig_t cfg{};
   cudaLaunchAttribute attr[ 1 ];
   if( CLUSTER ) {
      attr[ 0 ].id = cudaLaunchAttributeClusterDimension;
      attr[ 0 ].val.clusterDim.x = blocks;
      attr[ 0 ].val.clusterDim.y = 1;
      attr[ 0 ].val.clusterDim.z = 1;
   }
   else {
      attr[ 0 ].id = cudaLaunchAttributeCooperative;
      attr[ 0 ].val.cooperative = 1;
   }
   cfg.gridDim = dim3( blocks );
   cfg.blockDim = dim3( kResBlock );
   cfg.dynamicSmemBytes = smem;
   cfg.stream = s;
   cfg.attrs = attr;
   cfg.numAttrs = 1;
   B2S_TRY_CUDA( cudaLaunchKernelEx( &cfg, kern, a ) );
   return B2S_OK;
}

template< typename Real, bool BICG, bool CLUSTER >
static b2s_status
launch_resident_rows( const ResidentArgs< Real >& a, int blocks, cudaStream_t s )
{
   const int rpt = ( a.rows_per_block + kResBlock - 1 ) / kResBlock;
   if( rpt <= 1 )
      return launch_resident< Real, 1, BICG, CLUSTER >( a, blocks, s );
   if( rpt <= 2 )
      return launch_resident< Real, 2, BICG, CLUSTER >( a, blocks, s );
   if( rpt <= 4 )
      return launch_resident< Real, 4, BICG, CLUSTER >( a, blocks, s );
   if constexpr( ! CLUSTER && ! ( BICG && sizeof( Real ) == 8 ) )  // as many as resident_shape gives
      return launch_resident< Real, 8, BICG, CLUSTER >( a, blocks, s );
   set_error( "resident solver: %d rows per block", a.rows_per_block );
   return B2S_UNSUPPORTED;
}

template< typename Real >
b2s_status
resident_iterate( const b2s_matrix_t* A, int solver, const Real* vals, const Real* diag, const ResidentVecs< Real >& v,
                  Ctl* ctl, DevBuf& scratch, int iterations, int looks, double eps2, cudaStream_t s )
{
   ResidentArgs< Real > a{};
   a.n = A->rows;
   const ResidentShape shape = resident_shape( A, solver, sizeof( Real ) );
   if( shape.blocks == 0 ) {
      set_error( "resident solver: the matrix does not fit" );
      return B2S_UNSUPPORTED;
   }
   a.rows_per_block = shape.rows;
   a.width = A->max_row;
   a.rows.format = A->format;
   a.rows.alignedSize = A->alignedSize;
   a.rows.segmentSize = A->segmentSize;
   a.rows.offsets = A->format == B2S_CSR ? A->offsets.as< int32_t >() : A->sliceOffsets.as< int32_t >();
   for( a.rows.shift = 3; ( 1 << a.rows.shift ) < A->slice_size; )
      a.rows.shift++;
   a.col = A->columns.as< int32_t >();
   a.val = vals;
   a.diag = diag;
   a.v = v;
   a.ctl = ctl;
   a.slots = scratch.as< MeetSlots >();
   a.iterations = iterations;
   a.looks = looks > 0 ? looks : kMeetSpin;
   a.eps2 = eps2;
   if( solver == B2S_BICGSTAB )
      return shape.cluster ? launch_resident_rows< Real, true, true >( a, shape.blocks, s )
                           : launch_resident_rows< Real, true, false >( a, shape.blocks, s );
   return shape.cluster ? launch_resident_rows< Real, false, true >( a, shape.blocks, s )
                        : launch_resident_rows< Real, false, false >( a, shape.blocks, s );
}

template b2s_status resident_iterate< double >( const b2s_matrix_t*, int, const double*, const double*,
                                                const ResidentVecs< double >&, Ctl*, DevBuf&, int, int, double,
                                                cudaStream_t );
template b2s_status resident_iterate< float >( const b2s_matrix_t*, int, const float*, const float*,
                                               const ResidentVecs< float >&, Ctl*, DevBuf&, int, int, double,
                                               cudaStream_t );

}  // namespace b2s
