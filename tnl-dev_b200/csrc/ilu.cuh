// ILU(0) on the device: Preconditioners::ILU0 (Solvers/Linear/Preconditioners/ILU0.hpp:23-144)
// with its triangular solves (Solvers/Linear/Utils/TriangularSolve.h:24-110).
//
// The factors live in the pattern of A (CSR, rows sorted by column, diagonal
// stored): L with a unit diagonal strictly below, U on and above it.
//
// Both the factorization and the substitutions are sequential along
// dependency chains. They run as "sync-free" persistent kernels: a warp takes
// the next row from a ticket counter, waits until every row it depends on has
// published its result (a per-row flag holding the current pass's epoch),
// computes, and publishes its own row. Tickets hand the rows out level by
// level (the level of a row is one more than the deepest row it depends on,
// computed once when the factors are built), so every awaited row was claimed
// earlier by a warp that is already running, and all rows of a level are in
// flight together — the critical path is the number of levels, not the
// number of rows. Every wait is bounded: after kIluSpinLimit polls the warp
// raises the error word and returns, and the others leave as soon as they see
// it; the host turns the word into B2S_TIMEOUT.
//
// The substitutions of factors with short rows run by blocks of rows instead
// (ilu_block_trsv_kernel).
//
// Arithmetic follows TNL's loops element by element: for row i and each of
// its L entries k in increasing order, L_ik = L_ik / U_kk and every later
// entry j of the row takes L_ik * U_kj off (U_kj = 0 when absent); the
// substitutions subtract L_ij x_j (U_ij x_j) in increasing j and divide by
// U_ii last. The reference build (g++ -O3 -march=x86-64-v3) contracts the
// factorization updates into fused multiply-adds, leaves the FP64
// substitution sums uncontracted and vectorizes the FP32 ones by four with a
// fused remainder; the kernels evaluate every term the same way, so the
// results are TNL's bit for bit.
#pragma once

#include "b2s_internal.cuh"

#include <cstddef>
#include <type_traits>
#include <vector>

namespace b2s {

constexpr int kIluBlock = 256;
constexpr int kIluSpinLimit = 1 << 21;

struct IluState
{
   unsigned int ticket;  // next row (warp-per-row kernels) or block of rows to claim
   int epoch;            // the current pass; a row is done when its flag equals it
   int error;            // 1: a bounded wait gave up
   int skip;             // the current pass is gated off
};

template< typename Real >
struct IluView
{
   int32_t n;
   const int32_t* off;
   const int32_t* col;
   const int32_t* diag;  // position of A_ii in each row
   const int32_t* ord_l; // rows by level of L (the factorization and L^-1), -1 padded
   const int32_t* ord_u; // rows by level of U (U^-1), -1 padded
   int32_t n_l, n_u;     // lengths of the padded lists
   Real* lu;
   int32_t* flags;
   IluState* st;
};

struct NoGate
{
   __device__ bool skip() const { return false; }
};

// a multiply-subtract the way the reference build evaluates it
template< bool FUSED >
__device__ __forceinline__ double
msub( double a, double l, double u )
{
   return FUSED ? __fma_rn( -l, u, a ) : __dsub_rn( a, __dmul_rn( l, u ) );
}
template< bool FUSED >
__device__ __forceinline__ float
msub( float a, float l, float u )
{
   return FUSED ? __fmaf_rn( -l, u, a ) : __fsub_rn( a, __fmul_rn( l, u ) );
}
// Term q of the m terms of a substitution row, as the reference build sums
// it: FP64 products rounded, then subtracted; FP32 vectorized by four
// (rounded products subtracted in order) with the m mod 4 remaining terms
// fused.
template< typename Real >
__device__ __forceinline__ Real
sum_term( Real acc, Real v, Real xv, int q, int m )
{
   if constexpr( std::is_same< Real, float >::value ) {
      if( q >= m / 4 * 4 )
         return msub< true >( acc, v, xv );
   }
   return msub< false >( acc, v, xv );
}

__device__ __forceinline__ int
ld_acquire( const int32_t* p )
{
   int v;
   asm volatile( "ld.acquire.gpu.global.b32 %0, [%1];" : "=r"( v ) : "l"( p ) : "memory" );
   return v;
}
__device__ __forceinline__ void
st_release( int32_t* p, int v )
{
   asm volatile( "st.release.gpu.global.b32 [%0], %1;" ::"l"( p ), "r"( v ) : "memory" );
}

// bounded wait until row `j` has published in this epoch
__device__ __forceinline__ bool
ilu_wait( const int32_t* flag, int epoch, IluState* st )
{
   for( int it = 0; it < kIluSpinLimit; it++ ) {
      if( ld_acquire( flag ) == epoch )
         return true;
      if( ( it & 255 ) == 255 && *(volatile int*) &st->error )
         return false;
   }
   atomicExch( &st->error, 1 );
   return false;
}

// a new pass of the warp-per-row kernels: tickets from 0, a fresh epoch
template< class Gate >
__global__ void
ilu_begin_kernel( IluState* st, Gate gate )
{
   const bool off = gate.skip();
   st->skip = off ? 1 : 0;
   if( off )
      return;
   st->ticket = 0;
   st->epoch += 1;
}

// Rows per level are padded with -1 to a multiple of kIluRows in the
// level-ordered lists (1: no padding; the kernels skip -1 entries).
constexpr int kIluRows = 1;

// the factorization, one warp per row, in level order
template< typename Real >
__global__ void __launch_bounds__( kIluBlock )
ilu_factor_kernel( IluView< Real > L )
{
   const int lane = threadIdx.x & 31;
   IluState* st = L.st;
   const int epoch = *(volatile int*) &st->epoch;
   for( ;; ) {
      unsigned t = 0;
      if( lane == 0 )
         t = atomicAdd( &st->ticket, 1u );
      t = __shfl_sync( 0xffffffffu, t, 0 );
      if( t >= (unsigned) L.n_l )
         return;
      const int i = L.ord_l[ t ];
      if( i < 0 )
         continue;  // padding of a level
      const int b = L.off[ i ], e = L.off[ i + 1 ], d = L.diag[ i ];
      for( int ck = b; ck < d; ck++ ) {
         const int k = L.col[ ck ];  // k < i, an earlier level
         int ok = 1;
         if( lane == 0 )
            ok = ilu_wait( L.flags + k, epoch, st );
         if( ! __shfl_sync( 0xffffffffu, ok, 0 ) )
            return;
         const int dk = L.diag[ k ], ek = L.off[ k + 1 ];
         Real lik = 0;
         if( lane == 0 ) {
            lik = __ldcg( L.lu + ck ) / __ldcg( L.lu + dk );
            L.lu[ ck ] = lik;
         }
         lik = __shfl_sync( 0xffffffffu, lik, 0 );
         for( int cj = ck + 1 + lane; cj < e; cj += 32 ) {
            const int j = L.col[ cj ];
            int lo = dk, hi = ek;  // U part of row k: columns >= k, sorted
            while( lo < hi ) {
               const int mid = ( lo + hi ) >> 1;
               if( L.col[ mid ] < j )
                  lo = mid + 1;
               else
                  hi = mid;
            }
            const Real u = ( lo < ek && L.col[ lo ] == j ) ? __ldcg( L.lu + lo ) : Real( 0 );
            L.lu[ cj ] = msub< true >( __ldcg( L.lu + cj ), lik, u );
         }
         __syncwarp();
      }
      __threadfence();
      __syncwarp();
      if( lane == 0 )
         st_release( L.flags + i, epoch );
   }
}

// x = L^-1 b (UPPER = false, unit diagonal) or x = U^-1 b (UPPER = true),
// one warp per row in level order (lanes wait for the row's dependencies in
// parallel; the sum runs in TNL's order through shuffles); x may be b.
// PLAIN: every term a rounded product subtracted in order (the ILUT
// substitutions, whose loops the reference build does not vectorize).
// Serves factors whose rows are long or too many for the block kernel below.
template< typename Real, bool UPPER, bool PLAIN = false >
__global__ void __launch_bounds__( kIluBlock )
ilu_trsv_kernel( IluView< Real > L, const Real* b, Real* x )
{
   const int lane = threadIdx.x & 31;
   IluState* st = L.st;
   if( *(volatile int*) &st->skip )
      return;
   const int epoch = *(volatile int*) &st->epoch;
   const int32_t* ord = UPPER ? L.ord_u : L.ord_l;
   const int32_t nord = UPPER ? L.n_u : L.n_l;
   for( ;; ) {
      unsigned t = 0;
      if( lane == 0 )
         t = atomicAdd( &st->ticket, 1u );
      t = __shfl_sync( 0xffffffffu, t, 0 );
      if( t >= (unsigned) nord )
         return;
      const int i = ord[ t ];
      if( i < 0 )
         continue;  // padding of a level
      const int d = L.diag[ i ];
      const int b0 = UPPER ? d + 1 : L.off[ i ], b1 = UPPER ? L.off[ i + 1 ] : d;
      Real acc = b[ i ];
      for( int base = b0; base < b1; base += 32 ) {
         const int k = base + lane;
         Real v = 0, xv = 0;
         int ok = 1;
         if( k < b1 ) {
            const int j = L.col[ k ];
            v = L.lu[ k ];
            ok = ilu_wait( L.flags + j, epoch, st );
            if( ok )
               xv = __ldcg( x + j );
         }
         if( ! __all_sync( 0xffffffffu, ok ) )
            return;
         const int cnt = min( 32, b1 - base );
         for( int q = 0; q < cnt; q++ ) {
            const Real vq = __shfl_sync( 0xffffffffu, v, q ), xq = __shfl_sync( 0xffffffffu, xv, q );
            acc = PLAIN ? msub< false >( acc, vq, xq ) : sum_term< Real >( acc, vq, xq, base - b0 + q, b1 - b0 );
         }
      }
      if( UPPER )
         acc = acc / L.lu[ d ];
      if( lane == 0 ) {
         x[ i ] = acc;
         __threadfence();
         st_release( L.flags + i, epoch );
      }
      __syncwarp();
   }
}

// ---------------------------------------------------------------------------
// Substitutions by blocks of rows (short rows: stencils and the like).
//
// A substitution is a chain of as many steps as there are levels, so its time
// is the latency of one step. The warp-per-row kernel above pays a flag poll,
// a load of x, a fence and a flag store through L2 for every step: 4.9 us per
// level measured on a 128^3 stencil. Here a CTA owns a contiguous block of
// rows and keeps their x in shared memory; most of a stencil row's
// dependencies are in its own block, so most steps of the chain are a store
// and a poll of shared memory.
//   * The rows of a block are ordered by level and cut into batches of at most
//     32 rows of one level, a lane per row (so no lane waits for another of
//     its warp); warp w takes batches w, w + warps, ... of its block in order.
//   * A value is its own flag, in shared memory for the block's rows and in L2
//     for the others': it starts as a signalling NaN that no operation
//     returns, and whoever needs it looks again until it is there. So a step
//     needs no fence: one would wait for the loads ahead that are in flight
//     (with a fence, a flag or a count per batch: 1,200 cycles per step). A
//     computed value with those bits (copied through from b) is stored as the
//     quiet NaN. A warp that is early looks at one word of shared memory, not
//     at all of its rows', which would keep the load pipe from the warp whose
//     turn it is. The first look at other blocks' rows goes out before that.
//   * A batch's columns, values and diagonal are stored batch by batch in slot
//     order, so a warp loads them coalesced, one and two batches ahead of the
//     one whose turn it is. Where most lanes have a row, batches are stored 32
//     lanes wide (FULL); where few rows share a level, which would take up to 32
//     times the entries, with as many lanes as they have rows. The latter takes
//     a few more instructions and one more load in a row, per batch; both
//     substitutions of 10^3 50 / 55 us, 64^3 282 / 285 us.
//   * Blocks are claimed in dependency order from a ticket counter: a claimed
//     block waits only for blocks claimed before it, whose CTAs are running.
//     The CTA that takes the last ticket puts the counter back.
//   * Both passes publish in their own scratch vector (y: L^-1 b, z: U^-1 y);
//     each pass puts the other's scratch back to the signalling NaN for the
//     next application, so there is no pass to clear them, and b may be x.
// Every wait is bounded as above. A block may wait for all blocks before it,
// so the limits grow with the steps of the chain (TrsvPlan::steps). Rows per
// block: see choose_blocks.
// Measured, both substitutions of one application through the public call
// (warp per row before): 3D stencils 10^3 177 -> 52 us, 32^3 535 -> 132 us,
// 64^3 1,106 -> 284 us, 128^3 3,748 -> 1,009 us; 2D 140^2 1,233 -> 234 us.
constexpr int kTrsvBlock = 256;                // 128 to 512 measured alike
constexpr int kTrsvWarps = kTrsvBlock / 32;
constexpr int kTrsvSlots = 4;                  // slots of the next batch loaded ahead
constexpr int kTrsvSmemMax = 200 * 1024;       // x of one block in shared memory
// Polls that a wait makes: of shared memory (30 cycles or more each) and of L2
// (300 or more), a second or so at least, and for each step of the chain the
// time of 4,000 cycles; a step of the 128^3 stencil takes 2,500.
constexpr int kTrsvSpinLocal = 1 << 26, kTrsvSpinLocalStep = 128;
constexpr int kTrsvSpinRemote = 1 << 23, kTrsvSpinRemoteStep = 16;

template< typename Real >
struct TrsvBits;
template<>
struct TrsvBits< double >
{
   using type = unsigned long long;
   static constexpr type pending = 0xFFF3B25D5EA10F0Full, quiet = 1ull << 51;
};
template<>
struct TrsvBits< float >
{
   using type = unsigned int;
   static constexpr type pending = 0xFFB1D5EAu, quiet = 1u << 22;
};
__device__ __forceinline__ unsigned long long
trsv_bits( double v )
{
   return (unsigned long long) __double_as_longlong( v );
}
__device__ __forceinline__ unsigned int
trsv_bits( float v )
{
   return __float_as_uint( v );
}
__device__ __forceinline__ double
trsv_value( unsigned long long b )
{
   return __longlong_as_double( (long long) b );
}
__device__ __forceinline__ float
trsv_value( unsigned int b )
{
   return __uint_as_float( b );
}
__device__ __forceinline__ unsigned long long
trsv_ld_remote( const unsigned long long* p )
{
   unsigned long long v;
   asm volatile( "ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"( v ) : "l"( p ) : "memory" );
   return v;
}
__device__ __forceinline__ unsigned int
trsv_ld_remote( const unsigned int* p )
{
   unsigned int v;
   asm volatile( "ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"( v ) : "l"( p ) : "memory" );
   return v;
}
__device__ __forceinline__ void
trsv_st_remote( unsigned long long* p, unsigned long long v )
{
   asm volatile( "st.relaxed.gpu.global.b64 [%0], %1;" ::"l"( p ), "l"( v ) : "memory" );
}
__device__ __forceinline__ void
trsv_st_remote( unsigned int* p, unsigned int v )
{
   asm volatile( "st.relaxed.gpu.global.b32 [%0], %1;" ::"l"( p ), "r"( v ) : "memory" );
}

// one triangle's rows in block and batch order
template< typename Real >
struct TrsvView
{
   int32_t n, rows_per_block;
   int32_t spin_local, spin_remote;
   const int32_t* bfirst;  // first batch of each block (blocks + 1 entries)
   const int4* batch;      // x: place of a batch's first lane, y: its first slot, z: lanes, w: slots per lane
   const int32_t* row;     // rows in batch order (-1: a lane without one)
   const int32_t* len;     // their dependencies
   const int32_t* col;     // slot k of lane l of a batch at y + k * z + l
   const Real* val;
   const Real* dg;         // U_ii of the rows in batch order (upper only)
};

template< typename Real, bool UPPER, bool PLAIN, bool FULL, class Gate >
__global__ void __launch_bounds__( kTrsvBlock, 1 )
ilu_block_trsv_kernel( TrsvView< Real > T, IluState* st, const Real* b, typename TrsvBits< Real >::type* pub,
                       typename TrsvBits< Real >::type* other, Real* x, Gate gate )
{
   using Bits = typename TrsvBits< Real >::type;
   constexpr Bits pending = TrsvBits< Real >::pending;
   extern __shared__ __align__( 16 ) unsigned char trsv_smem[];
   Bits* xs = reinterpret_cast< Bits* >( trsv_smem );
   __shared__ int s_block;
   if( gate.skip() )
      return;
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   if( threadIdx.x == 0 ) {
      const unsigned t = atomicAdd( &st->ticket, 1u );
      if( t == gridDim.x - 1 )
         atomicExch( &st->ticket, 0u );
      s_block = UPPER ? (int) ( gridDim.x - 1 - t ) : (int) t;
   }
   __syncthreads();
   const int blk = s_block;
   const int c0 = blk * T.rows_per_block, c1 = min( T.n, c0 + T.rows_per_block );
   for( int i = threadIdx.x; i < c1 - c0; i += kTrsvBlock ) {
      xs[ i ] = pending;
      if( ! UPPER )
         other[ c0 + i ] = pending;
   }
   __syncthreads();
   const int last = T.bfirst[ blk + 1 ];
   bool ok = true;  // false once a wait gave up: this lane waits no more
   // a batch's lane: loaded three batches (head; two if FULL), two (meta) and one
   // (slots, right-hand side) ahead of its turn, so that no turn waits for them
   struct Meta
   {
      int row, len, slot, rows, width;
      Real dg;
   };
   struct Slots
   {
      Real b, val[ kTrsvSlots ];
      int col[ kTrsvSlots ];
   };
   auto load_head = [ & ]( int q ) { return q < last ? __ldg( T.batch + q ) : make_int4( 0, 0, 0, 0 ); };
   auto load_meta = [ & ]( int q, const int4& head )
   {
      Meta m{ -1, 0, 0, 0, 0, Real( 1 ) };
      if( FULL ? q < last : lane < head.z ) {
         const int at = FULL ? 32 * q + lane : head.x + lane;
         m.row = __ldg( T.row + at );
         m.len = __ldg( T.len + at );
         if( UPPER )
            m.dg = __ldg( T.dg + at );
      }
      const int4 h = FULL ? load_head( q ) : head;
      m.slot = h.y + lane;
      m.rows = FULL ? 32 : h.z;
      m.width = h.w;
      return m;
   };
   auto load_slots = [ & ]( const Meta& m, int k0, Slots& s )
   {
      const int step = FULL ? 32 : m.rows, g = m.slot + k0 * step;
#pragma unroll
      for( int k = 0; k < kTrsvSlots; k++ ) {
         s.col[ k ] = c0;  // no element: a place of this block
         s.val[ k ] = 0;
         if( k0 + k < m.len ) {
            s.col[ k ] = __ldg( T.col + g + k * step );
            s.val[ k ] = __ldg( T.val + g + k * step );
         }
      }
   };
   int q = T.bfirst[ blk ] + warp;
   const int4 none = make_int4( 0, 0, 0, 0 );
   Meta next = load_meta( q, FULL ? none : load_head( q ) );
   Meta after = load_meta( q + kTrsvWarps, FULL ? none : load_head( q + kTrsvWarps ) );
   int4 head = FULL ? none : load_head( q + 2 * kTrsvWarps );
   Slots ahead;
   auto load_ahead = [ & ]()
   {
      load_slots( next, 0, ahead );
      ahead.b = next.row >= 0 ? __ldcg( b + next.row ) : Real( 0 );
   };
   load_ahead();
   for( ; q < last; q += kTrsvWarps ) {
      const Meta m = next;
      Slots s = ahead;
      Real acc = s.b;
      // where the slots' values are: in xs, or (at < 0) in another block's,
      // whose first look goes out now
      Bits xr[ kTrsvSlots ];
      int at[ kTrsvSlots ];
      auto look = [ & ]( int k0 )
      {
#pragma unroll
         for( int k = 0; k < kTrsvSlots; k++ ) {
            const unsigned i = (unsigned) ( s.col[ k ] - c0 );
            const bool in = k0 + k < m.len, mine = i < (unsigned) ( c1 - c0 );
            at[ k ] = in && mine ? (int) i : -1;
            xr[ k ] = 0;
            if( in && ! mine )
               xr[ k ] = trsv_ld_remote( pub + s.col[ k ] );
         }
      };
      look( 0 );
      next = after;
      load_ahead();
      after = load_meta( q + 2 * kTrsvWarps, head );
      if( ! FULL )
         head = load_head( q + 3 * kTrsvWarps );
      for( int k0 = 0; k0 < m.width; k0 += kTrsvSlots ) {
         if( k0 > 0 ) {
            load_slots( m, k0, s );
            look( k0 );
         }
         // one value stands for the warp's: while it is missing the warp polls
         // a single word
         int some = -1;
#pragma unroll
         for( int k = 0; k < kTrsvSlots; k++ )
            some = max( some, at[ k ] );
         const unsigned have = __ballot_sync( 0xffffffffu, some >= 0 );
         if( have ) {
            some = __shfl_sync( 0xffffffffu, some, __ffs( have ) - 1 );
            for( int it = 0; *(volatile Bits*) &xs[ some ] == pending && ok; it++ )
               if( ( it & 1023 ) == 1023 && ( it >= T.spin_local || *(volatile int*) &st->error ) ) 
                  ok = false;
         }
         // The step's latency is what counts from here to the store of x: no
         // branches that part the warp, loads of shared memory side by side.
         Bits xv[ kTrsvSlots ];
         bool wait;
         int it = 0;
         do {
            wait = false;
#pragma unroll
            for( int k = 0; k < kTrsvSlots; k++ ) {
               xv[ k ] = *(volatile Bits*) &xs[ max( at[ k ], 0 ) ];
               if( xr[ k ] == pending )
                  xr[ k ] = trsv_ld_remote( pub + s.col[ k ] );
            }
#pragma unroll
            for( int k = 0; k < kTrsvSlots; k++ ) {
               xv[ k ] = at[ k ] < 0 ? xr[ k ] : xv[ k ];
               wait = wait || xv[ k ] == pending;
            }
            if( ( ++it & 255 ) == 0 && ( it >= T.spin_remote || *(volatile int*) &st->error ) ) 
               ok = false;
         } while( __any_sync( 0xffffffffu, wait && ok ) );
#pragma unroll
         for( int k = 0; k < kTrsvSlots; k++ ) {
            const Real x_k = trsv_value( xv[ k ] );
            const Real t = PLAIN ? msub< false >( acc, s.val[ k ], x_k ) : sum_term< Real >( acc, s.val[ k ], x_k, k0 + k, m.len );
            acc = k0 + k < m.len ? t : acc;
         }
      }
      if( UPPER )
         acc = acc / m.dg;
      Bits r = trsv_bits( acc );
      if( r == pending )
         r |= TrsvBits< Real >::quiet;
      if( m.row >= 0 ) {
         *(volatile Bits*) &xs[ m.row - c0 ] = r;
         trsv_st_remote( pub + m.row, r );
         if( UPPER ) {
            x[ m.row ] = trsv_value( r );
            other[ m.row ] = pending;  // this pass has read its right-hand side
         }
      }
   }
   if( ! ok )
      atomicExch( &st->error, 1 );
}

// the packed rows of one triangle (slots, lengths, diagonal) from the factors,
// a warp per batch
template< typename Real, bool UPPER >
__global__ void
trsv_pack_kernel( int32_t batches, const int4* __restrict__ batch, const int32_t* __restrict__ row,
                  const int32_t* __restrict__ off, const int32_t* __restrict__ diag, const int32_t* __restrict__ col,
                  const Real* __restrict__ lu, int32_t* __restrict__ len, int32_t* __restrict__ pcol,
                  Real* __restrict__ pval, Real* __restrict__ dg )
{
   const int64_t lanes = 32 * (int64_t) batches;
   for( int64_t t = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; t < lanes; t += (int64_t) gridDim.x * blockDim.x ) {
      const int4 h = batch[ t >> 5 ];
      const int l = (int) ( t & 31 );
      if( l >= h.z )
         continue;
      const int i = row[ h.x + l ];
      if( i < 0 ) {
         len[ h.x + l ] = 0;
         if( UPPER )
            dg[ h.x + l ] = 1;
         continue;
      }
      const int d = diag[ i ];
      const int b0 = UPPER ? d + 1 : off[ i ], b1 = UPPER ? off[ i + 1 ] : d;
      const int g = h.y + l;
      for( int k = b0; k < b1; k++ ) {
         pcol[ g + ( k - b0 ) * h.z ] = col[ k ];
         pval[ g + ( k - b0 ) * h.z ] = lu[ k ];
      }
      len[ h.x + l ] = b1 - b0;
      if( UPPER )
         dg[ h.x + l ] = lu[ d ];
   }
}

template< typename Bits >
__global__ void
trsv_clear_kernel( Bits* y, int64_t count, Bits v )
{
   for( int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < count; i += (int64_t) gridDim.x * blockDim.x )
      y[ i ] = v;
}

// One triangle in block and batch order (empty: the warp-per-row kernel runs).
template< typename Real >
struct TrsvPlan
{
   DevBuf bfirst, batch, row, len, col, val, dg;
   int32_t batches = 0;
   bool full = false;  // 32 lanes to every batch
   int64_t steps = 0;  // of the chain: over the levels, the longest row's in groups of kTrsvSlots

   static int32_t limit( int64_t base, int64_t per_step, int64_t steps )
   {
      return (int32_t) std::min< int64_t >( base + per_step * steps, 1 << 30 );
   }

   // looks: the polls after which a wait gives up (0: by the chain's length)
   TrsvView< Real > view( int32_t n, int32_t rows_per_block, int32_t looks ) const
   {
      return TrsvView< Real >{ n,
                               rows_per_block,
                               looks > 0 ? looks : limit( kTrsvSpinLocal, kTrsvSpinLocalStep, steps ),
                               looks > 0 ? looks : limit( kTrsvSpinRemote, kTrsvSpinRemoteStep, steps ),
                               bfirst.as< int32_t >(),
                               batch.as< int4 >(),
                               row.as< int32_t >(),
                               len.as< int32_t >(),
                               col.as< int32_t >(),
                               val.as< Real >(),
                               dg.as< Real >() };
   }
};

// The factors of one matrix in one value type, with their pass state.
template< typename Real >
struct IluFactors
{
   int32_t n = 0;
   DevBuf off_own, col_own;  // the CSR pattern when A is not CSR
   const int32_t* off = nullptr;
   const int32_t* col = nullptr;
   DevBuf diag, ord_l, ord_u, lu, flags, state;
   int grid = 0;
   int levels_l = 0, levels_u = 0;  // depth of the dependency chains
   int32_t n_ord_l = 0, n_ord_u = 0;
   bool plain_sum = false;  // ILUT factors: substitution terms subtracted one by one
   // substitutions by blocks of rows (blocks == 0: warp per row)
   TrsvPlan< Real > plan_l, plan_u;
   DevBuf yz;  // the two passes' scratch vectors
   int32_t blocks = 0, rows_per_block = 0;
   int32_t looks = 0;  // polls after which a wait of theirs gives up (0: by the chain's length)

   IluView< Real > view() const
   {
      return IluView< Real >{ n,         off,       col, diag.as< int32_t >(), ord_l.as< int32_t >(), ord_u.as< int32_t >(),
                              n_ord_l,   n_ord_u,   lu.as< Real >(),      flags.as< int32_t >(),  state.as< IluState >() };
   }

   // x = U^-1 L^-1 b on `s` (no synchronization; x may be b)
   template< class Gate = NoGate >
   b2s_status apply( const Real* b, Real* x, cudaStream_t s, Gate gate = Gate() ) const
   {
      if( n == 0 )
         return B2S_OK;
      if( blocks > 0 )
         return plain_sum ? apply_blocks< true >( b, x, s, gate ) : apply_blocks< false >( b, x, s, gate );
      const IluView< Real > v = view();
      ilu_begin_kernel< Gate ><<< 1, 1, 0, s >>>( v.st, gate );
      if( plain_sum )
         ilu_trsv_kernel< Real, false, true ><<< grid, kIluBlock, 0, s >>>( v, b, x );
      else
         ilu_trsv_kernel< Real, false ><<< grid, kIluBlock, 0, s >>>( v, b, x );
      ilu_begin_kernel< Gate ><<< 1, 1, 0, s >>>( v.st, gate );
      if( plain_sum )
         ilu_trsv_kernel< Real, true, true ><<< grid, kIluBlock, 0, s >>>( v, x, x );
      else
         ilu_trsv_kernel< Real, true ><<< grid, kIluBlock, 0, s >>>( v, x, x );
      B2S_TRY_CUDA( cudaGetLastError() );
      return B2S_OK;
   }

   template< bool PLAIN, class Gate >
   b2s_status apply_blocks( const Real* b, Real* x, cudaStream_t s, Gate gate ) const
   {
      using Bits = typename TrsvBits< Real >::type;
      Bits *y = yz.as< Bits >(), *z = y + n;
      const size_t smem = (size_t) rows_per_block * sizeof( Real );
      const Real* yr = reinterpret_cast< const Real* >( y );
      B2S_TRY( ( plan_l.full ? pass< false, PLAIN, true >( plan_l, b, y, z, x, smem, s, gate )
                             : pass< false, PLAIN, false >( plan_l, b, y, z, x, smem, s, gate ) ) );
      return plan_u.full ? pass< true, PLAIN, true >( plan_u, yr, z, y, x, smem, s, gate )
                         : pass< true, PLAIN, false >( plan_u, yr, z, y, x, smem, s, gate );
   }

   template< bool UPPER, bool PLAIN, bool FULL, class Bits, class Gate >
   b2s_status pass( const TrsvPlan< Real >& P, const Real* b, Bits* pub, Bits* other, Real* x, size_t smem, cudaStream_t s,
                    Gate gate ) const
   {
      auto kern = ilu_block_trsv_kernel< Real, UPPER, PLAIN, FULL, Gate >;
      B2S_TRY( allow_smem( reinterpret_cast< const void* >( kern ), smem ) );
      kern<<< blocks, kTrsvBlock, smem, s >>>( P.view( n, rows_per_block, looks ), state.as< IluState >(), b, pub, other, x,
                                               gate );
      B2S_TRY_CUDA( cudaGetLastError() );
      return B2S_OK;
   }

   // both scratch vectors to the pending value
   b2s_status clear_scratch( cudaStream_t s ) const
   {
      using Bits = typename TrsvBits< Real >::type;
      trsv_clear_kernel< Bits ><<< 256, 256, 0, s >>>( yz.as< Bits >(), 2 * (int64_t) n, TrsvBits< Real >::pending );
      B2S_TRY_CUDA( cudaGetLastError() );
      return B2S_OK;
   }

   // B2S_TIMEOUT when a bounded wait gave up since the last check (the word is reset)
   b2s_status check( cudaStream_t s ) const
   {
      if( n == 0 )
         return B2S_OK;
      IluState h{};
      B2S_TRY( copy_d2h( &h, state.p, sizeof( IluState ), s ) );
      if( h.error ) {
         const int zero = 0;
         B2S_TRY( copy_h2d( reinterpret_cast< char* >( state.p ) + offsetof( IluState, error ), &zero, sizeof( int ), s ) );
         if( blocks > 0 )
            B2S_TRY( clear_scratch( s ) );
         set_error( "ILU(0): a bounded wait for a dependency gave up" );
         return B2S_TIMEOUT;
      }
      return B2S_OK;
   }
};

// Factorize A (values in Real: A's own or its FP32 copy). Defined in ilu.cu.
template< typename Real >
b2s_status ilu_factorize( const b2s_matrix_t* A, const Real* values, IluFactors< Real >& F, cudaStream_t s );

// The level orders of F's L and U dependency graphs from the host copy of its
// pattern (hdiag: the first U position of each row), the pass state, and the
// block plans where the rows suit them.
template< typename Real >
b2s_status ilu_levels( IluFactors< Real >& F, const std::vector< int32_t >& hoff, const std::vector< int32_t >& hcol,
                       const std::vector< int32_t >& hdiag, cudaStream_t s );

// The block plans' slots from the computed factors.
template< typename Real >
b2s_status ilu_pack( IluFactors< Real >& F, cudaStream_t s );

// ILUT( p, tau ) factors of A in the ILU(0) factor structure, applied by the
// same kernels with PLAIN sums (ilut.cu).
template< typename Real >
b2s_status ilut_factorize( const b2s_matrix_t* A, int32_t p, double tau, IluFactors< Real >& F, cudaStream_t s );

}  // namespace b2s
