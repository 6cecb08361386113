// FP64 kernels of the supernodal factorization and solves (sm_100a).
//
// Every kernel consumes a flat task array built by Plan::build (plan.cpp):
// one CTA per task, no inter-CTA dependencies inside a launch, so a level's
// work for all of its supernodes is a handful of launches regardless of how
// many supernodes it has.  FP64 has no tcgen05 MMA kind, so the FP64 tile
// products use DMMA (mma.sync.m8n8k4.f64), the only FP64 tensor-core path on
// Blackwell.

#include "kernels.cuh"

#include <algorithm>
#include <cfloat>
#include <climits>
#include <type_traits>

namespace tb
{
namespace
{

constexpr int kGemmThreads  = 256;
constexpr int kGemmK        = 16;
constexpr int kGemmLd       = kTile + 4;   // padded smem row (2 wavefronts per fragment load)
constexpr int kSolveThreads = 256;

__device__ __forceinline__ void dmma_8x8x4( double (&d)[2], double a, double b )
{
    asm volatile( "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                  : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b) );
}

__device__ __forceinline__ void cp_async_16( void * smem_dst, const void * gmem_src, int src_bytes )
{
    const unsigned saddr = static_cast<unsigned>( __cvta_generic_to_shared( smem_dst ) );
    asm volatile( "cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(saddr), "l"(gmem_src), "r"(src_bytes) );
}
__device__ __forceinline__ void cp_async_commit() { asm volatile( "cp.async.commit_group;\n" ::: "memory" ); }
template<int N> __device__ __forceinline__ void cp_async_wait() { asm volatile( "cp.async.wait_group %0;\n" :: "n"(N) : "memory" ); }

// 8-byte asynchronous copy global -> shared, zero-filled when !valid (the
// source address is then not read, but must still be a mapped address).
// Tile loads are issued this way so that all of a thread's copies are in
// flight at once instead of one load-then-store round trip per element.
__device__ __forceinline__ void cp_async_8( double * smem_dst, const double * gmem_src, bool valid )
{
    const unsigned saddr = static_cast<unsigned>( __cvta_generic_to_shared( smem_dst ) );
    asm volatile( "cp.async.ca.shared.global [%0], [%1], 8, %2;\n" :: "r"(saddr), "l"(gmem_src), "r"(valid ? 8 : 0) );
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile( "cp.async.wait_all;\n" ::: "memory" ); }

// Programmatic dependent launch (sm_90+).  Kernels of the level schedule are
// launched with programmatic stream serialization: a kernel lets the next one
// in its stream launch as soon as all of its own CTAs are running
// (pdl_allow_next), and the next one's CTAs do the work that does not read
// the previous kernel's results (their own task records, factor blocks) and
// then wait for that kernel to complete with its memory visible (pdl_wait),
// so launch latency and independent loads overlap the previous kernel.
// Launched without the attribute, both are no-ops.
__device__ __forceinline__ void pdl_allow_next() { asm volatile( "griddepcontrol.launch_dependents;\n" ::: "memory" ); }
__device__ __forceinline__ void pdl_wait() { asm volatile( "griddepcontrol.wait;\n" ::: "memory" ); }

// Fire-and-forget additions into global memory: the read-modify-write runs in
// the L2 cache and the thread does not wait for it.
__device__ __forceinline__ void red_add_f64( double * p, double a )
{
    asm volatile( "red.global.add.f64 [%0], %1;\n" :: "l"(p), "d"(a) : "memory" );
}

__device__ __forceinline__ void red_add_f32( float * p, float a )
{
    asm volatile( "red.global.add.f32 [%0], %1;\n" :: "l"(p), "f"(a) : "memory" );
}

__device__ __forceinline__ void red_add_v4f32( float * p, float a, float b, float c, float d )
{
    asm volatile( "red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" :: "l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory" );
}

__device__ __forceinline__ void red_add_any( double * p, double a ) { red_add_f64( p, a ); }
__device__ __forceinline__ void red_add_any( float * p, float a ) { red_add_f32( p, a ); }

// ---------------------------------------------------------------- assembly
// arena[dst] = values[src] (+ reg on the diagonal): ReadNonzeroValues
// (Numeric.hpp:165-180) fused with FetchFromA (Multifrontal.hpp:249-321).
template<typename T>
__global__ void assemble_kernel( const double * __restrict__ values, const std::int64_t * __restrict__ src,
                                 const std::int64_t * __restrict__ dst, std::int64_t count,
                                 const double * __restrict__ reg, T * __restrict__ arena )
{
    const double r = *reg;
    for( std::int64_t e = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; e < count;
         e += (std::int64_t)gridDim.x * blockDim.x )
    {
        const std::uint64_t d = static_cast<std::uint64_t>( dst[e] );
        double v = values[src[e]];
        if( d & kDiagFlag ) { v += r; }
        arena[d & (kDiagFlag - 1)] = static_cast<T>( v );
    }
}

// ------------------------------------------------------------------ zeroing
// One warp per row of the task's rows, lanes over its columns [r, n).
template<typename T>
__device__ __forceinline__ void zero_body( const ZeroTask & t, T * __restrict__ arena )
{
    // a row's upper part [r, n): the entries up to the first 16-byte boundary, then 16-byte
    // stores, then the tail
    constexpr int kV = 16 / static_cast<int>( sizeof(T) );
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for( int r = t.row_begin + static_cast<int>( threadIdx.x >> 5 ); r < t.row_end; r += warps )
    {
        T * p = arena + t.offset + static_cast<std::int64_t>( r ) * t.ld + r;
        const int len = t.n - r;
        int head = static_cast<int>( ((16u - (reinterpret_cast<std::uintptr_t>( p ) & 15u)) & 15u) / sizeof(T) );
        head = min( head, len );
        if( lane < head ) { p[lane] = T( 0 ); }
        T * q = p + head;
        const int nv = (len - head) / kV;
        float4 * qv = reinterpret_cast<float4 *>( q );
        for( int v = lane; v < nv; v += 32 ) { qv[v] = make_float4( 0.f, 0.f, 0.f, 0.f ); }
        for( int c = nv * kV + lane; c < len - head; c += 32 ) { q[c] = T( 0 ); }
    }
}

template<typename T>
__global__ void zero_kernel( const ZeroTask * __restrict__ tasks, T * __restrict__ arena )
{
    pdl_allow_next();
    pdl_wait();
    zero_body( tasks[blockIdx.x], arena );
}

// ---------------------------------------------------------------- export
// Reference layout from the fronts: U0 of supernode s is the diagonal block
// of its front at row offset roff; column l of its U1 is front U0 column
// colmap[l] (>= 0) or front U1 column -colmap[l]-1.
template<typename T>
__global__ void export_kernel( const ExportTask * __restrict__ tasks, const std::int32_t * __restrict__ colmap_all,
                               const T * __restrict__ arena, double * __restrict__ tri, double * __restrict__ rec )
{
    const ExportTask t = tasks[blockIdx.x];
    const std::int32_t * colmap = colmap_all + t.colmap;
    for( int r = t.r_begin; r < t.r_end; ++r )
    {
        const std::int64_t fr = t.roff + r;
        const T * f0 = arena + t.fu0 + fr * t.fld0;
        const T * f1 = arena + t.fu1 + fr * t.fld1;
        double * d0 = tri + t.tri + (std::int64_t)r * t.n0s;
        for( int c = threadIdx.x; c < t.n0s; c += blockDim.x ) { d0[c] = (c >= r) ? static_cast<double>( f0[t.roff + c] ) : 0.0; }
        double * d1 = rec + t.rec + (std::int64_t)r * t.n1s;
        for( int l = threadIdx.x; l < t.n1s; l += blockDim.x )
        {
            const int cm = colmap[l];
            d1[l] = static_cast<double>( (cm >= 0) ? f0[cm] : f1[-cm - 1] );
        }
    }
}

// ------------------------------------------------------------- extend-add
// One warp per row of the child's update W; lanes walk the row's upper part
// (coalesced reads of W, lut-indexed adds into the parent front).
template<typename T>
__device__ __forceinline__ void extend_body( const ExtendTask & t, const std::int32_t * __restrict__ lut_all,
                                             T * __restrict__ arena )
{
    const std::int32_t * lut = lut_all + t.lut;
    const T * W = arena + t.w;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    constexpr int kU = 4;     // entries per lane in flight: the lut entries and W values of a group are
                              // loaded before any target is added to.  The targets get their additions
                              // as reductions in the memory system (no load round trip): a launch adds
                              // at most one child into any parent entry (one child rank per pass), so
                              // the sum is the plain target + W in the passes' order.
    for( int i = t.row_begin + warp; i < t.row_end; i += 8 )
    {
        const std::int64_t li = lut[i];
        const T * Wi = W + (std::int64_t)i * t.ldw;
        T * row0 = arena + t.u0 + li * t.ld0p;
        T * row1 = arena + t.u1 + li * t.ld1p;
        T * rowv = arena + t.v + li * t.ldvp;
        const bool upper_part = i < t.mid;
        for( int j0 = i + lane; j0 < t.m1; j0 += 32 * kU )
        {
            T v[kU];
            T * dst[kU];
#pragma unroll
            for( int u = 0; u < kU; ++u )
            {
                const int j = j0 + 32 * u;
                dst[u] = nullptr;
                v[u] = T( 0 );
                if( j < t.m1 )
                {
                    const int lj = lut[j];
                    v[u] = Wi[j];
                    dst[u] = upper_part ? ((j < t.mid) ? row0 + lj : row1 + lj) : rowv + lj;
                }
            }
#pragma unroll
            for( int u = 0; u < kU; ++u ) { if( dst[u] ) { red_add_any( dst[u], v[u] ); } }
        }
    }
}

template<typename T>
__global__ __launch_bounds__(256) void extend_kernel( const ExtendTask * __restrict__ tasks,
                                                      const std::int32_t * __restrict__ lut_all,
                                                      T * __restrict__ arena )
{
    pdl_allow_next();
    const ExtendTask t = tasks[blockIdx.x];
    pdl_wait();
    extend_body( t, lut_all, arena );
}

// Extend-add by parent rows (ExtendPullTask): the CTA adds its segments one
// child after the other, as reductions in the memory system; a fence and a
// barrier between two children make every reduction of the first performed
// before any of the next is issued, so every entry gets the sum of the passes
// by child rank, in the same order (the CTA owns its parent rows for the
// launch).  Inside a segment the (row, 128 columns) chunks go round-robin to
// the warps, so long rows of large update matrices spread over the CTA.
template<typename T>
__global__ __launch_bounds__(256) void extend_pull_kernel( const ExtendPullTask * __restrict__ tasks, const ExtendTask * __restrict__ segs,
                                                           const std::int32_t * __restrict__ lut_all, T * __restrict__ arena )
{
    constexpr int kU = 4, kChunk = 32 * kU, kWarps = 8;
    pdl_allow_next();
    const ExtendPullTask t = tasks[blockIdx.x];
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for( std::int64_t g = t.seg_first; g < t.seg_first + t.seg_count; ++g )
    {
        if( g > t.seg_first )
        {
            __threadfence();
            __syncthreads();
        }
        const ExtendTask e = segs[g];
        const std::int32_t * lut = lut_all + e.lut;
        const T * W = arena + e.w;
        int unit = 0;                                   // chunks before row i, over the segment
        for( int i = e.row_begin; i < e.row_end; ++i )
        {
            const int nch = (e.m1 - i + kChunk - 1) / kChunk;
            int k = (warp - unit % kWarps + kWarps) % kWarps;
            unit += nch;
            if( k >= nch ) { continue; }
            const std::int64_t li = lut[i];
            const T * Wi = W + (std::int64_t)i * e.ldw;
            T * row0 = arena + e.u0 + li * e.ld0p;
            T * row1 = arena + e.u1 + li * e.ld1p;
            T * rowv = arena + e.v + li * e.ldvp;
            const bool upper_part = i < e.mid;
            for( ; k < nch; k += kWarps )
            {
                if constexpr ( sizeof(T) == 4 )
                {
                    // FP32: lane quads of consecutive columns; a quad whose targets are four
                    // consecutive, 16-byte aligned entries goes out as one vector reduction
                    const int j0 = i + k * kChunk + 4 * lane;
                    T v[4];
                    T * dst[4];
#pragma unroll
                    for( int u = 0; u < 4; ++u )
                    {
                        const int j = j0 + u;
                        dst[u] = nullptr;
                        v[u] = T( 0 );
                        if( j < e.m1 )
                        {
                            const int lj = lut[j];
                            v[u] = Wi[j];
                            dst[u] = upper_part ? ((j < e.mid) ? row0 + lj : row1 + lj) : rowv + lj;
                        }
                    }
                    const bool quad = dst[3] != nullptr && dst[1] == dst[0] + 1 && dst[2] == dst[0] + 2 && dst[3] == dst[0] + 3
                                      && (reinterpret_cast<std::uintptr_t>( dst[0] ) & 15u) == 0;
                    if( quad ) { red_add_v4f32( reinterpret_cast<float *>( dst[0] ), v[0], v[1], v[2], v[3] ); }
                    else
                    {
#pragma unroll
                        for( int u = 0; u < 4; ++u ) { if( dst[u] ) { red_add_any( dst[u], v[u] ); } }
                    }
                }
                else
                {
                    const int j0 = i + k * kChunk + lane;
                    T v[kU];
                    T * dst[kU];
#pragma unroll
                    for( int u = 0; u < kU; ++u )
                    {
                        const int j = j0 + 32 * u;
                        dst[u] = nullptr;
                        v[u] = T( 0 );
                        if( j < e.m1 )
                        {
                            const int lj = lut[j];
                            v[u] = Wi[j];
                            dst[u] = upper_part ? ((j < e.mid) ? row0 + lj : row1 + lj) : rowv + lj;
                        }
                    }
#pragma unroll
                    for( int u = 0; u < kU; ++u ) { if( dst[u] ) { red_add_any( dst[u], v[u] ); } }
                }
            }
        }
    }
}

// TF32 rounding (round to nearest, ties away) of an FP32 value, as bits.
__device__ __forceinline__ unsigned to_tf32( float x )
{
    unsigned r;
    asm( "cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x) );
    return r;
}

// ------------------------------------------------------------------ panel
// Cholesky of a panel's nb x nb diagonal block, in shared memory and then
// in place (LAPACK potrf of FactorizeSupernode, Multifrontal.hpp:438-449).
// A row that forms a 1 x 1 reference supernode takes sqrt(|a|) as the
// reference does (:471) and never reports failure.
// Panel kernels work on the 64 x 64 diagonal block in 8 x 8 sub-blocks:
// sequential 8-step recurrences run in registers (unrolled 8 x 8), and every
// update between sub-blocks is an 8 x 8 x 8 product on the FP64 tensor cores
// (two DMMA m8n8k4).  The outer loops over sub-blocks stay rolled so the code
// fits the instruction cache.
constexpr int kPotrfThreads = 384;
constexpr int kTrsmThreads  = 256;
constexpr int kSub          = 8;                     // sub-block edge
constexpr int kSubs         = kPanel / kSub;         // 8 sub-blocks per panel edge
constexpr int kXld          = kRestChunk + 4;        // padded row of the staged rest columns
constexpr size_t kTrsmSmemBytes = sizeof(double) * (2 * kPanel * kXld);

// C(8x8) += A(8x8) * B(8x8) with A read through a(i, k), B through b(k, j)
// and C through c(i, j) (warp-wide; fragment layouts of mma.m8n8k4.f64).
template<typename FA, typename FB>
__device__ __forceinline__ void dmma_8x8x8( double (&acc)[2], FA a, FB b )
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for( int s = 0; s < 2; ++s )
    {
        dmma_8x8x4( acc, a( lane >> 2, (lane & 3) + 4 * s ), b( (lane & 3) + 4 * s, lane >> 2 ) );
    }
}

constexpr int kPld = kPanel + 4;                     // padded smem row of the panel's blocks: DMMA fragments of a
                                                     // block and of its transpose load without bank conflicts
constexpr size_t kPotrfSmemBytes = sizeof(double) * (2 * kPanel * kPld + kPanel + 2);

template<typename T> __device__ __forceinline__ double round_to( double v ) { return static_cast<double>( static_cast<T>( v ) ); }

// Panel factorization state in shared memory.  D: the diagonal block, upper
// triangle (A, overwritten by U tile row by tile row); Ti: the inverse
// T = U^{-1}, upper 8 x 8 tiles (the diagonal tiles are zero below the
// diagonal).  kLd: the leading dimension of both, 0: given at run time.
//
// kIllPivot (FP64): a diagonal tile with a pivot below 1 / kIllPivot of its
// diagonal entry (a pivot's ratio does not change when rows and columns are
// scaled), or with one that is not a positive finite number (its row is then
// scaled by what rsqrt gives: an infinite pivot's to zero), solves its row
// block by substitution.  The product with the tile's
// inverse is exact to a few roundings only while the inverse stays small: with
// every third row within 1e-10 (squared) of the one before, |U^T U - A| is 4
// u |A| by substitution and 12,800 by the product, and from 1e-11 on the
// product's errors make a later pivot negative.  The line lies where both
// agree: with rows within 1e-2 every such tile is below it and the product
// still as good.  Grid and vector Laplacians have no tile below it, a 131^2
// mesh 2 of 2,709; the check alone makes a factor 0 to 1.5% slower (31^3 grid
// 1454 -> 1468 us), substitution in every tile 1 to 8%.  (The same check beside
// the row tiles' products or after the tile's inverse took more: 45^2 grid 111
// us, 118 and 118.)
constexpr double kIllPivot = 16.0;

template<int kLd>
struct PotrfShared
{
    double * d;
    double * ti;
    int ldd, ldt;                                       // used when kLd == 0
    double * floor_s;                                   // mixed precision: the panel's pivot floors; FP64: ill()'s place
    int * flags;                                        // first failing row (-1: none); a tile to factor again; bit q: tile
                                                        // q has raised pivots (the last two: mixed precision)
    __device__ __forceinline__ double & D( int r, int c ) const { return d[r * (kLd > 0 ? kLd : ldd) + c]; }
    __device__ __forceinline__ double & Ti( int r, int c ) const { return ti[r * (kLd > 0 ? kLd : ldt) + c]; }
    __device__ __forceinline__ int & fail() const { return flags[0]; }
    __device__ __forceinline__ int & redo() const { return flags[1]; }
    __device__ __forceinline__ int & raised() const { return flags[2]; }
    __device__ __forceinline__ int & ill( int q ) const { return reinterpret_cast<int *>( floor_s )[q]; }   // FP64: see kIllPivot
};

// Cholesky of the diagonal tile q of D by one warp, and W = U_qq^{-1} into
// tile (q, q) of Ti.  Every lane holds the whole trailing tile in registers
// and runs the same branch-free recurrence, so that a pivot's chain is one
// reciprocal square root, one product and one fused multiply-add (93 cycles);
// lane j also carries column j of the identity through the elimination, whose
// row r is then L^{-1}_rj = W_jr (L = U_qq^T), off the pivot chain.  With FP32 storage U is rounded as it is
// stored and W inverts the rounded rows (the reciprocal of a stored pivot by
// one Newton step on the reciprocal square root, r = v (2 - u v)); the tile's
// row block is solved with the pivots before their rounding, by a second
// inverse kept in the strictly lower tile (7, q) of Ti.
//
// A non-positive pivot (FP64) records the first failing row and lets NaNs run
// on.  kFloored (mixed precision, run again for a tile that met a pivot at or
// below its floor, once the tile's row block is complete): a pivot lost to
// FP32 rounding (for a 1 x 1 supernode too: |a| can cancel to 0) is raised to
// its floor (static pivoting); the FP64 refinement corrects it.  The raised
// pivot also bounds the row's entries in the block by beta = sqrt(max |a_ii|),
// the growth bound of the modified Cholesky of Gill, Murray and Wright: a small
// pivot under a large row would otherwise make the next pivots of the block
// hugely negative, floored in turn, until FP32 overflows.  Without kFloored
// such a tile is left as it was and the function returns false.
template<typename T, bool kFloored, int kLd>
__device__ __forceinline__ bool potrf_diag_tile( const PotrfShared<kLd> & sh, const PanelTask & t, int q, int nb, const T * __restrict__ arena,
                                                 int * __restrict__ status, const double * __restrict__ pivot_floor )
{
    const int lane = threadIdx.x & 31;
    const int o = kSub * q;
    const unsigned singles = static_cast<unsigned>( (t.single_rows >> o) & 0xff );
    double a[kSub][kSub], w[kSub], w2[kSub];
#pragma unroll
    for( int r = 0; r < kSub; ++r )
    {
        w[r] = lane == r ? 1.0 : 0.0;
        w2[r] = w[r];
#pragma unroll
        for( int c = r; c < kSub; ++c ) { a[r][c] = sh.D( o + r, o + c ); }
    }
    // FP64: lane r (mod 8) keeps diagonal entry r and, below, its pivot and the pivot's reciprocal square root
    const double entry = sh.D( o + (lane & (kSub - 1)), o + (lane & (kSub - 1)) );
    double pivot = entry, inv = 0.0;
    __syncwarp();                                       // every lane has the tile before lane 0 writes rows over it
    auto store_row = [&]( int r, const double (&v)[kSub] )
    {
        if( lane != 0 ) { return; }
        if( r & 1 ) { sh.D( o + r, o + r ) = v[r]; }
#pragma unroll
        for( int c = 0; c < kSub; c += 2 )
        {
            if( c >= r ) { *reinterpret_cast<double2 *>( &sh.D( o + r, o + c ) ) = make_double2( v[c], v[c + 1] ); }
        }
    };
    unsigned nonpos = 0u, low = 0u;                     // rows whose pivot is not positive / not above its floor
#pragma unroll
    for( int r = 0; r < kSub; ++r )
    {
        double d = ((singles >> r) & 1) ? fabs( a[r][r] ) : a[r][r];   // 1 x 1 reference supernodes: sqrt(|a|)
        if constexpr ( sizeof(T) == 4 )
        {
            const double tau = sh.floor_s[o + r];
            if constexpr ( kFloored )
            {
                if( o + r < nb && !(d > tau) )
                {
                    // the row's largest entry: this tile's columns, the rest of the
                    // block and the row's rest columns in U0 and U1, which the trsm
                    // divides by the pivot
                    double m = 0.0;
#pragma unroll
                    for( int c = r + 1; c < kSub; ++c ) { m = fmax( m, fabs( a[r][c] ) ); }
                    for( int c = o + kSub + lane; c < nb; c += 32 ) { m = fmax( m, fabs( sh.D( o + r, c ) ) ); }
                    const std::int64_t grow = t.r0 + o + r;
                    for( int c = t.r0 + nb + lane; c < t.n0; c += 32 ) { m = fmax( m, fabs( static_cast<double>( arena[t.u0 + grow * t.ld0 + c] ) ) ); }
                    for( int c = lane; c < t.n1; c += 32 ) { m = fmax( m, fabs( static_cast<double>( arena[t.u1 + grow * t.ld1 + c] ) ) ); }
#pragma unroll
                    for( int s2 = 16; s2 > 0; s2 >>= 1 ) { m = fmax( m, __shfl_xor_sync( 0xffffffffu, m, s2 ) ); }
                    if( lane == 0 ) { atomicAdd( status + 2, 1 ); }
                    const double beta2 = pivot_floor[0];
                    d = fmax( tau, beta2 > 0.0 ? m * m / beta2 : 0.0 );
                }
            }
            else { if( o + r < nb && !(d > tau) ) { low |= 1u << r; } }
        }
        if( !(d > 0.0) ) { nonpos |= 1u << r; }
        const double iv = rsqrt( d );
        if( (lane & (kSub - 1)) == r ) { pivot = d; inv = iv; }
        double us[kSub];
        a[r][r] = d * iv;
        us[r] = round_to<T>( a[r][r] );
#pragma unroll
        for( int c = r + 1; c < kSub; ++c ) { a[r][c] *= iv; us[c] = round_to<T>( a[r][c] ); }
        w[r] *= iv * fma( -us[r], iv, 2.0 );
        w2[r] *= iv;
#pragma unroll
        for( int r2 = r + 1; r2 < kSub; ++r2 )
        {
#pragma unroll
            for( int c = r2; c < kSub; ++c ) { a[r2][c] -= a[r][r2] * a[r][c]; }
            w[r2] -= us[r2] * w[r];
            if constexpr ( sizeof(T) == 4 ) { w2[r2] -= us[r2] * w2[r]; }
        }
        // FP64: the row goes out as it is formed, in the shadow of the pivot chain
        if constexpr ( sizeof(T) == 8 ) { store_row( r, us ); }
        else
        {
#pragma unroll
            for( int c = r; c < kSub; ++c ) { a[r][c] = us[c]; }
        }
    }
    if constexpr ( sizeof(T) == 4 && !kFloored )
    {
        if( low != 0u && pivot_floor != nullptr ) { return false; }
    }
    if constexpr ( sizeof(T) == 8 )
    {
        const bool ill = __any_sync( 0xffffffffu, !(kIllPivot * pivot >= entry && pivot > 0.0 && pivot <= DBL_MAX) );
        if( lane == 0 ) { sh.ill( q ) = ill ? 1 : 0; }
        // the substitution's factors, below the diagonal of the last tile row, where T has zeros
        const int last = kSub * ((nb + kSub - 1) / kSub) - kSub;
        if( ill && o < last && lane < kSub ) { sh.Ti( last + lane, o + lane ) = inv; }
    }
    if constexpr ( kFloored ) { nonpos = 0u; }          // (a floor of zero or NaN is no failure: the refined solve reports it)
    nonpos &= ~singles;
    if( nb - o < kSub ) { nonpos &= (1u << (nb - o)) - 1u; }
    if( lane == 0 && nonpos != 0u && sh.fail() < 0 ) { sh.fail() = o + __ffs( nonpos ) - 1; }
    if( lane < kSub )
    {
#pragma unroll
        for( int i = 0; i < kSub; i += 2 )
        {
            *reinterpret_cast<double2 *>( &sh.Ti( o + lane, o + i ) ) = make_double2( w[i], w[i + 1] );
            if( sizeof(T) == 4 && o < kPanel - kSub ) { *reinterpret_cast<double2 *>( &sh.Ti( kPanel - kSub + lane, o + i ) ) = make_double2( w2[i], w2[i + 1] ); }
        }
    }
    if constexpr ( sizeof(T) == 4 )
    {
#pragma unroll
        for( int r = 0; r < kSub; ++r ) { store_row( r, a[r] ); }
    }
    __syncwarp();
    return true;
}

// The floored factorization of a tile: rare, kept out of the kernel's code.
template<typename T, int kLd>
__device__ __noinline__ void potrf_tile_floored( const PotrfShared<kLd> sh, const PanelTask & t, int q, int nb, const T * __restrict__ arena,
                                                 int * __restrict__ status, const double * __restrict__ pivot_floor )
{
    potrf_diag_tile<T, true>( sh, t, q, nb, arena, status, pivot_floor );
    if( (threadIdx.x & 31) == 0 ) { sh.raised() |= 1 << q; }
}

// U_bc = U_bb^{-T} A_bc for tile (b, c) of D (tile corners o, oc), one column per lane.  last: the
// last tile row, which holds the pivots' reciprocals.
template<typename T, int kLd>
__device__ __noinline__ void potrf_row_substitution( const PotrfShared<kLd> sh, int o, int oc, int last )
{
    const int lane = threadIdx.x & 31;
    if( lane < kSub )
    {
        double x[kSub];
#pragma unroll
        for( int r = 0; r < kSub; ++r ) { x[r] = sh.D( o + r, oc + lane ); }
#pragma unroll
        for( int r = 0; r < kSub; ++r )
        {
            x[r] *= sh.Ti( last + r, o + r );
#pragma unroll
            for( int r2 = r + 1; r2 < kSub; ++r2 ) { x[r2] -= sh.D( o + r, o + r2 ) * x[r]; }
        }
#pragma unroll
        for( int r = 0; r < kSub; ++r ) { sh.D( o + r, oc + lane ) = round_to<T>( x[r] ); }
    }
}

// Cholesky of a panel's diagonal block D and the inverse T of its factor
// (LAPACK potrf of FactorizeSupernode, Multifrontal.hpp:438-449, plus the
// inverse that the trsm and the solves use), right-looking by 8 x 8 tiles.
// Step b runs between two block barriers; barrier 1 divides it for the warps
// that do not run the pivot chain:
//   warp 0   row tile (b, b+1); arrives at barrier 1 without waiting there;
//            update and factorization of tile (b+1, b+1), and its inverse
//            W_{b+1} into tile (b+1, b+1) of Ti.
//   others   until barrier 1: the other row tiles U_bc, c > b+1, in place, and
//            T_ib = -S_ib W_b, i < b, over S_ib in tile (i, b) of Ti;
//            after it, with row block b complete: the trailing tiles but
//            (b+1, b+1), S_{i,b+1} = sum_{k=i..b} T_ik U_{k,b+1} into tile
//            (i, b+1) of Ti, and the stores of what step b-1 finished.
// Everything the others read of warp 0's tile (b+1, b+1) - U, W, the ill()
// flag - was written before the step's last barrier; everything warp 0 reads
// of row block b and of tile (b+1, b+1) it wrote itself or found complete at
// the step's start.  A step lasts as long as warp 0's chain (8 pivots of ~93
// cycles and two tile products) while the others' jobs fit beside it, which
// they do with nine warps; step -1 only factors tile 0.
//
// kThreads: 384 in the panel launches and the larger small fronts, 128 in the
// smaller ones, 256 in the persistent kernel.  The block (nb x nb, identity beyond
// up to a multiple of 8) is in sh.D; pending: its cp.async copies may still be
// in flight except tile 0's rows.  U goes to the arena, T to tinv.
template<typename T, int kThreads, int kLd>
__device__ __forceinline__ void potrf_core( const PotrfShared<kLd> & sh, const PanelTask & t, int nb, T * __restrict__ arena,
                                            int * __restrict__ status, const double * __restrict__ pivot_floor, double * __restrict__ tinv )
{
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    T * U0 = arena + t.u0 + (std::int64_t)t.r0 * t.ld0 + t.r0;
    const int nsub = (nb + kSub - 1) / kSub;
    const int i8 = lane >> 2, j8 = 2 * (lane & 3);        // this lane's entries of an 8 x 8 DMMA result
    // U_bc = W_b^T A_bc in place (tile (b, c) of D), rounded to the storage type.  By substitution
    // where W_b's entries may grow beyond what the product can cancel: FP64 tiles with a small pivot
    // (kIllPivot), mixed precision tiles with raised pivots.
    auto row_tile = [&]( int o, int oc )
    {
        if( sizeof(T) == 4 ? (sh.raised() >> (o / kSub)) & 1 : sh.ill( o / kSub ) )
        {
            potrf_row_substitution<T>( sh, o, oc, sizeof(T) == 4 ? kPanel - kSub : kSub * (nsub - 1) );
            return;
        }
        const int ow = sizeof(T) == 4 ? kPanel - kSub : o;
        double acc[2] = { 0.0, 0.0 };
        dmma_8x8x8( acc, [&]( int ii, int k ) { return sh.Ti( ow + k, o + ii ); }, [&]( int k, int jj ) { return sh.D( o + k, oc + jj ); } );
        __syncwarp();
        *reinterpret_cast<double2 *>( &sh.D( o + i8, oc + j8 ) ) = make_double2( round_to<T>( acc[0] ), round_to<T>( acc[1] ) );
    };
    // tile (r, c) of D -= U_b,r^T U_b,c (summed apart and subtracted once: one rounding at the tile's
    // own magnitude per step)
    auto trailing_tile = [&]( int o, int orow, int oc )
    {
        double2 * d = reinterpret_cast<double2 *>( &sh.D( orow + i8, oc + j8 ) );
        const double2 v = *d;
        double acc[2] = { 0.0, 0.0 };
        dmma_8x8x8( acc, [&]( int ii, int k ) { return sh.D( o + k, orow + ii ); }, [&]( int k, int jj ) { return sh.D( o + k, oc + jj ); } );
        *d = make_double2( v.x - acc[0], v.y - acc[1] );
    };
    // What step b finished, to global memory, in kSub + nsub units of 32 threads: U's row u of tile
    // row b (columns from the diagonal on), then 8 rows of T's column block b (zero below the
    // diagonal; the nsub leading tiles are all that the trsm and the solves read).
    const int nbp = kSub * nsub;
    double * out = tinv + (std::int64_t)t.panel * (kPanel * kPanel);
    auto store_unit = [&]( int b, int u )
    {
        const int o = kSub * b;
        if( u < kSub )
        {
            const int r = o + u, c = 2 * lane;
            if( r >= nb || c >= nb ) { return; }
            const double2 v = *reinterpret_cast<const double2 *>( &sh.D( r, c ) );
            T * dst = U0 + (std::int64_t)r * t.ld0 + c;
            if( r <= c && c + 1 < nb )
            {
                if constexpr ( sizeof(T) == 8 ) { *reinterpret_cast<double2 *>( dst ) = v; }
                else { *reinterpret_cast<float2 *>( dst ) = make_float2( static_cast<float>( v.x ), static_cast<float>( v.y ) ); }
            }
            else
            {
                if( r <= c ) { dst[0] = static_cast<T>( v.x ); }
                if( r <= c + 1 && c + 1 < nb ) { dst[1] = static_cast<T>( v.y ); }
            }
        }
        else
        {
            const int r = kSub * (u - kSub) + (lane >> 2), c = o + 2 * (lane & 3);
            const double2 v = *reinterpret_cast<const double2 *>( &sh.Ti( r, c ) );
            *reinterpret_cast<double2 *>( out + r * kPanel + c ) = r < o + kSub ? v : make_double2( 0.0, 0.0 );
        }
    };
    // step -1 only factors tile 0 (while the rest of the block arrives)
    for( int b = -1; b < nsub; ++b )
    {
        const int o = kSub * b, o1 = o + kSub;
        const int rem = nsub - 1 - b;                   // trailing tile rows / columns
        if( warp == 0 )
        {
            if( rem > 0 )
            {
                if( b >= 0 )
                {
                    row_tile( o, o1 );
                    __syncwarp();
                    asm volatile( "bar.arrive 1, %0;\n" :: "n"(kThreads) : "memory" );
                    trailing_tile( o, o1, o1 );
                    __syncwarp();
                }
                if( !potrf_diag_tile<T, false>( sh, t, b + 1, nb, arena, status, pivot_floor ) && lane == 0 ) { sh.redo() = 1; }
            }
        }
        else if( b >= 0 )
        {
            // the warps that share warp 0's SM sub-partition (warp index mod 4)
            // take no job, so that the pivot chain does not wait behind one
            const int first = (warp & 3) == 0 ? INT_MAX : warp - 1 - (warp >> 2);
            constexpr int kStep = kThreads / 128 * 3;
            const int rows = rem > 0 ? rem - 1 : 0;
            for( int job = first; job < rows + b; job += kStep )
            {
                if( job < rows ) { row_tile( o, o1 + kSub * (job + 1) ); }
                else
                {
                    const int oi = kSub * (job - rows);
                    double acc[2] = { 0.0, 0.0 };
                    dmma_8x8x8( acc, [&]( int ii, int k ) { return sh.Ti( oi + ii, o + k ); }, [&]( int k, int jj ) { return sh.Ti( o + k, o + jj ); } );
                    __syncwarp();
                    *reinterpret_cast<double2 *>( &sh.Ti( oi + i8, o + j8 ) ) = make_double2( -acc[0], -acc[1] );
                }
            }
            if( rem > 0 )
            {
                asm volatile( "bar.sync 1, %0;\n" :: "n"(kThreads) : "memory" );
                const int tiles = rem * (rem + 1) / 2 - 1;              // all but (b+1, b+1)
                const int jobs = tiles + b + 1;
                int c = b + 2, left = first;            // a trailing tile's column, and its place in it
                for( int job = first; job < jobs + (b > 0 ? kSub + nsub : 0); job += kStep )
                {
                    if( job >= jobs ) { store_unit( b - 1, job - jobs ); }
                    else if( job < tiles )
                    {
                        // tile (b + 1 + left, c), column by column of the trailing triangle after (b+1, b+1)
                        while( left >= c - b ) { left -= c - b; ++c; }
                        trailing_tile( o, o1 + kSub * left, kSub * c );
                        left += kStep;
                    }
                    else
                    {
                        // S_i,b+1 into tile (i, b+1) of Ti
                        const int oi = kSub * (job - tiles);
                        double acc[2] = { 0.0, 0.0 };
                        for( int ok = oi; ok <= o; ok += kSub )
                        {
                            dmma_8x8x8( acc, [&]( int ii, int kk ) { return sh.Ti( oi + ii, ok + kk ); },
                                             [&]( int kk, int jj ) { return sh.D( ok + kk, o1 + jj ); } );
                        }
                        *reinterpret_cast<double2 *>( &sh.Ti( oi + i8, o1 + j8 ) ) = make_double2( acc[0], acc[1] );
                    }
                }
            }
        }
        if( b < 0 ) { cp_async_wait_all(); }
        __syncthreads();
        if constexpr ( sizeof(T) == 4 )
        {
            if( sh.redo() )
            {
                // a pivot of tile (b+1, b+1) needed its floor: factor the tile again
                // now that its row block is complete
                if( warp == 0 ) { potrf_tile_floored<T>( sh, t, b + 1, nb, arena, status, pivot_floor ); }
                __syncthreads();
                if( tid == 0 ) { sh.redo() = 0; }
                __syncthreads();
            }
        }
    }
    for( int u = warp; u < 2 * (kSub + nsub); u += kThreads / 32 )
    {
        const bool last = u >= kSub + nsub;
        if( last || nsub > 1 ) { store_unit( nsub - (last ? 1 : 2), last ? u - kSub - nsub : u ); }
    }
    if( tid == 0 && sh.fail() >= 0 )
    {
        atomicOr( status, 1 );
        atomicMin( status + 1, t.row0 + t.r0 + sh.fail() );
    }
}

// The panel's diagonal block (64 x kPld cells of dynamic shared memory), then potrf_core.
// kPend (FP64): the t.pend pending rows' update of the block comes first, D -= P^T P with P the rows
// r0 - pend .. r0 - 1 of the block's columns, in chunks of 64 rows through T's and D's space; a warp
// holds three of the 36 upper 8 x 8 tiles.  The panel chain is then trsm -> potrf, with the rest of
// the row's update beside the potrf, instead of trsm -> GEMM -> potrf (a launch of 8-20 us).  The K
// order and the single subtraction are the GEMM tile's: the same bits.
template<typename T, int kThreads, bool kPend>
__device__ __forceinline__ void potrf_body( const PanelTask & t, T * __restrict__ arena, int * __restrict__ status,
                                            const double * __restrict__ pivot_floor, double * __restrict__ tinv )
{
    extern __shared__ __align__(16) double panel_smem[];
    const int tid = threadIdx.x;
    const int nb = min( kPanel, t.n0 - t.r0 );
    PotrfShared<kPld> sh;
    sh.d = panel_smem;
    sh.ti = panel_smem + kPanel * kPld;
    sh.ldd = sh.ldt = kPld;
    sh.floor_s = panel_smem + 2 * kPanel * kPld;
    sh.flags = reinterpret_cast<int *>( sh.floor_s + kPanel );

    T * U0 = arena + t.u0 + (std::int64_t)t.r0 * t.ld0 + t.r0;
    if constexpr ( kPend )
    {
        static_assert( sizeof(T) == 8 && kThreads == 384, "12 warps hold 36 tiles" );
        if( t.pend > 0 )
        {
            const int lane = tid & 31, warp = tid >> 5;
            const int nch = t.pend / kPanel;
            const T * P = arena + t.u0 + (std::int64_t)(t.r0 - t.pend) * t.ld0 + t.r0;
            auto load_chunk = [&]( int ch )
            {
                double * dst = (ch & 1) ? sh.d : sh.ti;
                for( int idx = 2 * tid; idx < kPanel * kPanel; idx += 2 * kThreads )
                {
                    const int r = idx / kPanel, c = idx % kPanel;
                    cp_async_16( dst + r * kPld + c, c < nb ? P + (std::int64_t)(ch * kPanel + r) * t.ld0 + c : P, c + 1 < nb ? 16 : c < nb ? 8 : 0 );
                }
                cp_async_commit();
            };
            // tiles (ti, tj) of warp w: the w-th, 12 + w-th and 24 + w-th of the upper ones, by columns
            int ti[3], tj[3];
#pragma unroll
            for( int e = 0; e < 3; ++e )
            {
                int left = warp + 12 * e, col = 0;
                while( left > col ) { left -= col + 1; ++col; }
                ti[e] = left;
                tj[e] = col;
            }
            double acc[3][2];
#pragma unroll
            for( int e = 0; e < 3; ++e ) { acc[e][0] = 0.0; acc[e][1] = 0.0; }
            load_chunk( 0 );
            if( nch > 1 ) { load_chunk( 1 ); }
            for( int ch = 0; ch < nch; ++ch )
            {
                if( ch + 1 < nch ) { cp_async_wait<1>(); } else { cp_async_wait<0>(); }
                __syncthreads();
                const double * src = ((ch & 1) ? sh.d : sh.ti) + (lane >> 2);
#pragma unroll 4
                for( int k = lane & 3; k < kPanel; k += 4 )
                {
#pragma unroll
                    for( int e = 0; e < 3; ++e ) { dmma_8x8x4( acc[e], src[k * kPld + kSub * ti[e]], src[k * kPld + kSub * tj[e]] ); }
                }
                __syncthreads();
                if( ch + 2 < nch ) { load_chunk( ch + 2 ); }
            }
#pragma unroll
            for( int e = 0; e < 3; ++e )
            {
                const int r = kSub * ti[e] + (lane >> 2), c = kSub * tj[e] + 2 * (lane & 3);
                double2 v = make_double2( r == c ? 1.0 : 0.0, r == c + 1 ? 1.0 : 0.0 );   // identity beyond nb
                if( r < nb )
                {
                    // (below the diagonal of a diagonal tile: zeros, never used)
                    v = make_double2( 0.0, 0.0 );
                    const T * src = U0 + (std::int64_t)r * t.ld0 + c;
                    if( c + 1 < nb ) { v = *reinterpret_cast<const double2 *>( src ); }
                    else if( c < nb ) { v.x = src[0]; }
                    if( c < nb ) { v.x -= acc[e][0]; }
                    if( c + 1 < nb ) { v.y -= acc[e][1]; }
                }
                *reinterpret_cast<double2 *>( &sh.D( r, c ) ) = v;
            }
            if( tid == 0 ) { sh.fail() = -1; sh.redo() = 0; sh.raised() = 0; }
            __syncthreads();
            potrf_core<T, kThreads>( sh, t, nb, arena, status, pivot_floor, tinv );
            return;
        }
    }
    // 16-byte pieces of the rows (16-byte aligned: offsets and leading dimensions are multiples of
    // kLdAlign entries), all of a thread's in flight together; pieces below the diagonal are not read
    // later and not loaded; identity padding beyond nb
    constexpr int kV = 16 / static_cast<int>( sizeof(T) );
    constexpr int kAll = kPanel * kPanel / kV, kPieces = (kAll + kThreads - 1) / kThreads;
    if constexpr ( sizeof(T) == 8 )
    {
#pragma unroll
        for( int u = 0; u < kPieces; ++u )
        {
            const int idx = kV * (tid + u * kThreads), r = idx / kPanel, c = idx % kPanel;
            if( r >= kPanel ) {}
            else if( r >= nb ) { sh.D( r, c ) = r == c ? 1.0 : 0.0; sh.D( r, c + 1 ) = r == c + 1 ? 1.0 : 0.0; }
            else if( c + 1 >= r ) { cp_async_16( &sh.D( r, c ), c < nb ? U0 + (std::int64_t)r * t.ld0 + c : U0, c + 1 < nb ? 16 : c < nb ? 8 : 0 ); }
            if( u == 0 ) { cp_async_commit(); }         // the first rows: tile 0 starts when they are in
        }
        cp_async_commit();
    }
    else
    {
        float4 v[kPieces];
#pragma unroll
        for( int u = 0; u < kPieces; ++u )
        {
            const int idx = kV * (tid + u * kThreads), r = idx / kPanel, c = idx % kPanel;
            v[u] = make_float4( 0.f, 0.f, 0.f, 0.f );
            if( r < nb && c < nb && c + 3 >= r ) { v[u] = *reinterpret_cast<const float4 *>( U0 + (std::int64_t)r * t.ld0 + c ); }
        }
#pragma unroll
        for( int u = 0; u < kPieces; ++u )
        {
            const int idx = kV * (tid + u * kThreads), r = idx / kPanel, c = idx % kPanel;
            if( r >= kPanel ) { continue; }
            const double pad = r >= nb ? 1.0 : 0.0;
            const float f[4] = { v[u].x, v[u].y, v[u].z, v[u].w };
#pragma unroll
            for( int e = 0; e < 4; ++e ) { sh.D( r, c + e ) = r < nb && c + e < nb ? static_cast<double>( f[e] ) : r == c + e ? pad : 0.0; }
        }
    }
    // the pivot floors after the block's copies are in flight (their loads overlap)
    if( pivot_floor != nullptr && tid < nb ) { sh.floor_s[tid] = pivot_floor[1 + t.row0 + t.r0 + tid]; }
    if( tid == 0 ) { sh.fail() = -1; sh.redo() = 0; sh.raised() = 0; }
    cp_async_wait<1>();
    __syncthreads();

    potrf_core<T, kThreads>( sh, t, nb, arena, status, pivot_floor, tinv );
}

template<typename T, bool kPend>
__global__ __launch_bounds__(kPotrfThreads, 1) void potrf_kernel( const PanelTask * __restrict__ tasks,
                                                               T * __restrict__ arena, int * __restrict__ status,
                                                               const double * __restrict__ pivot_floor,
                                                               double * __restrict__ tinv )
{
    const PanelTask t = tasks[blockIdx.x];
    pdl_wait();
    // only now: the trsm may read the rest columns before its own wait (kPrefetch), so everything
    // before this launch must be complete when it starts
    pdl_allow_next();
    potrf_body<T, kPotrfThreads, kPend>( t, arena, status, pivot_floor, tinv );
}

// ------------------------------------------------------------ small fronts
// A whole front with at most one panel of pivot rows (FrontTask) in one CTA's
// shared memory: assembled rows, children added in rank order, potrf, rest
// columns, update matrix.  The operations on each entry are those of the
// separate launches in the same order (FP64: the same factor bit for bit),
// without their passes over the front in global memory: zeroing, one
// read-modify-write per child and one for the update, the rest columns
// written and read back.  Blocks of a few dozen rows leave the bound to
// latencies (the children's rows, the pivot chain), so what counts is CTAs
// per SM and warps per CTA: the plan picks 128, 256 or 384 threads (three,
// two, one CTA per SM) by the launch's front count and shared memory.
//
// The update matrix is kept by blocks of 8 rows from the diagonal on.  FP64
// storage only.
__device__ __forceinline__ int front_v_row( int n1p, int row )
{
    const int rb = row >> 3, width = n1p - 8 * rb;
    return 8 * (rb * n1p - 4 * rb * (rb - 1)) + (row & 7) * width - 8 * rb;      // + column
}

template<int kThreads>
__global__ __launch_bounds__(kThreads, kThreads == 128 ? 3 : kThreads == 256 ? 2 : 1)
void front_kernel( const FrontTask * __restrict__ tasks, const ExtendTask * __restrict__ segs, const std::int32_t * __restrict__ lut_all,
                   double * __restrict__ arena, int * __restrict__ status, double * __restrict__ tinv )
{
    extern __shared__ __align__(16) double fsm[];
    pdl_allow_next();
    const FrontTask ft = tasks[blockIdx.x];
    const PanelTask & t = ft.p;
    constexpr int kWarps = kThreads / 32;
    constexpr int kV = 2;                                 // entries of a 16-byte piece
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = t.n0, n1 = t.n1;
    const int n0p = (n0 + 7) & ~7, n1p = (n1 + 7) & ~7;
    PotrfShared<0> sh;
    sh.ldd = n0p + n1p + 4;
    sh.ldt = n0p + 4;
    sh.d = fsm;
    sh.ti = sh.d + n0p * sh.ldd;
    double * V = sh.ti + n0p * sh.ldt;
    sh.floor_s = V + 4 * n1p * (n1p / 8 + 1);
    sh.flags = reinterpret_cast<int *>( sh.floor_s + kPanel );
    double * X = sh.d + n0p;                              // rest columns, rows sh.ldd apart
    const int ldx = sh.ldd;

    if( ft.has_v ) { for( int e = 2 * tid; e < 4 * n1p * (n1p / 8 + 1); e += 2 * kThreads ) { *reinterpret_cast<double2 *>( V + e ) = make_double2( 0.0, 0.0 ); } }
    if( tid == 0 ) { sh.fail() = -1; sh.redo() = 0; sh.raised() = 0; }
    pdl_wait();
    // the assembled rows: diagonal block (identity beyond n0; below the diagonal not read later), rest columns
    {
        const double * U0 = arena + t.u0;
        const double * U1 = arena + t.u1;
        // 16-byte pieces: a lane keeps its columns and steps over the warp's rows
        const int per0 = n0p / kV, per = (n0p + n1p) / kV;
        for( int q = lane; q < per; q += 32 )
        {
            const bool diag = q < per0;
            const int c = kV * (diag ? q : q - per0), lim = diag ? n0 : n1;
            const int ld = diag ? t.ld0 : t.ld1;
            const double * src = (diag ? U0 : U1) + c + (std::int64_t)warp * ld;
            double * dst = sh.d + warp * ldx + kV * q;
            const int rows = c < lim ? min( n0, diag ? c + kV : n0 ) : 0;      // rows with entries of these columns
            const int bytes = c + 1 < lim ? 16 : 8;
#pragma unroll 2
            for( int r = warp; r < n0p; r += kWarps, src += (std::int64_t)kWarps * ld, dst += kWarps * ldx )
            {
                if( r < rows ) { cp_async_16( dst, src, bytes ); }
                else if( r >= n0 || c >= lim ) { *reinterpret_cast<double2 *>( dst ) = make_double2( diag && r == c ? 1.0 : 0.0, diag && r == c + 1 ? 1.0 : 0.0 ); }
            }
        }
        cp_async_wait_all();
    }
    __syncthreads();
    // children, one after the other (a barrier between two).  A warp's unit is kRows rows of a
    // 32-column chunk of the child's upper triangle; the next unit's loads (the next child's first
    // unit too) are in flight while this one is added, so that a child costs its additions and not
    // a round trip to memory (two columns per lane measured the same: the pairs' shared-memory
    // conflicts cost what the shared address arithmetic saves).
    constexpr int kRows = 8, kSegs = 16;
    struct Seg { const double * W; const std::int32_t * lut; int m1, mid, ldw; };
    __shared__ Seg seg_s[kSegs];
    // v: the unit's entries; li: lane u's row position in the parent (u < kRows); lj: the lane's column
    struct Unit { double v[kRows]; int li; int lj; };
    const int v0 = static_cast<int>( V - sh.d );
    for( int g0 = 0; g0 < ft.seg_count; g0 += kSegs )
    {
        const int ng = min( kSegs, ft.seg_count - g0 );
        if( g0 > 0 ) { __syncthreads(); }
        if( tid < ng )
        {
            const ExtendTask & e = segs[ft.seg_first + g0 + tid];
            seg_s[tid] = { arena + e.w, lut_all + e.lut, e.m1, e.mid, e.ldw };
        }
        __syncthreads();
        auto load = [&]( Unit & un, int g, int j0, int i0 )
        {
            const Seg & e = seg_s[g];
            const int j = j0 + lane, il = i0 + (lane & (kRows - 1)) * kWarps;
            un.lj = j < e.m1 ? e.lut[j] : 0;
            un.li = il < e.m1 ? e.lut[il] : 0;
            const double * w = e.W + (std::int64_t)i0 * e.ldw + j;
            const std::int64_t step = static_cast<std::int64_t>( kWarps ) * e.ldw;
            const int last = j < e.m1 ? j - i0 : -1;
#pragma unroll
            for( int u = 0; u < kRows; ++u ) { un.v[u] = u * kWarps <= last ? w[u * step] : 0.0; }
        };
        Unit cur;
        int g = 0, j0 = 0, i0 = warp;
        load( cur, 0, 0, i0 );
        while( g < ng )
        {
            const int m1 = seg_s[g].m1, mid = seg_s[g].mid;
            // the following unit
            int gn = g, jn = j0, in = i0 + kRows * kWarps;
            if( in >= min( m1, j0 + 32 ) ) { jn += 32; in = warp; }
            if( jn >= m1 ) { ++gn; jn = 0; }
            Unit nxt;
            if( gn < ng ) { load( nxt, gn, jn, in ); }
            // offsets of the unit's rows from sh.d: lane u forms row u's, the others take it from there
            const bool pivot_row = i0 + (lane & (kRows - 1)) * kWarps < mid;
            const int base = pivot_row ? cur.li * ldx : v0 + front_v_row( n1p, cur.li );
            const int j = j0 + lane, last = j < m1 ? j - i0 : -1;
            const int cp = cur.lj + (j < mid ? 0 : n0p);                  // the column in a pivot row
            double * dst[kRows];
            double x[kRows];
#pragma unroll
            for( int u = 0; u < kRows; ++u )
            {
                const int row = __shfl_sync( 0xffffffffu, base, u );
                dst[u] = sh.d + row + (i0 + u * kWarps < mid ? cp : cur.lj);
                x[u] = u * kWarps <= last ? *dst[u] : 0.0;
            }
#pragma unroll
            for( int u = 0; u < kRows; ++u )
            {
                if( u * kWarps <= last ) { *dst[u] = x[u] + cur.v[u]; }
            }
            if( gn != g ) { __syncthreads(); }
            cur = nxt;
            g = gn; j0 = jn; i0 = in;
        }
    }
    potrf_core<double, kThreads>( sh, t, n0, arena, status, nullptr, tinv );
    if( n1 == 0 ) { return; }
    // rest columns X <- T^T X in place: a warp takes all row blocks of an 8-column tile
    const int nsub = n0p / kSub, n1t = n1p / kSub;
    const int fi = lane >> 2, fj = 2 * (lane & 3);
    for( int ct = warp; ct < n1t; ct += kWarps )
    {
        double acc[kSubs][2];
#pragma unroll
        for( int rb = 0; rb < kSubs; ++rb ) { acc[rb][0] = 0.0; acc[rb][1] = 0.0; }
#pragma unroll
        for( int kb = 0; kb < kSubs; ++kb )
        {
            if( kb >= nsub ) { break; }
            double b[2];
#pragma unroll
            for( int q = 0; q < 2; ++q ) { b[q] = X[(kSub * kb + (lane & 3) + 4 * q) * ldx + kSub * ct + fi]; }
#pragma unroll
            for( int rb = kb; rb < kSubs; ++rb )
            {
                if( rb >= nsub ) { break; }
#pragma unroll
                for( int q = 0; q < 2; ++q ) { dmma_8x8x4( acc[rb], sh.Ti( kSub * kb + (lane & 3) + 4 * q, kSub * rb + fi ), b[q] ); }
            }
        }
        __syncwarp();
        const int c = kSub * ct + fj;
#pragma unroll
        for( int rb = 0; rb < kSubs; ++rb )
        {
            if( rb >= nsub ) { break; }
            const int r = kSub * rb + fi;
            const double2 x = make_double2( acc[rb][0], acc[rb][1] );
            *reinterpret_cast<double2 *>( X + r * ldx + c ) = x;
            if( r < n0 && c < n1 )
            {
                // (a row's padding takes the tile's zero column: rows are padded to four entries)
                double * dst = arena + t.u1 + (std::int64_t)r * t.ld1 + c;
                *reinterpret_cast<double2 *>( dst ) = x;
            }
        }
    }
    if( !ft.has_v ) { return; }
    __syncthreads();
    // update matrix V - X^T X, 16 x 16 blocks of its upper triangle round the warps
    const int nm = (n1t + 1) / 2;
    int I = 0, J = warp;
    while( I < nm )
    {
        if( J >= nm ) { J = J - nm + I + 1; ++I; if( I >= nm || J >= nm ) { continue; } }
        double acc[2][2][2];
#pragma unroll
        for( int a = 0; a < 2; ++a )
        {
#pragma unroll
            for( int b = 0; b < 2; ++b ) { acc[a][b][0] = 0.0; acc[a][b][1] = 0.0; }
        }
        const int r0 = 16 * I, c0 = 16 * J;
        const int r1 = r0 + 8 < n1p ? r0 + 8 : r0, c1 = c0 + 8 < n1p ? c0 + 8 : c0;     // (a missing half repeats the first)
#pragma unroll 4
        for( int k = lane & 3; k < n0p; k += 4 )
        {
            const double * x = X + k * ldx + fi;
            const double a0 = x[r0], a1 = x[r1], b0 = x[c0], b1 = x[c1];
            dmma_8x8x4( acc[0][0], a0, b0 );
            dmma_8x8x4( acc[0][1], a0, b1 );
            dmma_8x8x4( acc[1][0], a1, b0 );
            dmma_8x8x4( acc[1][1], a1, b1 );
        }
#pragma unroll
        for( int a = 0; a < 2; ++a )
        {
#pragma unroll
            for( int b = 0; b < 2; ++b )
            {
                const int row = r0 + 8 * a + fi, col = c0 + 8 * b + fj;
                if( row >= n1 || col >= n1 || (I == J && a > b) ) { continue; }
                const double2 v = *reinterpret_cast<const double2 *>( V + front_v_row( n1p, row ) + col );
                const double x0 = v.x - acc[a][b][0], x1 = v.y - acc[a][b][1];
                double * dst = arena + ft.v + (std::int64_t)row * t.ld1 + col;
                if( row <= col ) { *reinterpret_cast<double2 *>( dst ) = make_double2( x0, x1 ); }
                else if( row == col + 1 ) { dst[1] = x1; }
            }
        }
        J += kWarps;
    }
}

// X = D^{-T} U for the rest columns [c0, c0 + cw) of a panel (trsm of
// FactorizeSupernode, Multifrontal.hpp:452-466) as the product X = T^T U with
// the inverse T = D^{-1} that the panel's potrf left in tinv: X row block rb
// takes the K blocks 0..rb.  A chunk lies in U0 or in U1, so that its rows are
// read and written in aligned vectors.  Warp w takes the chunk's column tile w
// with all eight row blocks' sums in registers: 72 independent-by-eight DMMAs
// follow 88 fragment loads, and the results go to global memory from the
// registers.  Bound: the launch's latency (load, 72 DMMAs a warp, store) on
// the panel chain.

// Operand-image entry of U row k, rest column `col` of a panel whose rest
// columns start at U0 column r1 (m of them in U0, the rest U1 columns).
__device__ __forceinline__ std::int64_t img_offset( const PanelTask & t, int k, int col, int r1, int m )
{
    const int ucol = col < m ? r1 + col : col - m;
    const int ct = col < m ? ucol / kImgRows : t.img_t0 + ucol / kImgRows;
    const std::int64_t blk = t.img + static_cast<std::int64_t>( k / kImgK ) * 2 * t.img_tf + ct;
    return blk * (kImgRows * kImgK) + (ucol % kImgRows) * kImgK + (k % kImgK);
}

// kPrefetch: the launch before is the potrf, which let this one start only
// after its own wait, and nothing else is waited for: the rest columns are
// loaded before the wait.  (FP64 level launches: their update runs on another
// stream, so that the wait comes first.)
template<typename T, bool kPdl, bool kPrefetch>
__device__ __forceinline__ void trsm_body( const PanelTask & t, T * __restrict__ arena, const double * __restrict__ tinv,
                                           double * tsm, float * __restrict__ img = nullptr )
{
    double (*Ti)[kXld] = reinterpret_cast<double (*)[kXld]>( tsm );
    double (*X)[kXld] = reinterpret_cast<double (*)[kXld]>( tsm + kPanel * kXld );
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int nb = min( kPanel, t.n0 - t.r0 );
    const int nbb = (nb + kSub - 1) / kSub;
    const int r1 = t.r0 + nb;
    const int m = t.n0 - r1;
    const int rest = m + t.n1;
    const bool in0 = t.c0 < m;                            // the chunk's columns: U0's or U1's
    const int cw = min( kRestChunk, (in0 ? m : rest) - t.c0 );
    const int ld = in0 ? t.ld0 : t.ld1;
    T * U = (in0 ? arena + t.u0 + r1 + t.c0 : arena + t.u1 + (t.c0 - m)) + (std::int64_t)t.r0 * ld;
    static_assert( kRestChunk == kPanel && kTrsmThreads / 32 == kRestChunk / kSub, "trsm assumes square blocks and a warp per column tile" );
    constexpr int kV = 16 / static_cast<int>( sizeof(T) );
    constexpr int kPieces = kPanel * kRestChunk / kV / kTrsmThreads;
    [[maybe_unused]] float4 xf[sizeof(T) == 4 ? kPieces : 1];
    if constexpr ( kPdl && !kPrefetch ) { pdl_wait(); }
#pragma unroll
    for( int u = 0; u < kPieces; ++u )
    {
        const int idx = kV * (tid + u * kTrsmThreads), r = idx / kRestChunk, c = idx % kRestChunk;
        const bool in = r < nb && c < cw;
        if constexpr ( sizeof(T) == 8 ) { cp_async_16( &X[r][c], in ? U + (std::int64_t)r * ld + c : U, in ? (c + 1 < cw ? 16 : 8) : 0 ); }
        else { xf[u] = in ? *reinterpret_cast<const float4 *>( U + (std::int64_t)r * ld + c ) : make_float4( 0.f, 0.f, 0.f, 0.f ); }
    }
    if constexpr ( kPdl && kPrefetch ) { pdl_wait(); }
    {
        // only the leading (nb rounded up to 8)^2 block of T is read
        const double * Tg = tinv + (std::int64_t)t.panel * (kPanel * kPanel);
        const int nbp = kSub * nbb;
#pragma unroll
        for( int u = 0; u < kPanel * kPanel / (2 * kTrsmThreads); ++u )
        {
            const int idx = 2 * (tid + u * kTrsmThreads);
            if( (idx >> 6) < nbp && (idx & 63) < nbp ) { cp_async_16( &Ti[idx >> 6][idx & 63], Tg + idx, 16 ); }
        }
    }
    if constexpr ( sizeof(T) == 4 )
    {
#pragma unroll
        for( int u = 0; u < kPieces; ++u )
        {
            const int idx = kV * (tid + u * kTrsmThreads), r = idx / kRestChunk, c = idx % kRestChunk;
            // (a row's padding beyond cw may hold anything: zero)
            const double x[4] = { xf[u].x, c + 1 < cw ? xf[u].y : 0.0, c + 2 < cw ? xf[u].z : 0.0, c + 3 < cw ? xf[u].w : 0.0 };
            *reinterpret_cast<double2 *>( &X[r][c] ) = make_double2( x[0], x[1] );
            *reinterpret_cast<double2 *>( &X[r][c + 2] ) = make_double2( x[2], x[3] );
        }
    }
    cp_async_wait_all();
    __syncthreads();
    const int c = kSub * warp;                            // this warp's column tile
    if( c < cw )
    {
        const int fi = lane >> 2, fj = 2 * (lane & 3);
        double acc[kSubs][2];
#pragma unroll
        for( int rb = 0; rb < kSubs; ++rb ) { acc[rb][0] = 0.0; acc[rb][1] = 0.0; }
#pragma unroll
        for( int kb = 0; kb < kSubs; ++kb )
        {
            if( kb >= nbb ) { break; }
#pragma unroll
            for( int q = 0; q < 2; ++q )
            {
                const int k = kSub * kb + (lane & 3) + 4 * q;
                const double b = X[k][c + fi];
                const double * Tk = Ti[k] + fi;
#pragma unroll
                for( int rb = kb; rb < kSubs; ++rb ) { dmma_8x8x4( acc[rb], Tk[kSub * rb], b ); }   // (rb >= nbb: unused sums)
            }
        }
#pragma unroll
        for( int rb = 0; rb < kSubs; ++rb )
        {
            const int r = kSub * rb + fi;
            if( r >= nb || c + fj >= cw ) { continue; }
            T * dst = U + (std::int64_t)r * ld + c + fj;
            const bool two = c + fj + 1 < cw;
            const T v0 = static_cast<T>( acc[rb][0] ), v1 = static_cast<T>( acc[rb][1] );
            if constexpr ( sizeof(T) == 8 )
            {
                if( two ) { *reinterpret_cast<double2 *>( dst ) = make_double2( v0, v1 ); }
                else { dst[0] = v0; }
            }
            else
            {
                if( two ) { *reinterpret_cast<float2 *>( dst ) = make_float2( v0, v1 ); }
                else { dst[0] = v0; }
                if( img != nullptr && t.img >= 0 )
                {
                    // the stored FP32 values split into TF32 hi + lo, for the tensor-core tiles: the image
                    // is K-major, so eight lanes write eight consecutive k of a column (one 32-byte sector)
                    const std::int64_t lo_off = static_cast<std::int64_t>( t.img_tf ) * (kImgRows * kImgK);
#pragma unroll
                    for( int e = 0; e < 2; ++e )
                    {
                        if( e == 1 && !two ) { continue; }
                        const float v = e == 0 ? v0 : v1;
                        const unsigned hi = to_tf32( v );
                        const std::int64_t o = img_offset( t, t.r0 + r, t.c0 + c + fj + e, r1, m );
                        img[o] = __uint_as_float( hi );
                        img[o + lo_off] = __uint_as_float( to_tf32( v - __uint_as_float( hi ) ) );
                    }
                }
            }
        }
    }
    if constexpr ( sizeof(T) == 4 )
    {
        // the last panel: image rows n0 .. (n0 rounded up to the 32-row k-chunk) are zero, so
        // that the update matrix's tiles (K = n0) can read whole chunks
        if( img != nullptr && t.img >= 0 && t.r0 + nb == t.n0 )
        {
            const int pad = (kImgK - t.n0 % kImgK) % kImgK;
            for( int idx = threadIdx.x; idx < pad * cw; idx += kTrsmThreads )
            {
                const int k = t.n0 + idx / cw, col = t.c0 + idx % cw;
                const std::int64_t o = img_offset( t, k, col, r1, m );
                img[o] = 0.0f;
                img[o + static_cast<std::int64_t>( t.img_tf ) * (kImgRows * kImgK)] = 0.0f;
            }
        }
    }
}

template<typename T, bool kPrefetch>
__global__ __launch_bounds__(kTrsmThreads) void trsm_kernel( const PanelTask * __restrict__ tasks,
                                                             T * __restrict__ arena, const double * __restrict__ tinv,
                                                             float * __restrict__ img )
{
    extern __shared__ __align__(16) double tsm[];
    pdl_allow_next();
    trsm_body<T, true, kPrefetch>( tasks[blockIdx.x], arena, tinv, tsm, img );
}

// ------------------------------------------------------------------- gemm
// C[m0:m0+64, c0:c0+64] -= A[:, m0:]^T B[:, c0:] for row-major K x M / K x N
// panels: 8 warps in a 2 x 4 arrangement, each a 32 x 16 block of 8 x 8
// DMMA tiles.  K is streamed through a kGemmStages-deep ring of shared-memory
// stages filled by 16-byte cp.async copies (every operand row starts on a
// 16-byte boundary: the plan pads leading dimensions to kLdAlign), so the
// copies of the next chunks overlap the MMAs of the current one.
constexpr int kGemmStages = 3;
constexpr int kGemmStageDoubles = 2 * kGemmK * kGemmLd;          // A and B of one stage
constexpr size_t kGemmSmemBytes = sizeof(double) * kGemmStages * kGemmStageDoubles;

__device__ __forceinline__ void gemm_body( const GemmTask & t, double * __restrict__ arena, double * gsm )
{
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int wm = warp & 1, wn = warp >> 1;
    const double * A = arena + t.a;
    const double * B = arena + t.b;

    double acc[4][2][2];
#pragma unroll
    for( int i = 0; i < 4; ++i )
#pragma unroll
        for( int j = 0; j < 2; ++j ) { acc[i][j][0] = 0.0; acc[i][j][1] = 0.0; }

    // Each stage holds kGemmK rows of 64 doubles for A and for B = 512
    // 16-byte chunks per operand; thread tid copies chunks tid + 256 * l.
    constexpr int kChunks = kGemmK * kTile / 2 / kGemmThreads;       // 2 per operand
    auto issue = [&]( int stage, int k0 )
    {
        double * As = gsm + stage * kGemmStageDoubles;
        double * Bs = As + kGemmK * kGemmLd;
#pragma unroll
        for( int l = 0; l < kChunks; ++l )
        {
            const int idx = tid + kGemmThreads * l;
            const int r = idx / (kTile / 2), c = 2 * (idx % (kTile / 2));
            const int k = k0 + r;
            const int am = t.M - (t.m0 + c), bn = t.N - (t.c0 + c);
            const int abytes = (k < t.K) ? (am >= 2 ? 16 : (am == 1 ? 8 : 0)) : 0;
            const int bbytes = (k < t.K) ? (bn >= 2 ? 16 : (bn == 1 ? 8 : 0)) : 0;
            cp_async_16( As + r * kGemmLd + c, abytes ? A + (std::int64_t)k * t.lda + t.m0 + c : A, abytes );
            cp_async_16( Bs + r * kGemmLd + c, bbytes ? B + (std::int64_t)k * t.ldb + t.c0 + c : B, bbytes );
        }
    };

    const int nk = (t.K + kGemmK - 1) / kGemmK;
#pragma unroll
    for( int s = 0; s < kGemmStages - 1; ++s )
    {
        if( s < nk ) { issue( s, s * kGemmK ); }
        cp_async_commit();
    }
    for( int kc = 0; kc < nk; ++kc )
    {
        cp_async_wait<kGemmStages - 2>();
        __syncthreads();
        {
            const int nxt = kc + kGemmStages - 1;
            if( nxt < nk ) { issue( nxt % kGemmStages, nxt * kGemmK ); }
            cp_async_commit();
        }
        const double * As = gsm + (kc % kGemmStages) * kGemmStageDoubles;
        const double * Bs = As + kGemmK * kGemmLd;
#pragma unroll
        for( int kk = 0; kk < kGemmK; kk += 4 )
        {
            double af[4], bf[2];
#pragma unroll
            for( int i = 0; i < 4; ++i ) { af[i] = As[(kk + (lane & 3)) * kGemmLd + wm * 32 + i * 8 + (lane >> 2)]; }
#pragma unroll
            for( int j = 0; j < 2; ++j ) { bf[j] = Bs[(kk + (lane & 3)) * kGemmLd + wn * 16 + j * 8 + (lane >> 2)]; }
#pragma unroll
            for( int i = 0; i < 4; ++i )
#pragma unroll
                for( int j = 0; j < 2; ++j ) { dmma_8x8x4( acc[i][j], af[i], bf[j] ); }
        }
    }
    cp_async_wait<0>();
    // the ring is reused by the next task of a persistent CTA
    __syncthreads();

    // C -= acc as reductions in the memory system (no load round trip); every C
    // entry gets one contribution per launch, so the result is the plain C - acc
    double * C = arena + t.c;
#pragma unroll
    for( int i = 0; i < 4; ++i )
    {
        const int row = t.m0 + wm * 32 + i * 8 + (lane >> 2);
        if( row >= t.M ) { continue; }
        double * Crow = C + (std::int64_t)row * t.ldc;
#pragma unroll
        for( int j = 0; j < 2; ++j )
        {
            const int col = t.c0 + wn * 16 + j * 8 + (lane & 3) * 2;
            if( col < t.N && (!t.upper || row <= col) ) { red_add_f64( Crow + col, -acc[i][j][0] ); }
            if( col + 1 < t.N && (!t.upper || row <= col + 1) ) { red_add_f64( Crow + col + 1, -acc[i][j][1] ); }
        }
    }
}

// FP32 storage: the same tiles as split-precision 3xTF32 products on the
// 5th-generation tensor cores (x = hi + lo with hi, lo TF32; a b ~ a_lo b_hi +
// a_hi b_lo + a_hi b_hi, FP32 accumulation in tensor memory).  K is streamed
// in chunks of 32 rows through two shared-memory stages; every chunk is read
// from global memory into registers one chunk ahead (a warp reads 4 rows of
// 8 consecutive floats), split, and stored in the canonical K-major
// no-swizzle layout of tcgen05 operands: core matrices of 8 (m or n) rows x
// 4 k (16 B per row, 128 B per core matrix), the 8 row groups 128 B apart
// (stride byte offset) and the k groups of 4 1024 B apart (leading byte
// offset).  One thread issues the 12 tcgen05.mma (M = N = 64, K = 8) of a
// chunk and commits them to the stage's mbarrier; the stage is refilled once
// that barrier has completed.  The 64 x 64 accumulator is read back with
// tcgen05.ld, staged in shared memory and subtracted from C with coalesced
// 16-byte accesses (the plan keeps C offsets and leading dimensions
// multiples of 4 floats).
constexpr int kTcK = 32;                               // k rows per chunk
constexpr int kTcPart = kTcK * kTile * 4;              // one operand part (64 x 32 TF32): 8 KB
constexpr int kTcStage = 4 * kTcPart;                  // A_hi, A_lo, B_hi, B_lo
constexpr size_t kGemmSmemBytesF = 2 * kTcStage;       // 64 KB
constexpr int kTcSld = kTile + 4;                      // staged result row (floats)
constexpr int kTcCols = 64;                            // tensor-memory columns per CTA (FP32 accumulator 64 x 64)
constexpr unsigned kTcMaxPolls = 1u << 24;             // bound on the polls of one mbarrier wait
constexpr unsigned long long kTcTimeoutNs = 1000000000ull;
constexpr int kStatusTcTimeout = 2;                    // status[0] bit: a tensor-core completion wait ran out
static_assert( kGemmSmemBytesF >= sizeof(float) * kTile * kTcSld, "result staging does not fit" );

__device__ __forceinline__ std::uint32_t smem_u32( const void * p )
{
    return static_cast<std::uint32_t>( __cvta_generic_to_shared( p ) );
}

__device__ __forceinline__ unsigned long long tc_now()
{
    unsigned long long t;
    asm volatile( "mov.u64 %0, %%globaltimer;\n" : "=l"(t) );
    return t;
}

__device__ __forceinline__ int ld_acquire_i32( const int * p )
{
    int v;
    asm volatile( "ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory" );
    return v;
}

// Waits until the mbarrier phase of the given parity has completed; false
// when the wait ran out (polls or time).
__device__ __forceinline__ bool tc_wait( std::uint32_t bar, std::uint32_t parity )
{
    const unsigned long long start = tc_now();
    for( unsigned i = 0; i < kTcMaxPolls; ++i )
    {
        std::uint32_t done;
        asm volatile( "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                      : "=r"(done) : "r"(bar), "r"(parity) : "memory" );
        if( done ) { return true; }
        if( (i & 1023u) == 1023u && tc_now() - start > kTcTimeoutNs ) { return false; }
    }
    return false;
}

// Per-CTA tensor-core state: the accumulator's tensor-memory address, the two
// stage mbarriers and the number of commits made to each (the parity of the
// next completion to wait for), carried across the tasks of a persistent CTA.
struct TcState
{
    std::uint32_t tmem;
    std::uint32_t bar;            // shared address of bar[0]; bar[1] = bar + 8
    unsigned commits0, commits1;  // commits made to bar[0] / bar[1]
    __device__ unsigned commits( int s ) const { return s ? commits1 : commits0; }
};

// All threads of the CTA; warp 0 allocates the accumulator columns.
__device__ __forceinline__ TcState tc_setup( std::uint64_t * bars, std::uint32_t * s_tmem )
{
    if( threadIdx.x == 0 )
    {
        asm volatile( "mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32( bars )) );
        asm volatile( "mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32( bars + 1 )) );
        asm volatile( "fence.mbarrier_init.release.cluster;\n" ::: "memory" );
    }
    if( (threadIdx.x >> 5) == 0 )
    {
        asm volatile( "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" :: "r"(smem_u32( s_tmem )), "r"(kTcCols) );
        asm volatile( "tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" );
    }
    asm volatile( "tcgen05.fence::before_thread_sync;\n" ::: "memory" );
    __syncthreads();
    asm volatile( "tcgen05.fence::after_thread_sync;\n" ::: "memory" );
    TcState tc;
    tc.tmem = *s_tmem;
    tc.bar = smem_u32( bars );
    tc.commits0 = 0;
    tc.commits1 = 0;
    return tc;
}

// All threads of the CTA, after its last task: frees the accumulator columns.
__device__ __forceinline__ void tc_teardown( const TcState & tc )
{
    asm volatile( "tcgen05.fence::before_thread_sync;\n" ::: "memory" );
    __syncthreads();
    if( (threadIdx.x >> 5) == 0 )
    {
        asm volatile( "tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" :: "r"(tc.tmem), "r"(kTcCols) );
    }
}

// Shared-memory matrix descriptor of one K-major no-swizzle operand part:
// start address, leading byte offset 1024 (next 4 k), stride byte offset 128
// (next 8 rows), descriptor version 1 (sm_100), no swizzle.
__device__ __forceinline__ std::uint64_t tc_desc( std::uint32_t addr )
{
    return static_cast<std::uint64_t>( (addr >> 4) & 0x3FFFu ) | (static_cast<std::uint64_t>( 1024 >> 4 ) << 16)
         | (static_cast<std::uint64_t>( 128 >> 4 ) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::tf32: FP32 accumulator, TF32 A and B, both
// K-major, N = 64 (bits 17-22: N / 8), M = 64 (bits 24-28: M / 16).
constexpr std::uint32_t kTcIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((64u >> 3) << 17) | ((64u >> 4) << 24);

__device__ __forceinline__ void gemm_body( const GemmTask & t, float * __restrict__ arena, double * smem, TcState & tc,
                                           int * status )
{
    unsigned char * sm = reinterpret_cast<unsigned char *>( smem );
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // this thread's elements of every chunk: k = 4 i + kl (i = 0..7), row mn of A and of B
    const int mn = 8 * warp + (lane & 7), kl = lane >> 3;
    const bool a_ok = t.m0 + mn < t.M, b_ok = t.c0 + mn < t.N;
    const float * A = arena + t.a;
    const float * B = arena + t.b;
    const std::int64_t acol = t.m0 + mn, bcol = t.c0 + mn;
    const int soff = warp * 128 + (lane & 7) * 16 + kl * 4;   // K-major offset of (mn, kl) in a part
    const int nk = (t.K + kTcK - 1) / kTcK;
    float ra[8], rb[8];
    auto load = [&]( int c )
    {
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            const int k = c * kTcK + 4 * i + kl;
            ra[i] = (k < t.K && a_ok) ? A[(std::int64_t)k * t.lda + acol] : 0.0f;
            rb[i] = (k < t.K && b_ok) ? B[(std::int64_t)k * t.ldb + bcol] : 0.0f;
        }
    };
    if( nk > 0 ) { load( 0 ); }
    bool ok = true;
    for( int c = 0; c < nk; ++c )
    {
        const int s = c & 1;
        unsigned char * st = sm + s * kTcStage;
        float ca[8], cb[8];
#pragma unroll
        for( int i = 0; i < 8; ++i ) { ca[i] = ra[i]; cb[i] = rb[i]; }
        if( c + 1 < nk ) { load( c + 1 ); }
        // the stage is free once the MMAs of its previous chunk have completed
        const bool mine = (tc.commits( s ) == 0) || tc_wait( tc.bar + 8 * s, (tc.commits( s ) & 1u) ^ 1u );
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            const unsigned ha = to_tf32( ca[i] ), hb = to_tf32( cb[i] );
            const int o = i * 1024 + soff;
            *reinterpret_cast<unsigned *>( st + o ) = ha;
            *reinterpret_cast<unsigned *>( st + kTcPart + o ) = to_tf32( ca[i] - __uint_as_float( ha ) );
            *reinterpret_cast<unsigned *>( st + 2 * kTcPart + o ) = hb;
            *reinterpret_cast<unsigned *>( st + 3 * kTcPart + o ) = to_tf32( cb[i] - __uint_as_float( hb ) );
        }
        asm volatile( "fence.proxy.async.shared::cta;\n" ::: "memory" );
        if( __syncthreads_or( mine ? 0 : 1 ) ) { ok = false; break; }
        if( tid == 0 )
        {
            asm volatile( "tcgen05.fence::after_thread_sync;\n" ::: "memory" );
            const std::uint32_t base = smem_u32( st );
#pragma unroll
            for( int ks = 0; ks < kTcK / 8; ++ks )
            {
                const std::uint32_t off = ks * 2048;
                const std::uint64_t ahi = tc_desc( base + off ), alo = tc_desc( base + kTcPart + off );
                const std::uint64_t bhi = tc_desc( base + 2 * kTcPart + off ), blo = tc_desc( base + 3 * kTcPart + off );
                const std::uint64_t ad[3] = { alo, ahi, ahi }, bd[3] = { bhi, blo, bhi };
#pragma unroll
                for( int u = 0; u < 3; ++u )
                {
                    const std::uint32_t accumulate = (c > 0 || ks > 0 || u > 0) ? 1u : 0u;
                    asm volatile( "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                  "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n"
                                  :: "r"(tc.tmem), "l"(ad[u]), "l"(bd[u]), "r"(kTcIdesc), "r"(accumulate) );
                }
            }
            asm volatile( "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                          :: "r"(tc.bar + 8 * s) : "memory" );
        }
        if( s ) { ++tc.commits1; } else { ++tc.commits0; }
    }
    // every commit of both stages complete: the accumulator is final and the
    // stages are free for the next task
    bool fine = ok;
#pragma unroll
    for( int s = 0; s < 2; ++s )
    {
        if( fine && tc.commits( s ) > 0 ) { fine = tc_wait( tc.bar + 8 * s, (tc.commits( s ) & 1u) ^ 1u ); }
    }
    if( __syncthreads_or( fine ? 0 : 1 ) )
    {
        if( tid == 0 )
        {
            atomicOr( status, kStatusTcTimeout );
            // one more bounded wait for the MMAs in flight before the memory is reused
            for( int s = 0; s < 2; ++s ) { if( tc.commits( s ) > 0 ) { tc_wait( tc.bar + 8 * s, (tc.commits( s ) & 1u) ^ 1u ); } }
        }
        __syncthreads();
        return;
    }
    if( nk == 0 ) { return; }
    asm volatile( "tcgen05.fence::after_thread_sync;\n" ::: "memory" );
    float * S = reinterpret_cast<float *>( sm );
    {
        // warp w reads accumulator rows 16 (w % 4) .. +15 (tensor-memory lanes 32 (w % 4) .. +15 for
        // M = 64), columns 32 (w / 4) .. +31
        const int q = warp & 3, h = warp >> 2;
        std::uint32_t v[32];
        asm volatile( "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
                      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                      : "r"(tc.tmem + ((std::uint32_t)(32 * q) << 16) + 32 * h) );
        asm volatile( "tcgen05.wait::ld.sync.aligned;\n" ::: "memory" );
        asm volatile( "tcgen05.fence::before_thread_sync;\n" ::: "memory" );
        if( lane < 16 )
        {
            float4 * dst = reinterpret_cast<float4 *>( S + (16 * q + lane) * kTcSld + 32 * h );
#pragma unroll
            for( int j = 0; j < 8; ++j )
            {
                dst[j] = make_float4( __uint_as_float( v[4 * j] ), __uint_as_float( v[4 * j + 1] ),
                                      __uint_as_float( v[4 * j + 2] ), __uint_as_float( v[4 * j + 3] ) );
            }
        }
    }
    __syncthreads();
    float * C = arena + t.c;
    const int cq = 4 * (tid & 15);
    const int col = t.c0 + cq;
#pragma unroll
    for( int i = 0; i < 4; ++i )
    {
        const int r = (tid >> 4) + 16 * i;
        const int row = t.m0 + r;
        if( row >= t.M || col >= t.N ) { continue; }
        const float4 d = *reinterpret_cast<const float4 *>( S + r * kTcSld + cq );
        float * Cp = C + (std::int64_t)row * t.ldc + col;
        if( col + 3 < t.N && (!t.upper || row <= col) )
        {
            red_add_v4f32( Cp, -d.x, -d.y, -d.z, -d.w );
        }
        else
        {
            const float dv[4] = { d.x, d.y, d.z, d.w };
#pragma unroll
            for( int j = 0; j < 4; ++j )
            {
                if( col + j < t.N && (!t.upper || row <= col + j) ) { atomicAdd( Cp + j, -dv[j] ); }
            }
        }
    }
    // the staged result and the accumulator are reused by the next task
    __syncthreads();
}

// One CTA per SM slot, looping over the launch's tiles with its tensor memory
// held throughout.
__global__ __launch_bounds__(kGemmThreads, 3) void gemm_tc_kernel( const GemmTask * __restrict__ tasks, int count,
                                                                  float * __restrict__ arena, int * status )
{
    extern __shared__ __align__(16) double gsm[];
    __shared__ std::uint64_t bars[2];
    __shared__ std::uint32_t s_tmem;
    pdl_allow_next();
    pdl_wait();
    TcState tc = tc_setup( bars, &s_tmem );
    for( int i = blockIdx.x; i < count; i += gridDim.x ) { gemm_body( tasks[i], arena, gsm, tc, status ); }
    tc_teardown( tc );
}

__global__ __launch_bounds__(kGemmThreads) void gemm_tn_kernel( const GemmTask * __restrict__ tasks,
                                                                double * __restrict__ arena )
{
    extern __shared__ __align__(16) double gsm[];
    pdl_allow_next();
    const GemmTask t = tasks[blockIdx.x];
    pdl_wait();
    gemm_body( t, arena, gsm );
}

// ------------------------------------------------------------------ solves
// The supernodal solves (LowerSolver.hpp:143-305, UpperSolver.hpp:127-255)
// run as one launch per (level, panel step) and sweep.  The triangular solves
// with the 64 x 64 diagonal blocks become products with their inverses
// (computed by the panel potrf), so every CTA of a step can form the panel's
// solution itself and no CTA waits for another.

constexpr int kTld = kPanel + 4;   // padded shared-memory row of 64-wide blocks (conflict-free DMMA fragments)

// acc[ct] (8 x 8 tile ct of this warp's 8 output rows, NCT tiles) += sum over
// the K blocks [kb0, kb1) of A(i, kk) * B(kk, ct * 8 + j).
template<int NCT, typename FA, typename FB>
__device__ __forceinline__ void warp_rows_product( double (&acc)[NCT][2], int kb0, int kb1, FA a, FB b )
{
    for( int kb = kb0; kb < kb1; ++kb )
    {
#pragma unroll
        for( int ct = 0; ct < NCT; ++ct )
        {
            dmma_8x8x8( acc[ct], [&]( int i, int kk ) { return a( i, kb * 8 + kk ); },
                                 [&]( int kk, int j ) { return b( kb * 8 + kk, ct * 8 + j ); } );
        }
    }
}

// Stages rows row(0..nr) (leading dimension ld, k columns) of a sweep vector x
// into V (64 x KP, leading dimension KP + 4); cells outside nr x k are zero.
// 16-byte copies where every row starts on a 16-byte boundary (x does).
template<int KP, typename RowOf>
__device__ __forceinline__ void stage_rows( double * V, const double * x, RowOf row, int nr, int ld, int k )
{
    constexpr int ldv = KP + 4;
    if( ((ld | k) & 1) == 0 )
    {
#pragma unroll
        for( int u = 0; u < kPanel * KP / 512; ++u )
        {
            const int idx = 2 * (threadIdx.x + 256 * u), r = idx / KP, c = idx % KP;
            const bool ok = r < nr && c < k;
            cp_async_16( V + r * ldv + c, ok ? x + row( r ) * ld + c : x, ok ? 16 : 0 );
        }
    }
    else
    {
#pragma unroll 4
        for( int idx = threadIdx.x; idx < kPanel * KP; idx += 256 )
        {
            const int r = idx / KP, c = idx % KP;
            const bool ok = r < nr && c < k;
            cp_async_8( V + r * ldv + c, ok ? x + row( r ) * ld + c : x, ok );
        }
    }
}

// One solve step.  Forward (U^T y = b): every task forms x_q = T_q^T y_q for
// the panel's rows of `in`; the owner writes x_q to `out`, and a task with
// rest rows subtracts P^T x_q from its (up to) 64 rest rows of `in` (rows of
// the front in place, ancestor rows by atomic adds: other fronts of the level
// may target them).  Backward (U x = y): `out` starts at zero on the panel's
// rows; a task adds T_q (y_q - P x_r) (owner) or -T_q P x_r, with x_r its rest
// rows of `out`, already final.  The owner is the task with c0 <= 0: the
// first rest chunk, or a rest-less task for a front's last panel without
// rest.  Warp w owns rows 8w..8w+7 of every 64 x KP product (KP = k rounded
// up to a power of two >= 8) as 8 x 8 DMMA tiles and skips row and K blocks
// beyond the panel's nb rows and the task's cw rest rows; only the used
// block of T is copied.  The body is instantiated per KP: with the tile
// counts known at compile time the tile loops unroll and the accumulators
// take only the registers they need (a task ran 11.6 us with KP a run-time
// value and 7 us with it fixed, 64^3 Laplacian with 16 RHS).
//
// atomic_own: rows of the task's own front are updated with atomics too (the
// task-graph solve, where panels of one front can run concurrently).
//
// kPdl: launched with programmatic stream serialization; the factor blocks (T,
// the rest block) and the rest rows' indices are loaded before pdl_wait, the
// vectors the previous step writes only after it.
template<typename T, int KP, bool kPdl = false>
__device__ __forceinline__ void solve_step_body( const SolveRestTask & t, int upper, const T * __restrict__ arena,
                                                 const double * __restrict__ tinv,
                                                 const std::int32_t * __restrict__ sn_inner,
                                                 double * in, double * out, int ld, int k, bool atomic_own, double * ssm )
{
    constexpr int kp = KP;
    constexpr int lkp = KP == 8 ? 3 : KP == 16 ? 4 : KP == 32 ? 5 : 6;
    constexpr int ldv = kp + 4;
    double (*sT)[kTld] = reinterpret_cast<double (*)[kTld]>( ssm );
    double * sX = ssm + kPanel * kTld;              // [64][ldv]: x_q (forward) / x_r (backward)
    double * sY = sX + kPanel * ldv;                // [64][ldv]: y_q
    __shared__ std::int64_t trow[kSolveRest];
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int nct = kp >> 3;
    const int nb = min( kPanel, t.n0 - t.r0 );
    const int nbb = (nb + 7) >> 3;
    const int r1 = t.r0 + nb;
    const int m = t.n0 - r1;
    const bool owner = t.c0 <= 0;
    const bool has_rest = t.c0 >= 0;
    const int cw = has_rest ? t.c1 - t.c0 : 0;
    const std::int64_t prow = (std::int64_t)t.row0 + t.r0;

    {
        // only the leading (nb rounded up to 8)^2 block of T is read below
        const double * Tg = tinv + (std::int64_t)t.panel * (kPanel * kPanel);
        const int nbp = 8 * nbb;
#pragma unroll
        for( int u = 0; u < kPanel * kPanel / (2 * kSolveThreads); ++u )
        {
            const int idx = 2 * (tid + u * kSolveThreads);
            const bool used = (idx >> 6) < nbp && (idx & 63) < nbp;
            cp_async_16( &sT[idx >> 6][idx & 63], used ? Tg + idx : Tg, used ? 16 : 0 );
        }
    }
    if( tid < kSolveRest )
    {
        const int col = t.c0 + tid;
        trow[tid] = (tid < cw) ? ((col < m) ? (std::int64_t)t.row0 + r1 + col
                                            : (std::int64_t)sn_inner[t.inner + (col - m)]) : -1;
    }
    // The panel's rest block P (factor data: final before any solve step) goes straight into
    // registers as this warp's DMMA A fragments (lane: row lane / 4 of the 8-row tile, K index
    // lane % 4 + 4 s of each 8-wide K block kb), loaded before the wait on the previous launch.
    // Forward: A(i, K) = P[K][o + i] (K over the panel's rows); back: A(i, K) = P[o + i][K]
    // (K over the rest columns).  Without a staged copy of P a CTA needs 35 KB (FP64) or
    // 17 KB (FP32) less shared memory, so more CTAs share an SM.
    const T * U0 = arena + t.u0 + (std::int64_t)t.r0 * t.ld0;
    const T * U1 = arena + t.u1 + (std::int64_t)t.r0 * t.ld1;
    const int o = warp * 8;
    T pf[kPanel / 8][2];
    {
        auto rest_at = [&]( int i, int cc ) -> T
        {
            const int col = t.c0 + cc;
            return (col < m) ? U0[(std::int64_t)i * t.ld0 + r1 + col] : U1[(std::int64_t)i * t.ld1 + (col - m)];
        };
#pragma unroll
        for( int kb = 0; kb < kPanel / 8; ++kb )
        {
#pragma unroll
            for( int s = 0; s < 2; ++s )
            {
                const int kk = 8 * kb + (lane & 3) + 4 * s;
                const int i = upper ? o + (lane >> 2) : kk;          // panel row
                const int cc = upper ? kk : o + (lane >> 2);         // rest column
                pf[kb][s] = (has_rest && i < nb && cc < cw) ? rest_at( i, cc ) : T( 0 );
            }
        }
    }
    if constexpr ( kPdl ) { pdl_wait(); }
    // y_q: the panel's rows of `in` (forward: every task; backward: the owner)
    const bool need_y = !upper || owner;
    stage_rows<KP>( sY, in, [&]( int i ) { return prow + i; }, need_y ? nb : 0, ld, k );
    __syncthreads();
    // x_r: the rest rows of `out`, final
    if( upper ) { stage_rows<KP>( sX, out, [&]( int i ) { return trow[i]; }, cw, ld, k ); }
    cp_async_wait_all();
    __syncthreads();

    const int fi = lane >> 2, fj = 2 * (lane & 3);     // accumulator fragment: row fi, columns fj, fj + 1
    double acc[nct][2];
    // acc += P-part (A fragments in pf) times rows of sX, K blocks [0, kbn)
    auto rest_product = [&]( int kbn )
    {
#pragma unroll
        for( int kb = 0; kb < kPanel / 8; ++kb )
        {
            if( kb >= kbn ) { break; }
#pragma unroll
            for( int ct = 0; ct < nct; ++ct )
            {
#pragma unroll
                for( int s = 0; s < 2; ++s )
                {
                    dmma_8x8x4( acc[ct], static_cast<double>( pf[kb][s] ),
                                sX[(8 * kb + (lane & 3) + 4 * s) * ldv + ct * 8 + (lane >> 2)] );
                }
            }
        }
    };
#pragma unroll
    for( int ct = 0; ct < nct; ++ct ) { acc[ct][0] = 0.0; acc[ct][1] = 0.0; }
    if( !upper )
    {
        // x_q = T^T y_q (T^T lower triangular: K blocks 0..warp)
        if( o < nb )
        {
            warp_rows_product<nct>( acc, 0, warp + 1, [&]( int i, int kk ) { return sT[kk][o + i]; },
                                                      [&]( int kk, int c ) { return sY[kk * ldv + c]; } );
#pragma unroll
            for( int ct = 0; ct < nct; ++ct )
            {
                sX[(o + fi) * ldv + ct * 8 + fj]     = acc[ct][0];
                sX[(o + fi) * ldv + ct * 8 + fj + 1] = acc[ct][1];
            }
        }
        __syncthreads();
        if( owner )
        {
            for( int idx = tid; idx < (kPanel << lkp); idx += kSolveThreads )
            {
                const int i = idx >> lkp, c = idx & (kp - 1);
                if( i < nb && c < k ) { out[(prow + i) * ld + c] = sX[i * ldv + c]; }
            }
        }
        if( !has_rest || o >= cw ) { return; }
        // rest rows: y_r -= P^T x_q
#pragma unroll
        for( int ct = 0; ct < nct; ++ct ) { acc[ct][0] = 0.0; acc[ct][1] = 0.0; }
        rest_product( nbb );
        const int jj = o + fi;
        if( jj < cw )
        {
            double * dst = in + trow[jj] * ld;
            const bool own_row = t.c0 + jj < m;
#pragma unroll
            for( int ct = 0; ct < nct; ++ct )
            {
#pragma unroll
                for( int e = 0; e < 2; ++e )
                {
                    const int c = ct * 8 + fj + e;
                    if( c < k )
                    {
                        if( own_row && !atomic_own ) { dst[c] -= acc[ct][e]; } else { atomicAdd( dst + c, -acc[ct][e] ); }
                    }
                }
            }
        }
    }
    else
    {
        // sY rows of this warp <- (owner ? y_q : 0) - P x_r
        if( has_rest && o < nb )
        {
            rest_product( (cw + 7) >> 3 );
#pragma unroll
            for( int ct = 0; ct < nct; ++ct )
            {
#pragma unroll
                for( int e = 0; e < 2; ++e )
                {
                    double & v = sY[(o + fi) * ldv + ct * 8 + fj + e];
                    v = (owner ? v : 0.0) - acc[ct][e];
                }
            }
        }
        __syncthreads();
        if( o >= nb ) { return; }
        // z = T (.) (T upper triangular: K blocks warp..nbb-1)
#pragma unroll
        for( int ct = 0; ct < nct; ++ct ) { acc[ct][0] = 0.0; acc[ct][1] = 0.0; }
        warp_rows_product<nct>( acc, warp, nbb, [&]( int i, int kk ) { return sT[o + i][kk]; },
                                                [&]( int kk, int c ) { return sY[kk * ldv + c]; } );
        const int i = o + fi;
        if( i < nb )
        {
            double * dst = out + (prow + i) * ld;
#pragma unroll
            for( int ct = 0; ct < nct; ++ct )
            {
#pragma unroll
                for( int e = 0; e < 2; ++e )
                {
                    const int c = ct * 8 + fj + e;
                    if( c < k ) { atomicAdd( dst + c, acc[ct][e] ); }
                }
            }
        }
    }
}

// The same step of a tiny front (Launch::small_count) by one warp: no shared
// memory, every operand is loaded from global memory as the DMMA fragment it is
// used as, 16 columns of the right-hand sides at a time, and the product with T
// changes from accumulator to operand layout by shuffles.  A CTA per such front
// spent its time on two block barriers and on occupancy (2 to 4 an SM); of a
// grid's leaves half have one row and six rest rows.  C2 with 16 right-hand
// sides 1.22 -> 1.11 ms, 56^3 with 64 2.01 -> 1.89 ms, 96 meshes 481 -> 403 us.
template<typename T, int KP>
__device__ __forceinline__ void solve_warp_body( const SolveRestTask & t, int upper, const T * __restrict__ arena,
                                                 const double * __restrict__ tinv, const std::int32_t * __restrict__ sn_inner,
                                                 double * in, double * out, int ld, int k )
{
    constexpr int NC = KP == 8 ? 1 : 2;                  // 8-column tiles at a time
    constexpr int NT = kTinyRows / 8;
    const int lane = threadIdx.x & 31, fq = lane >> 2, fr = lane & 3;
    const int nb = t.n0, nt = (nb + 7) >> 3;             // (one panel: every rest column lies in U1)
    const bool owner = t.c0 <= 0;
    const int c0 = max( t.c0, 0 ), cw = t.c0 >= 0 ? t.c1 - t.c0 : 0;
    const std::int64_t prow = t.row0;
    const double * Tg = tinv + (std::int64_t)t.panel * (kPanel * kPanel);
    const T * P = arena + t.u1 + c0;
    const std::int32_t * rest = sn_inner + t.inner + c0;
    // accumulator tile (row fq, columns 2 fr, 2 fr + 1) -> operand (row fr + 4 s, column fq)
    auto turned = [&]( const double (&v)[2], int s )
    {
        const int src = 4 * (fr + 4 * s) + (fq >> 1);
        const double a = __shfl_sync( 0xffffffffu, v[0], src ), b = __shfl_sync( 0xffffffffu, v[1], src );
        return (fq & 1) ? b : a;
    };
    for( int cb = 0; cb < k; cb += 8 * NC )
    {
        double v[NT][2][NC];                             // operand: y, then x (forward); y - P x_r (back)
        if( !upper )
        {
#pragma unroll
            for( int kb = 0; kb < NT; ++kb )
            {
#pragma unroll
                for( int s = 0; s < 2; ++s )
                {
#pragma unroll
                    for( int ct = 0; ct < NC; ++ct )
                    {
                        const int r = 8 * kb + fr + 4 * s, c = cb + 8 * ct + fq;
                        v[kb][s][ct] = r < nb && c < k ? in[(prow + r) * ld + c] : 0.0;
                    }
                }
            }
#pragma unroll
            for( int rt = NT - 1; rt >= 0; --rt )
            {
                if( rt >= nt ) { continue; }
                double acc[NC][2] = {};
#pragma unroll
                for( int kb = 0; kb <= rt; ++kb )
                {
#pragma unroll
                    for( int s = 0; s < 2; ++s )
                    {
                        const double a = Tg[(8 * kb + fr + 4 * s) * kPanel + 8 * rt + fq];
#pragma unroll
                        for( int ct = 0; ct < NC; ++ct ) { dmma_8x8x4( acc[ct], a, v[kb][s][ct] ); }
                    }
                }
#pragma unroll
                for( int ct = 0; ct < NC; ++ct )
                {
                    const int r = 8 * rt + fq, c = cb + 8 * ct + 2 * fr;
                    if( owner && r < nb )
                    {
                        if( c < k ) { out[(prow + r) * ld + c] = acc[ct][0]; }
                        if( c + 1 < k ) { out[(prow + r) * ld + c + 1] = acc[ct][1]; }
                    }
#pragma unroll
                    for( int s = 0; s < 2; ++s ) { v[rt][s][ct] = turned( acc[ct], s ); }
                }
            }
#pragma unroll 1
            for( int o = 0; o < cw; o += 8 )
            {
                const bool ok = o + fq < cw;
                const std::int64_t row = ok ? rest[o + fq] : 0;
                double a[NT][2];
#pragma unroll
                for( int kb = 0; kb < NT; ++kb )
                {
#pragma unroll
                    for( int s = 0; s < 2; ++s )
                    {
                        const int r = 8 * kb + fr + 4 * s;
                        a[kb][s] = ok && r < nb ? static_cast<double>( P[(std::int64_t)r * t.ld1 + o + fq] ) : 0.0;
                    }
                }
                double acc[NC][2] = {};
#pragma unroll
                for( int kb = 0; kb < NT; ++kb )
                {
                    if( kb >= nt ) { break; }
#pragma unroll
                    for( int s = 0; s < 2; ++s )
                    {
#pragma unroll
                        for( int ct = 0; ct < NC; ++ct ) { dmma_8x8x4( acc[ct], a[kb][s], v[kb][s][ct] ); }
                    }
                }
                if( ok )
                {
#pragma unroll
                    for( int ct = 0; ct < NC; ++ct )
                    {
                        const int c = cb + 8 * ct + 2 * fr;
                        if( c < k ) { red_add_f64( in + row * ld + c, -acc[ct][0] ); }
                        if( c + 1 < k ) { red_add_f64( in + row * ld + c + 1, -acc[ct][1] ); }
                    }
                }
            }
        }
        else
        {
            double acc[NT][NC][2] = {};
#pragma unroll 1
            for( int o = 0; o < cw; o += 8 )
            {
#pragma unroll
                for( int s = 0; s < 2; ++s )
                {
                    const int j = o + fr + 4 * s;
                    const std::int64_t row = j < cw ? rest[j] : 0;
                    double x[NC];
#pragma unroll
                    for( int ct = 0; ct < NC; ++ct )
                    {
                        const int c = cb + 8 * ct + fq;
                        x[ct] = j < cw && c < k ? out[row * ld + c] : 0.0;
                    }
#pragma unroll
                    for( int rt = 0; rt < NT; ++rt )
                    {
                        if( rt >= nt ) { break; }
                        const int r = 8 * rt + fq;
                        const double a = r < nb && j < cw ? static_cast<double>( P[(std::int64_t)r * t.ld1 + j] ) : 0.0;
#pragma unroll
                        for( int ct = 0; ct < NC; ++ct ) { dmma_8x8x4( acc[rt][ct], a, x[ct] ); }
                    }
                }
            }
#pragma unroll
            for( int rt = 0; rt < NT; ++rt )
            {
#pragma unroll
                for( int ct = 0; ct < NC; ++ct )
                {
                    const int r = 8 * rt + fq, c = cb + 8 * ct + 2 * fr;
                    double d[2];
#pragma unroll
                    for( int e = 0; e < 2; ++e ) { d[e] = (owner && r < nb && c + e < k ? in[(prow + r) * ld + c + e] : 0.0) - acc[rt][ct][e]; }
#pragma unroll
                    for( int s = 0; s < 2; ++s ) { v[rt][s][ct] = turned( d, s ); }
                }
            }
#pragma unroll
            for( int rt = 0; rt < NT; ++rt )
            {
                if( rt >= nt ) { break; }
                double z[NC][2] = {};
#pragma unroll
                for( int kb = rt; kb < NT; ++kb )
                {
                    if( kb >= nt ) { break; }
#pragma unroll
                    for( int s = 0; s < 2; ++s )
                    {
                        const double a = Tg[(8 * rt + fq) * kPanel + 8 * kb + fr + 4 * s];
#pragma unroll
                        for( int ct = 0; ct < NC; ++ct ) { dmma_8x8x4( z[ct], a, v[kb][s][ct] ); }
                    }
                }
                const int r = 8 * rt + fq;
                if( r < nb )
                {
#pragma unroll
                    for( int ct = 0; ct < NC; ++ct )
                    {
                        const int c = cb + 8 * ct + 2 * fr;
                        if( c < k ) { red_add_f64( out + (prow + r) * ld + c, z[ct][0] ); }
                        if( c + 1 < k ) { red_add_f64( out + (prow + r) * ld + c + 1, z[ct][1] ); }
                    }
                }
            }
        }
    }
}

// One kernel per right-hand-side width KP, so that each gets the registers it needs: a CTA for
// each of the first `ctas` tasks, a warp for each of the others.
template<typename T, int KP>
__global__ __launch_bounds__(kSolveThreads) void solve_step_kernel( const SolveRestTask * __restrict__ tasks, int ctas, int count, int upper,
                                                                    const T * __restrict__ arena,
                                                                    const double * __restrict__ tinv,
                                                                    const std::int32_t * __restrict__ sn_inner,
                                                                    double * in, double * out, int ld, int k )
{
    extern __shared__ __align__(16) double ssm[];
    pdl_allow_next();
    if( static_cast<int>( blockIdx.x ) < ctas )
    {
        solve_step_body<T, KP, true>( tasks[blockIdx.x], upper, arena, tinv, sn_inner, in, out, ld, k, false, ssm );
        return;
    }
    const int i = ctas + (blockIdx.x - ctas) * (kSolveThreads / 32) + (threadIdx.x >> 5);
    if( i >= count ) { return; }
    const SolveRestTask t = tasks[i];
    pdl_wait();
    solve_warp_body<T, KP>( t, upper, arena, tinv, sn_inner, in, out, ld, k );
}

// The solve's task graph (Plan::solve_*) as one persistent launch per sweep:
// CTAs take tasks in list order, thread 0 waits (bounded) until the task's
// inputs are final, the CTA runs the step body with atomic updates of every
// row, and thread 0 signals after a fence.  Forward: wait for the panel's
// expected contributions, signal every target panel.  Back: wait until every
// target panel has all of its tasks done, signal the task's own panel.
template<typename T, int KP>
__global__ __launch_bounds__(kSolveThreads) void solve_dag_kernel( const SolveDagArgs a, const T * __restrict__ arena,
                                                                   double * in, double * out, int ld, int k )
{
    extern __shared__ __align__(16) double ssm[];
    __shared__ int s_idx, s_ok;
    const int tid = threadIdx.x;
    for( ;; )
    {
        if( tid == 0 )
        {
            int idx = a.ntasks, ok = 0;
            if( *reinterpret_cast<volatile int *>( a.error ) == 0 ) { idx = atomicAdd( a.next, 1 ); }
            if( idx < a.ntasks )
            {
                const int ti = a.order[idx];
                const int g = ti - a.first_task;
                const unsigned long long start = tc_now();
                if( a.trace ) { a.trace[4 * (std::int64_t)idx] = start; a.trace[4 * (std::int64_t)idx + 3] = blockIdx.x; }
                ok = 1;
                // forward: one wait (the task's panel); back: one per target panel
                const int nw = a.upper ? static_cast<int>( a.target_ptr[g + 1] - a.target_ptr[g] ) : 1;
                for( int w = 0; w < nw && ok; ++w )
                {
                    const int pnl = a.upper ? a.targets[a.target_ptr[g] + w] : a.tasks[ti].panel - a.first_panel;
                    const int need = a.upper ? a.panel_tasks[pnl] : a.fwd_expected[pnl];
                    unsigned spins = 0;
                    while( ld_acquire_i32( a.counters + pnl ) < need )
                    {
                        ++spins;
                        if( (spins & 31u) == 0 )
                        {
                            if( *reinterpret_cast<volatile int *>( a.error ) != 0 ) { ok = 0; break; }
                            if( tc_now() - start > a.timeout_ns || spins > kDagMaxSpins )
                            {
                                atomicCAS( a.error, 0, idx + 1 );
                                ok = 0;
                                break;
                            }
                        }
                        __nanosleep( 64 );
                    }
                }
                if( a.trace ) { a.trace[4 * (std::int64_t)idx + 1] = tc_now(); }
            }
            s_idx = idx;
            s_ok = ok;
        }
        __syncthreads();
        const int idx = s_idx;
        if( idx >= a.ntasks || !s_ok ) { break; }
        const int ti = a.order[idx];
        solve_step_body<T, KP>( a.tasks[ti], a.upper, arena, a.tinv, a.sn_inner, in, out, ld, k, true, ssm );
        __threadfence();
        __syncthreads();
        if( tid == 0 )
        {
            if( a.trace ) { a.trace[4 * (std::int64_t)idx + 2] = tc_now(); }
            const int g = ti - a.first_task;
            if( a.upper ) { atomicAdd( a.counters + (a.tasks[ti].panel - a.first_panel), 1 ); }
            else
            {
                for( std::int64_t e = a.target_ptr[g]; e < a.target_ptr[g + 1]; ++e ) { atomicAdd( a.counters + a.targets[e], 1 ); }
            }
        }
    }
}

// ------------------------------------------------- persistent factorization
// The whole numeric factorization as one launch: each CTA repeatedly takes
// the next task of the plan's dependency-ordered list (an atomic ticket),
// waits until the task's counters reach their targets, runs the task body
// and increments its counters.  Tasks are taken in list order and every wait
// is satisfied by tasks earlier in the list, so the earliest unfinished task
// can always proceed; waits are nevertheless bounded in time, and a wait that
// runs out records the task in `error` and makes every CTA stop.
//
// Counter protocol: every thread fences its own writes of the task, the CTA
// synchronises, and thread 0 increments the counters (release); a waiting
// thread 0 reads counters with ld.acquire.gpu and the CTA synchronises
// before any thread touches the task's data.
constexpr int kDagThreads = 256;
constexpr size_t kDagSmemBytes = kPotrfSmemBytes > kGemmSmemBytes ? kPotrfSmemBytes : kGemmSmemBytes;
static_assert( kDagSmemBytes >= kTrsmSmemBytes && kDagSmemBytes >= kGemmSmemBytesF, "persistent kernel shared memory too small" );

__device__ __forceinline__ int ld_acquire( const int * p )
{
    int v;
    asm volatile( "ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory" );
    return v;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile( "mov.u64 %0, %%globaltimer;\n" : "=l"(t) );
    return t;
}

// Thread 0 only: 1 when all waits of the task are met, 0 on timeout or when
// another CTA has reported an error.
__device__ int dag_wait( const DagTask & t, const DagArgs & a, int idx )
{
    const unsigned long long start = global_ns();
    for( int i = 0; i < kDagWaits; ++i )
    {
        if( t.wait[i] < 0 ) { continue; }
        const int * c = a.counters + t.wait[i];
        unsigned spins = 0;
        while( ld_acquire( c ) < t.target[i] )
        {
            ++spins;
            if( (spins & 31u) == 0 )
            {
                if( *reinterpret_cast<volatile int *>( a.error ) != 0 ) { return 0; }
                if( global_ns() - start > a.timeout_ns || spins > kDagMaxSpins )
                {
                    atomicCAS( a.error, 0, idx + 1 );
                    return 0;
                }
            }
            __nanosleep( 100 );
        }
    }
    return 1;
}

template<typename T>
__global__ __launch_bounds__(kDagThreads, 3) void factor_dag_kernel( const DagArgs a )
{
    T * arena = static_cast<T *>( a.arena );
    extern __shared__ __align__(16) double dsm[];
    __shared__ int s_idx, s_ok;
    __shared__ std::uint64_t tc_bars[2];
    __shared__ std::uint32_t tc_tmem;
    const int tid = threadIdx.x;
    TcState tc{};
    if constexpr ( sizeof(T) == 4 ) { tc = tc_setup( tc_bars, &tc_tmem ); }
    for( ;; )
    {
        if( tid == 0 )
        {
            int idx = a.ntasks, ok = 0;
            if( *reinterpret_cast<volatile int *>( a.error ) == 0 ) { idx = atomicAdd( a.next, 1 ); }
            if( idx < a.ntasks )
            {
                const unsigned long long taken = a.trace ? global_ns() : 0ull;
                ok = dag_wait( a.tasks[idx], a, idx );
                if( a.trace )
                {
                    a.trace[4 * (std::int64_t)idx]     = taken;
                    a.trace[4 * (std::int64_t)idx + 1] = global_ns();
                    a.trace[4 * (std::int64_t)idx + 3] = blockIdx.x;
                }
            }
            s_idx = idx;
            s_ok = ok;
        }
        __syncthreads();
        const int idx = s_idx;
        if( idx >= a.ntasks || !s_ok ) { break; }
        const DagTask t = a.tasks[idx];
        switch( static_cast<LaunchKind>( t.kind ) )
        {
            case LaunchKind::Zero:   zero_body( a.zero[t.index], arena ); break;
            case LaunchKind::Extend: extend_body( a.extend[t.index], a.lut, arena ); break;
            case LaunchKind::Potrf:  potrf_body<T, kDagThreads, false>( a.potrf[t.index], arena, a.status, a.pivot_floor, a.tinv ); break;
            case LaunchKind::Trsm:   trsm_body<T, false, false>( a.panel[t.index], arena, a.tinv, dsm ); break;
            case LaunchKind::Gemm:
                if constexpr ( sizeof(T) == 4 ) { gemm_body( a.gemm[t.index], arena, dsm, tc, a.status ); }
                else { gemm_body( a.gemm[t.index], arena, dsm ); }
                break;
            default: break;
        }
        __threadfence();
        __syncthreads();
        if( tid == 0 )
        {
            if( a.trace ) { a.trace[4 * (std::int64_t)idx + 2] = global_ns(); }
            if( t.signal[0] >= 0 ) { atomicAdd( a.counters + t.signal[0], 1 ); }
            if( t.signal[1] >= 0 ) { atomicAdd( a.counters + t.signal[1], 1 ); }
        }
    }
    if constexpr ( sizeof(T) == 4 ) { tc_teardown( tc ); }
}

// ------------------------------------------------------ permutations, SpMV
// W rows (kw columns) <- rows p[i] of B (k columns), columns k..kw-1 zero.
__global__ void gather_rows_kernel( const double * __restrict__ B, int ldB, const std::int32_t * __restrict__ p,
                                    double * __restrict__ W, int ldw, int n, int k, int kw )
{
    const std::int64_t total = (std::int64_t)n * kw;
    for( std::int64_t e = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; e < total;
         e += (std::int64_t)gridDim.x * blockDim.x )
    {
        const std::int64_t i = e / kw;
        const int c = static_cast<int>( e % kw );
        W[i * ldw + c] = c < k ? B[(std::int64_t)p[i] * ldB + c] : 0.0;
    }
}

__global__ void scatter_rows_kernel( const double * __restrict__ W, int ldw, const std::int32_t * __restrict__ p_inv,
                                     double alpha, double beta, double * __restrict__ Y, int ldY, int n, int k )
{
    const std::int64_t total = (std::int64_t)n * k;
    for( std::int64_t e = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; e < total;
         e += (std::int64_t)gridDim.x * blockDim.x )
    {
        const std::int64_t i = e / k;
        const int c = static_cast<int>( e % k );
        double y = (alpha == 0.0) ? 0.0 : alpha * W[(std::int64_t)p_inv[i] * ldw + c];
        if( beta != 0.0 ) { y += beta * Y[i * ldY + c]; }
        Y[i * ldY + c] = y;
    }
}

// R = B - A X, one warp per row, lanes over the row's entries.
// R = B - (A + shift I) X (B != nullptr) or R = (A + shift I) X (B == nullptr)
// for row-major blocks with leading dimensions.  One warp per row: the lanes
// form 32 / KP groups of KP columns (KP = k rounded up to a power of two, at
// most 32); group g takes the row's entries g, g + G, ... (one broadcast load
// of the entry, one contiguous load of KP values of x's row), the groups'
// sums meet by log2(G) shuffles, and group 0 writes the row.  Blocks of 32
// columns when k > 32.
template<int KP>
__global__ __launch_bounds__(256) void spmv_rows_kernel( int n, const std::int64_t * __restrict__ outer, const std::int32_t * __restrict__ inner,
                                                         const double * __restrict__ vals, double shift,
                                                         const double * __restrict__ X, int ldx, const double * __restrict__ B, int ldb,
                                                         double * __restrict__ R, int ldr, int k )
{
    constexpr int G = 32 / KP;
    const int lane = threadIdx.x & 31;
    const int g = lane / KP, c = lane % KP;
    const std::int64_t warp = (blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x) >> 5;
    const std::int64_t warps = ((std::int64_t)gridDim.x * blockDim.x) >> 5;
    for( std::int64_t i = warp; i < n; i += warps )
    {
        const std::int64_t e0 = outer[i], e1 = outer[i + 1];
        for( int c0 = 0; c0 < k; c0 += KP )
        {
            const int col = c0 + c;
            const bool live = col < k;
            double s = 0.0;
#pragma unroll 4
            for( std::int64_t e = e0 + g; e < e1; e += G )
            {
                const double v = vals[e];
                const std::int64_t j = inner[e];
                if( live ) { s = fma( v, X[j * ldx + col], s ); }
            }
#pragma unroll
            for( int o = KP; o < 32; o <<= 1 ) { s += __shfl_xor_sync( 0xffffffffu, s, o ); }
            if( g == 0 && live )
            {
                const double ax = s + shift * X[i * ldx + col];
                R[i * ldr + col] = B ? B[i * ldb + col] - ax : ax;
            }
        }
    }
}

// The same product for k >= 3: a group of KP lanes takes a whole row (KP
// columns of it, blocks of 32 when k > 32), 32 / KP rows per warp, with no
// cross-lane sum; the rows a warp holds together are consecutive, so rows
// with the same pattern (the dofs of one node) share their x loads in L1.
template<int KP>
__global__ __launch_bounds__(256) void spmv_group_kernel( int n, const std::int64_t * __restrict__ outer, const std::int32_t * __restrict__ inner,
                                                          const double * __restrict__ vals, double shift,
                                                          const double * __restrict__ X, int ldx, const double * __restrict__ B, int ldb,
                                                          double * __restrict__ R, int ldr, int k )
{
    constexpr int G = 32 / KP;
    const int lane = threadIdx.x & 31;
    const int g = lane / KP, c = lane % KP;
    const std::int64_t grp = ((blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x) >> 5) * G + g;
    const std::int64_t groups = (((std::int64_t)gridDim.x * blockDim.x) >> 5) * G;
    for( std::int64_t i = grp; i < n; i += groups )
    {
        const std::int64_t e0 = outer[i], e1 = outer[i + 1];
        for( int c0 = 0; c0 < k; c0 += KP )
        {
            const int col = c0 + c;
            if( col >= k ) { continue; }
            // four independent sums keep four gathers of x in flight per lane
            double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
            std::int64_t e = e0;
            for( ; e + 4 <= e1; e += 4 )
            {
                const double v0 = vals[e], v1 = vals[e + 1], v2 = vals[e + 2], v3 = vals[e + 3];
                const std::int64_t j0 = inner[e], j1 = inner[e + 1], j2 = inner[e + 2], j3 = inner[e + 3];
                s0 = fma( v0, X[j0 * ldx + col], s0 );
                s1 = fma( v1, X[j1 * ldx + col], s1 );
                s2 = fma( v2, X[j2 * ldx + col], s2 );
                s3 = fma( v3, X[j3 * ldx + col], s3 );
            }
            for( ; e < e1; ++e ) { s0 = fma( vals[e], X[(std::int64_t)inner[e] * ldx + col], s0 ); }
            const double ax = ((s0 + s1) + (s2 + s3)) + shift * X[i * ldx + col];
            R[i * ldr + col] = B ? B[i * ldb + col] - ax : ax;
        }
    }
}

// out[c] += sum_i X[i][c] Y[i][c] (out zeroed by the caller).  The lanes form
// groups of KP columns as in spmv_rows_kernel, so that a warp reads whole
// rows; per block the columns' sums meet in shared memory and go out with one
// atomic addition per column.
template<int KP>
__global__ __launch_bounds__(256) void column_dots_kernel( const double * __restrict__ X, int ldx, const double * __restrict__ Y, int ldy,
                                                           int n, int k, double * __restrict__ out )
{
    constexpr int G = 32 / KP;
    __shared__ double part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane / KP, c = lane % KP;
    const std::int64_t gw = (blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x) >> 5;
    const std::int64_t warps = ((std::int64_t)gridDim.x * blockDim.x) >> 5;
    for( int c0 = 0; c0 < k; c0 += KP )
    {
        const int col = c0 + c;
        double s = 0.0;
        if( col < k )
        {
#pragma unroll 4
            for( std::int64_t i = gw * G + g; i < n; i += warps * G ) { s = fma( X[i * ldx + col], Y[i * ldy + col], s ); }
        }
#pragma unroll
        for( int o = KP; o < 32; o <<= 1 ) { s += __shfl_xor_sync( 0xffffffffu, s, o ); }
        if( g == 0 ) { part[warp][c] = s; }
        __syncthreads();
        if( threadIdx.x < KP && c0 + threadIdx.x < k )
        {
            double t = 0.0;
#pragma unroll
            for( int w = 0; w < 8; ++w ) { t += part[w][threadIdx.x]; }
            if( t != 0.0 ) { atomicAdd( out + c0 + threadIdx.x, t ); }
        }
        __syncthreads();
    }
}

// Conjugate-gradient updates with per-column scalars kept on the device:
// alpha_c = rz[c] / pq[c];  x += alpha p;  r -= alpha q.
__global__ void cg_update_xr_kernel( int n, int k, const double * __restrict__ rz, const double * __restrict__ pq,
                                     const double * __restrict__ p, const double * __restrict__ q,
                                     double * __restrict__ x, double * __restrict__ r )
{
    const std::int64_t total = (std::int64_t)n * k;
    for( std::int64_t e = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; e < total; e += (std::int64_t)gridDim.x * blockDim.x )
    {
        const int c = static_cast<int>( e % k );
        const double a = pq[c] != 0.0 ? rz[c] / pq[c] : 0.0;
        x[e] += a * p[e];
        r[e] -= a * q[e];
    }
}

// beta_c = rz_new[c] / rz_old[c];  p = z + beta p.
__global__ void cg_update_p_kernel( int n, int k, const double * __restrict__ rz_new, const double * __restrict__ rz_old,
                                    const double * __restrict__ z, double * __restrict__ p )
{
    const std::int64_t total = (std::int64_t)n * k;
    for( std::int64_t e = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; e < total; e += (std::int64_t)gridDim.x * blockDim.x )
    {
        const int c = static_cast<int>( e % k );
        const double b = rz_old[c] != 0.0 ? rz_new[c] / rz_old[c] : 0.0;
        p[e] = z[e] + b * p[e];
    }
}

// GMRES (GMRES.hpp): out[i k + c] += Q_i(:, c) . q(:, c) for the nq Krylov
// vectors Q_i (n x k each, nk apart); blockIdx.y = i.
__global__ void multi_dots_kernel( const double * __restrict__ Q, std::int64_t nk, const double * __restrict__ q,
                                   int n, int k, double * __restrict__ out )
{
    const double * Qi = Q + blockIdx.y * nk;
    for( int c = 0; c < k; ++c )
    {
        double s = 0.0;
        for( std::int64_t i = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; i < n; i += (std::int64_t)gridDim.x * blockDim.x )
        {
            s += Qi[i * k + c] * q[i * k + c];
        }
#pragma unroll
        for( int o = 16; o > 0; o >>= 1 ) { s += __shfl_xor_sync( 0xffffffffu, s, o ); }
        if( (threadIdx.x & 31) == 0 && s != 0.0 ) { atomicAdd( out + blockIdx.y * k + c, s ); }
    }
}

// q += sign * sum_{i < nq} coef[i k + c] Q_i(:, c).
__global__ void multi_axpy_kernel( const double * __restrict__ Q, std::int64_t nk, int nq, const double * __restrict__ coef,
                                   double sign, double * __restrict__ q, int n, int k )
{
    const std::int64_t total = (std::int64_t)n * k;
    for( std::int64_t e = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; e < total; e += (std::int64_t)gridDim.x * blockDim.x )
    {
        const int c = static_cast<int>( e % k );
        double s = 0.0;
        for( int i = 0; i < nq; ++i ) { s += coef[i * k + c] * Q[i * nk + e]; }
        q[e] += sign * s;
    }
}

// x(:, c) /= sqrt(sq[c]) where sq[c] > 0 (normalises by squared column norms).
__global__ void col_normalize_kernel( double * __restrict__ x, int n, int k, const double * __restrict__ sq )
{
    const std::int64_t total = (std::int64_t)n * k;
    for( std::int64_t e = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; e < total; e += (std::int64_t)gridDim.x * blockDim.x )
    {
        const int c = static_cast<int>( e % k );
        if( sq[c] > 0.0 ) { x[e] /= sqrt( sq[c] ); }
    }
}

__global__ void axpy_kernel( std::int64_t n, double a, const double * __restrict__ x, double * __restrict__ y )
{
    for( std::int64_t i = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; i < n; i += (std::int64_t)gridDim.x * blockDim.x )
    {
        y[i] += a * x[i];
    }
}

// Y = alpha X + beta Y (beta == 0: Y is not read).
__global__ void combine_kernel( int n, int k, double alpha, const double * __restrict__ X, int ldx,
                                double beta, double * __restrict__ Y, int ldy )
{
    const std::int64_t total = (std::int64_t)n * k;
    for( std::int64_t e = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; e < total; e += (std::int64_t)gridDim.x * blockDim.x )
    {
        const std::int64_t i = e / k;
        const int c = static_cast<int>( e % k );
        double y = alpha * X[i * ldx + c];
        if( beta != 0.0 ) { y += beta * Y[i * ldy + c]; }
        Y[i * ldy + c] = y;
    }
}

template<typename T>
__global__ void gather_diag_kernel( const std::int64_t * __restrict__ offsets, const T * __restrict__ arena,
                                    double * __restrict__ out, int n )
{
    for( std::int64_t i = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; i < n; i += (std::int64_t)gridDim.x * blockDim.x )
    {
        out[i] = static_cast<double>( arena[offsets[i]] );
    }
}

__global__ void init_status_kernel( int * status )
{
    status[0] = 0;
    status[1] = INT_MAX;
    status[2] = 0;
}

// Launch with programmatic stream serialization (see pdl_allow_next).
template<typename... KArgs, typename... Args>
void launch( bool programmatic, void (*kernel)( KArgs... ), unsigned grid, unsigned block, size_t smem, cudaStream_t st, Args... args )
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3( grid );
    cfg.blockDim = dim3( block );
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    cudaLaunchKernelEx( &cfg, kernel, static_cast<KArgs>( args )... );
}

template<typename... KArgs, typename... Args>
void launch_pdl( void (*kernel)( KArgs... ), unsigned grid, unsigned block, size_t smem, cudaStream_t st, Args... args )
{
    launch( true, kernel, grid, block, smem, st, args... );
}

int grid_for( std::int64_t work, int threads )
{
    const std::int64_t blocks = (work + threads - 1) / threads;
    return static_cast<int>( blocks < 1 ? 1 : (blocks > 148 * 32 ? 148 * 32 : blocks) );
}

// ------------------------------------------------------ super-panel solve
// Large fronts solve 512 pivot rows per step (SuperPanel, plan.hpp): the
// inverse T of the 512 x 512 diagonal block, formed after the factorization
// from the 64-row panel inverses, replaces eight sequential panel steps by
// one product with T.  64 x 64 blocks throughout; warp w owns output rows
// 8w..8w+7 as 8 x 8 DMMA tiles.
// Doubles of shared memory a padded 64 x 64 block of T takes (see super_rest_kernel).
template<typename T> __host__ __device__ constexpr int super_block_doubles() { return sizeof(T) == 4 ? kPanel * (kPanel + 8) / 2 : kPanel * kPld; }

__device__ __forceinline__ int super_block_rows( const SuperPanel & sp, int b ) { return min( kPanel, sp.rows - b * kPanel ); }

// One 64 x 64 block product of a super-panel's inverse (SuperInvTask): part 0
// W_ij = sum_k U_ik T_kj, part 1 T_ij = -sum_k T_ik W_kj, or the copy of panel
// i's inverse.  The sum over k streams through two stages of 32 columns of the
// left and 32 rows of the right blocks.  Doubling needs 14 block products in a
// row where the back substitution by distance from the diagonal needed 35
// (C2: 0.37 ms of launches -> 0.18, timed one by one); diagonal blocks are read
// from the panels' inverses.
constexpr int kInvK = 32;
constexpr int kInvLda = kInvK + 4;                      // (conflict-free DMMA fragments, as kPld)
constexpr int kInvStage = kPanel * kInvLda + kInvK * kPld;
constexpr size_t kSuperInvSmem = sizeof(double) * 2 * kInvStage;

template<typename T>
__global__ __launch_bounds__(256) void super_inv_kernel( const SuperInvTask * __restrict__ tasks, int part, const SuperPanel * __restrict__ sps,
                                                         const T * __restrict__ arena, const double * __restrict__ tinv,
                                                         double * __restrict__ tbuf, int * __restrict__ grown )
{
    extern __shared__ __align__(16) double ism[];
    pdl_allow_next();
    const SuperInvTask task = tasks[blockIdx.x];
    const SuperPanel & sp = sps[task.sp];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i = task.i, j = task.j;
    const int ldt = sp.ldt;
    double * Tb = tbuf + sp.t;
    auto block = [&]( int r, int c ) { return Tb + (std::int64_t)(kPanel * r) * ldt + kPanel * c; };
    auto panel_inverse = [&]( int b ) { return tinv + (std::int64_t)sp.panel[b] * (kPanel * kPanel); };
    const int nbi = super_block_rows( sp, i );
    pdl_wait();
    if( i == j )
    {
        const double * src = panel_inverse( i );
        double * out = block( i, i );
        for( int idx = 2 * tid; idx < kPanel * kPanel; idx += 512 )
        {
            const int r = idx >> 6, c = idx & 63;
            double2 v = make_double2( 0.0, 0.0 );
            if( r < nbi && c < nbi )
            {
                v.x = src[idx];
                if( c + 1 < nbi ) { v.y = src[idx + 1]; }
            }
            *reinterpret_cast<double2 *>( out + (std::int64_t)r * ldt + c ) = v;
        }
        if( sp.guard )
        {
            // a column's entries of U over its diagonal entry, squared and summed over the block's rows
            // so far, four threads a column
            const int c = tid & 63;
            const int diag = kPanel * i + min( c, nbi - 1 );
            const T * U = arena + sp.u0 + (std::int64_t)sp.r0 * sp.ld0 + sp.r0 + diag;
            const double inv = 1.0 / static_cast<double>( U[(std::int64_t)diag * sp.ld0] );
            double sum = 0.0;
#pragma unroll 16
            for( int r = tid >> 6; r <= diag; r += 4 )
            {
                const double q = static_cast<double>( U[(std::int64_t)r * sp.ld0] ) * inv;
                sum = fma( q, q, sum );
            }
            ism[tid] = sum;
            __syncthreads();
            if( tid < kPanel ) { sum = (ism[tid] + ism[tid + 64]) + (ism[tid + 128] + ism[tid + 192]); }
            const int above = __syncthreads_or( tid < kPanel && !(sum <= kGuardGrowth) );
            if( tid == 0 ) { grown[kGuardBlocks * task.sp + i] = above; }
        }
        return;
    }
    const int k0 = part == 0 ? task.mid : i, k1 = part == 0 ? j + 1 : task.mid;      // blocks of the sum
    const int steps = (k1 - k0) * (kPanel / kInvK);
    constexpr int kV = 16 / static_cast<int>( sizeof(T) );
    [[maybe_unused]] float4 uf[2];
    // stage st <- step q: columns [c0, c0 + 32) of the left block (i, k), rows [c0, c0 + 32) of the right one
    auto load = [&]( int q )
    {
        const int k = k0 + q / (kPanel / kInvK), c0 = (q % (kPanel / kInvK)) * kInvK;
        double * As = ism + (q & 1) * kInvStage;
        double * Bs = As + kPanel * kInvLda;
        const int nbk = super_block_rows( sp, k );
        if( part == 0 )
        {
            const T * U = arena + sp.u0 + (std::int64_t)(sp.r0 + kPanel * i) * sp.ld0 + sp.r0 + kPanel * k + c0;
#pragma unroll
            for( int u = 0; u < kPanel * kInvK / kV / 256; ++u )
            {
                const int idx = kV * (tid + 256 * u), r = idx / kInvK, c = idx % kInvK;
                const int left = r < nbi ? nbk - c0 - c : 0;                          // valid columns from c on
                if constexpr ( sizeof(T) == 8 ) { cp_async_16( As + r * kInvLda + c, left > 0 ? U + (std::int64_t)r * sp.ld0 + c : U, left > 1 ? 16 : left > 0 ? 8 : 0 ); }
                else
                {
                    uf[u] = left > 0 ? *reinterpret_cast<const float4 *>( U + (std::int64_t)r * sp.ld0 + c ) : make_float4( 0.f, 0.f, 0.f, 0.f );
                    if( left < 4 ) { uf[u].w = 0.f; if( left < 3 ) { uf[u].z = 0.f; } if( left < 2 ) { uf[u].y = 0.f; } }
                }
            }
        }
        else
        {
            const bool diag = k == i;
            const double * A = diag ? panel_inverse( i ) + c0 : block( i, k ) + c0;
            const int lda = diag ? kPanel : ldt;
#pragma unroll
            for( int u = 0; u < kPanel * kInvK / 512; ++u )
            {
                const int idx = 2 * (tid + 256 * u), r = idx / kInvK, c = idx % kInvK;
                const int left = diag ? (r < nbi ? nbi - c0 - c : 0) : 2;
                cp_async_16( As + r * kInvLda + c, left > 0 ? A + (std::int64_t)r * lda + c : A, left > 1 ? 16 : left > 0 ? 8 : 0 );
            }
        }
        {
            const bool diag = part == 0 && k == j;
            const double * B = (diag ? panel_inverse( j ) : part == 0 ? block( k, j ) : block( j, k )) + (std::int64_t)c0 * (diag ? kPanel : ldt);
            const int ldb = diag ? kPanel : ldt;
#pragma unroll
            for( int u = 0; u < kPanel * kInvK / 512; ++u )
            {
                const int idx = 2 * (tid + 256 * u), r = idx / kPanel, c = idx % kPanel;
                const int left = diag ? (c0 + r < nbk ? nbk - c : 0) : 2;
                cp_async_16( Bs + r * kPld + c, left > 0 ? B + (std::int64_t)r * ldb + c : B, left > 1 ? 16 : left > 0 ? 8 : 0 );
            }
        }
        cp_async_commit();
    };
    // FP32 storage: the left block's values, loaded a step ahead, widened into their stage
    auto widen = [&]( int q )
    {
        if constexpr ( sizeof(T) == 4 )
        {
            if( part != 0 ) { return; }
            double * As = ism + (q & 1) * kInvStage;
#pragma unroll
            for( int u = 0; u < 2; ++u )
            {
                const int idx = 4 * (tid + 256 * u), r = idx / kInvK, c = idx % kInvK;
                *reinterpret_cast<double2 *>( As + r * kInvLda + c ) = make_double2( uf[u].x, uf[u].y );
                *reinterpret_cast<double2 *>( As + r * kInvLda + c + 2 ) = make_double2( uf[u].z, uf[u].w );
            }
        }
    };
    double acc[8][2];
#pragma unroll
    for( int ct = 0; ct < 8; ++ct ) { acc[ct][0] = 0.0; acc[ct][1] = 0.0; }
    load( 0 );
    widen( 0 );
    for( int q = 0; q < steps; ++q )
    {
        cp_async_wait<0>();
        __syncthreads();                                 // stage q complete; the other stage is free
        if( q + 1 < steps ) { load( q + 1 ); }
        const double * As = ism + (q & 1) * kInvStage + (8 * warp + (lane >> 2)) * kInvLda + (lane & 3);
        const double * Bs = ism + (q & 1) * kInvStage + kPanel * kInvLda + (lane & 3) * kPld + (lane >> 2);
#pragma unroll
        for( int kk = 0; kk < kInvK; kk += 4 )
        {
            const double a = As[kk];
#pragma unroll
            for( int ct = 0; ct < 8; ++ct ) { dmma_8x8x4( acc[ct], a, Bs[kk * kPld + 8 * ct] ); }
        }
        if( q + 1 < steps ) { widen( q + 1 ); }
    }
    double * out = part == 0 ? block( j, i ) : block( i, j );
    const double sign = part == 0 ? 1.0 : -1.0;
#pragma unroll
    for( int ct = 0; ct < 8; ++ct )
    {
        *reinterpret_cast<double2 *>( out + (std::int64_t)(8 * warp + (lane >> 2)) * ldt + 8 * ct + 2 * (lane & 3) )
            = make_double2( sign * acc[ct][0], sign * acc[ct][1] );
    }
}

// The diag step of a guarded super-panel whose inverse is not used (kGuardGrowth), panel by panel in
// one CTA: forward x_q = T_q^T (y_q - sum_{p<q} U_pq^T x_p), back x_q = T_q (y_q + z_q - sum_{p>q} U_qp x_p),
// with the panels' own inverses T_q and the x_p read back from `out`.  Rare: plain loads.
template<typename T, int KP>
__device__ __noinline__ void super_diag_panels( const SuperPanel & sp, const T * __restrict__ arena, const double * __restrict__ tinv, int upper,
                                                const double * in, const double * zbuf, double * out, int ld, int k, double * dsm )
{
    constexpr int nct = KP / 8;
    constexpr int ldv = KP + 4;
    double (*B)[kPld] = reinterpret_cast<double (*)[kPld]>( dsm );
    double * V = dsm + kPanel * kPld;                  // [64][ldv]
    double * X = V + kPanel * ldv;                     // [64][ldv]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nblk = (sp.rows + kPanel - 1) / kPanel;
    const std::int64_t brow = (std::int64_t)sp.row0 + sp.r0;
    const T * U = arena + sp.u0 + (std::int64_t)sp.r0 * sp.ld0 + sp.r0;
    // this warp's rows of B^T S (forward) or B S (back)
    auto product = [&]( double (&acc)[nct][2], const double * S )
    {
#pragma unroll
        for( int ct = 0; ct < nct; ++ct ) { acc[ct][0] = 0.0; acc[ct][1] = 0.0; }
        for( int kb = 0; kb < kSubs; ++kb )
        {
#pragma unroll
            for( int ct = 0; ct < nct; ++ct )
            {
                if( upper ) { dmma_8x8x8( acc[ct], [&]( int i, int kk ) { return B[8 * warp + i][8 * kb + kk]; },
                                                   [&]( int kk, int j ) { return S[(8 * kb + kk) * ldv + 8 * ct + j]; } ); }
                else        { dmma_8x8x8( acc[ct], [&]( int i, int kk ) { return B[8 * kb + kk][8 * warp + i]; },
                                                   [&]( int kk, int j ) { return S[(8 * kb + kk) * ldv + 8 * ct + j]; } ); }
            }
        }
    };
    double acc[nct][2];
    for( int s = 0; s < nblk; ++s )
    {
        const int q = upper ? nblk - 1 - s : s;
        const int nbq = super_block_rows( sp, q );
        const std::int64_t qrow = brow + kPanel * q;
        for( int idx = tid; idx < kPanel * KP; idx += 256 )
        {
            const int r = idx / KP, c = idx % KP;
            double v = 0.0;
            if( r < nbq && c < k ) { v = in[(qrow + r) * ld + c] + (upper ? zbuf[(qrow + r) * ld + c] : 0.0); }
            V[r * ldv + c] = v;
        }
        for( int e = 0; e < s; ++e )
        {
            const int p = upper ? nblk - 1 - e : e, a = min( p, q ), b = max( p, q );
            const int nba = super_block_rows( sp, a ), nbb = super_block_rows( sp, b ), nbp = super_block_rows( sp, p );
            for( int idx = tid; idx < kPanel * kPanel; idx += 256 )
            {
                const int r = idx >> 6, c = idx & 63;
                B[r][c] = r < nba && c < nbb ? static_cast<double>( U[(std::int64_t)(kPanel * a + r) * sp.ld0 + kPanel * b + c] ) : 0.0;
            }
            for( int idx = tid; idx < kPanel * KP; idx += 256 )
            {
                const int r = idx / KP, c = idx % KP;
                X[r * ldv + c] = r < nbp && c < k ? out[(brow + kPanel * p + r) * ld + c] : 0.0;
            }
            __syncthreads();
            product( acc, X );
            double * v = V + (8 * warp + (lane >> 2)) * ldv + 2 * (lane & 3);
#pragma unroll
            for( int ct = 0; ct < nct; ++ct ) { v[8 * ct] -= acc[ct][0]; v[8 * ct + 1] -= acc[ct][1]; }
            __syncthreads();
        }
        const double * tq = tinv + (std::int64_t)sp.panel[q] * (kPanel * kPanel);
        for( int idx = tid; idx < kPanel * kPanel; idx += 256 )
        {
            const int r = idx >> 6, c = idx & 63;
            B[r][c] = r < nbq && c < nbq ? tq[idx] : 0.0;
        }
        __syncthreads();
        product( acc, V );
        const int r = 8 * warp + (lane >> 2);
        if( r < nbq )
        {
            double * dst = out + (qrow + r) * ld;
#pragma unroll
            for( int ct = 0; ct < nct; ++ct )
            {
                const int c = 8 * ct + 2 * (lane & 3);
                if( c < k ) { dst[c] = acc[ct][0]; }
                if( c + 1 < k ) { dst[c + 1] = acc[ct][1]; }
            }
        }
        __syncthreads();
    }
}

// One block pair of a super-panel's diag step.  Forward (task (o, b), b <= o):
// x_o += T_bo^T y_b; back (b >= o): x_o += T_ob (y_b + z_b).  y: `in`, z: the
// rest steps' sums in `zbuf`, x: `out`, whose block rows are zero before the
// step (the pairs of one block row add into it).  KP = k rounded up to a power
// of two >= 8.  One 64 x 64 block of T and one 64 x k block of vectors per
// CTA, all copies in flight together.  A guarded super-panel that does not use
// its inverse leaves its diag step to the CTA of its first pair.
template<typename T, int KP>
__device__ __forceinline__ void super_diag_body( const SuperSolveTask & task, const SuperPanel * __restrict__ sps,
                                                 const double * __restrict__ tbuf, const int * __restrict__ grown,
                                                 const T * __restrict__ arena, const double * __restrict__ tinv, int upper, const double * in,
                                                 const double * zbuf, double * out, int ld, int k, double * dsm )
{
    const SuperPanel & sp = sps[task.sp];
    if( sp.guard )
    {
        static_assert( kGuardBlocks == 4, "one int4 a super-panel" );
        const int4 g = *reinterpret_cast<const int4 *>( grown + kGuardBlocks * task.sp );
        // (blocks beyond the super-panel's rows are never written)
        if( (g.x | (sp.rows > kPanel ? g.y : 0) | (sp.rows > 2 * kPanel ? g.z : 0) | (sp.rows > 3 * kPanel ? g.w : 0)) != 0 )
        {
            if( task.blk != 0 || task.c0 != 0 ) { return; }
            pdl_wait();
            super_diag_panels<T, KP>( sp, arena, tinv, upper, in, zbuf, out, ld, k, dsm );
            return;
        }
    }
    constexpr int nct = KP / 8;
    constexpr int ldv = KP + 4;
    double (*Tb)[kPld] = reinterpret_cast<double (*)[kPld]>( dsm );
    double * V = dsm + kPanel * kPld;                  // [64][ldv]
    double * Z = V + kPanel * ldv;                     // [64][ldv], back sweep only
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int o = task.blk, b = task.c0;
    const int nbb = super_block_rows( sp, b );
    const std::int64_t brow = (std::int64_t)sp.row0 + sp.r0;
    const int ldt = sp.ldt;
    // forward: block (b, o) of T, read transposed; back: block (o, b).  The
    // blocks are zero outside their valid rows and columns.
    const double * tb = upper ? tbuf + sp.t + (std::int64_t)(kPanel * o) * ldt + kPanel * b
                              : tbuf + sp.t + (std::int64_t)(kPanel * b) * ldt + kPanel * o;
#pragma unroll
    for( int u = 0; u < kPanel * kPanel / 512; ++u )
    {
        const int idx = 2 * (tid + 256 * u);
        cp_async_16( &Tb[idx >> 6][idx & 63], tb + (idx >> 6) * ldt + (idx & 63), 16 );
    }
    pdl_wait();
    auto rows = [&]( int r ) { return brow + kPanel * b + r; };
    stage_rows<KP>( V, in, rows, nbb, ld, k );
    if( upper ) { stage_rows<KP>( Z, zbuf, rows, nbb, ld, k ); }
    cp_async_wait_all();
    if( upper )
    {
        __syncthreads();
        for( int idx = tid; idx < kPanel * KP; idx += 256 ) { V[(idx / KP) * ldv + idx % KP] += Z[(idx / KP) * ldv + idx % KP]; }
    }
    __syncthreads();
    double acc[nct][2];
#pragma unroll
    for( int ct = 0; ct < nct; ++ct ) { acc[ct][0] = 0.0; acc[ct][1] = 0.0; }
    for( int kb = 0; kb < kSubs; ++kb )
    {
#pragma unroll
        for( int ct = 0; ct < nct; ++ct )
        {
            if( upper ) { dmma_8x8x8( acc[ct], [&]( int i, int kk ) { return Tb[8 * warp + i][8 * kb + kk]; },
                                               [&]( int kk, int j ) { return V[(8 * kb + kk) * ldv + 8 * ct + j]; } ); }
            else        { dmma_8x8x8( acc[ct], [&]( int i, int kk ) { return Tb[8 * kb + kk][8 * warp + i]; },
                                               [&]( int kk, int j ) { return V[(8 * kb + kk) * ldv + 8 * ct + j]; } ); }
        }
    }
    const int nbo = super_block_rows( sp, o );
    const int r = 8 * warp + (lane >> 2);
    if( r < nbo )
    {
        double * dst = out + (brow + kPanel * o + r) * ld;
#pragma unroll
        for( int ct = 0; ct < nct; ++ct )
        {
            const int c = 8 * ct + 2 * (lane & 3);
            if( c < k ) { red_add_f64( dst + c, acc[ct][0] ); }
            if( c + 1 < k ) { red_add_f64( dst + c + 1, acc[ct][1] ); }
        }
    }
}

// A diag step and, in the level's first one, the level's panel steps beside it
// (its one-panel fronts; the two touch different fronts' rows, ancestor rows by
// reductions): one launch less on the level's chain.  With the 16-byte copies
// and padded rows of this and the rest step: C2 with 16 right-hand sides 1.56
// -> 1.22 ms, 56^3 with 64 2.93 -> 2.01 ms.
template<typename T, int KP>
__global__ __launch_bounds__(256) void super_diag_kernel( const SuperSolveTask * __restrict__ tasks, int ndiag,
                                                          const SolveRestTask * __restrict__ steps, const SuperPanel * __restrict__ sps,
                                                          const double * __restrict__ tbuf, const int * __restrict__ grown,
                                                          const T * __restrict__ arena,
                                                          const double * __restrict__ tinv, const std::int32_t * __restrict__ sn_inner,
                                                          int upper, double * in, const double * zbuf, double * out, int ld, int k )
{
    extern __shared__ __align__(16) double dsm[];
    pdl_allow_next();
    if( static_cast<int>( blockIdx.x ) < ndiag )
    {
        super_diag_body<T, KP>( tasks[blockIdx.x], sps, tbuf, grown, arena, tinv, upper, in, zbuf, out, ld, k, dsm );
    }
    else
    {
        solve_step_body<T, KP, true>( steps[blockIdx.x - ndiag], upper, arena, tinv, sn_inner, in, out, ld, k, false, dsm );
    }
}

// One (block, rest chunk) pair of a super-panel's rest step, rest columns
// [c0, c1) of block b.  Forward: y_rest -= U_{b,rest}^T x_b (x_b: `out`, final
// after the diag step; y: `in`, every row by reductions, as the eight blocks
// add into the same rows).  Back: z_b -= U_{b,rest} x_rest (x_rest: `out`,
// final; z: reductions into `zbuf`).
template<typename T, int KP>
__global__ __launch_bounds__(256) void super_rest_kernel( const SuperSolveTask * __restrict__ tasks, const SuperPanel * __restrict__ sps,
                                                          const T * __restrict__ arena, const std::int32_t * __restrict__ sn_inner,
                                                          int upper, double * in, double * zbuf, const double * out, int ld, int k )
{
    extern __shared__ __align__(16) double rsm[];
    pdl_allow_next();
    const SuperSolveTask task = tasks[blockIdx.x];
    const SuperPanel sp = sps[task.sp];
    constexpr int nct = KP / 8;
    constexpr int ldv = KP + 4;
    __shared__ std::int64_t trow[kSolveRest];
    // the factor block in the factor's type (FP32 storage: half the shared memory), widened as read;
    // leading dimensions without bank conflicts in the fragment reads (FP32: 68 by rows, 72 by columns)
    T * Ps = reinterpret_cast<T *>( rsm );
    const int ldp = sizeof(T) == 4 && !upper ? kPanel + 8 : kPld;
    double * V = rsm + super_block_doubles<T>();        // [64][ldv]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r1 = sp.r0 + sp.rows;
    const int m = sp.n0 - r1;
    const int cw = task.c1 - task.c0;
    const int b = task.blk;
    const int nbb = super_block_rows( sp, b );
    const std::int64_t brow = (std::int64_t)sp.row0 + sp.r0;
    if( tid < kSolveRest )
    {
        const int col = task.c0 + tid;
        trow[tid] = (tid < cw) ? ((col < m) ? (std::int64_t)sp.row0 + r1 + col : (std::int64_t)sn_inner[sp.inner + (col - m)]) : -1;
    }
    // P: rows of block b (U rows r0 + 64 b + rr), the chunk's rest columns
    const T * U0 = arena + sp.u0;
    const T * U1 = arena + sp.u1;
    // (a chunk lies in U0 or in U1 alone, both 16-byte aligned there)
    constexpr int kV = 16 / static_cast<int>( sizeof(T) );
    const T * src0 = task.c0 < m ? U0 + (std::int64_t)(sp.r0 + kPanel * b) * sp.ld0 + r1 + task.c0
                                 : U1 + (std::int64_t)(sp.r0 + kPanel * b) * sp.ld1 + (task.c0 - m);
    const int lds = task.c0 < m ? sp.ld0 : sp.ld1;
#pragma unroll
    for( int u = 0; u < kPanel * kPanel / kV / 256; ++u )
    {
        const int idx = kV * (tid + 256 * u), rr = idx >> 6, jj = idx & 63;
        const int left = rr < nbb ? min( cw - jj, kV ) : 0;
        cp_async_16( Ps + rr * ldp + jj, left > 0 ? src0 + (std::int64_t)rr * lds + jj : src0, left > 0 ? left * static_cast<int>( sizeof(T) ) : 0 );
    }
    pdl_wait();
    __syncthreads();                                    // trow
    // x_rest: the chunk's rows of `out`; x_b
    if( upper ) { stage_rows<KP>( V, out, [&]( int r ) { return trow[r]; }, cw, ld, k ); }
    else { stage_rows<KP>( V, out, [&]( int r ) { return brow + kPanel * b + r; }, nbb, ld, k ); }
    cp_async_wait_all();
    __syncthreads();
    double acc[nct][2];
#pragma unroll
    for( int ct = 0; ct < nct; ++ct ) { acc[ct][0] = 0.0; acc[ct][1] = 0.0; }
    for( int kb = 0; kb < kSubs; ++kb )
    {
#pragma unroll
        for( int ct = 0; ct < nct; ++ct )
        {
            // forward: acc(jj, c) = sum_rr P[rr][jj] x_b[rr][c]; back: acc(rr, c) = sum_jj P[rr][jj] x_rest[jj][c]
            if( upper ) { dmma_8x8x8( acc[ct], [&]( int i, int kk ) { return static_cast<double>( Ps[(8 * warp + i) * ldp + 8 * kb + kk] ); },
                                               [&]( int kk, int j ) { return V[(8 * kb + kk) * ldv + 8 * ct + j]; } ); }
            else        { dmma_8x8x8( acc[ct], [&]( int i, int kk ) { return static_cast<double>( Ps[(8 * kb + kk) * ldp + 8 * warp + i] ); },
                                               [&]( int kk, int j ) { return V[(8 * kb + kk) * ldv + 8 * ct + j]; } ); }
        }
    }
    const int r = 8 * warp + (lane >> 2);
    if( upper ? r < nbb : r < cw )
    {
        double * row = upper ? zbuf + (brow + kPanel * b + r) * ld : in + trow[r] * ld;
#pragma unroll
        for( int ct = 0; ct < nct; ++ct )
        {
            const int c = 8 * ct + 2 * (lane & 3);
            if( c < k ) { red_add_f64( row + c, -acc[ct][0] ); }
            if( c + 1 < k ) { red_add_f64( row + c + 1, -acc[ct][1] ); }
        }
    }
}

} // namespace

template<typename T>
void launch_assemble( const double * values, const std::int64_t * src, const std::int64_t * dst,
                      std::int64_t count, const double * reg, T * arena, cudaStream_t st )
{
    if( count <= 0 ) { return; }
    assemble_kernel<<<grid_for( count, 256 ), 256, 0, st>>>( values, src, dst, count, reg, arena );
}

template<typename T>
void launch_zero( const ZeroTask * tasks, int count, T * arena, cudaStream_t st )
{
    if( count > 0 ) { launch_pdl( zero_kernel<T>, count, 256, 0, st, tasks, arena ); }
}

template<typename T>
void launch_export( const ExportTask * tasks, int count, const std::int32_t * colmap, const T * arena,
                    double * tri, double * rec, cudaStream_t st )
{
    if( count > 0 ) { export_kernel<<<count, 128, 0, st>>>( tasks, colmap, arena, tri, rec ); }
}

template<typename T>
void launch_extend( const ExtendTask * tasks, int count, const std::int32_t * lut, T * arena, cudaStream_t st )
{
    if( count > 0 ) { launch_pdl( extend_kernel<T>, count, 256, 0, st, tasks, lut, arena ); }
}

template<typename T>
void launch_extend_pull( const ExtendPullTask * tasks, int count, const ExtendTask * segs, const std::int32_t * lut, T * arena,
                         cudaStream_t st )
{
    if( count > 0 ) { launch_pdl( extend_pull_kernel<T>, count, 256, 0, st, tasks, segs, lut, arena ); }
}

void launch_fronts( const FrontTask * tasks, int count, int threads, int smem, const ExtendTask * segs, const std::int32_t * lut, double * arena,
                    int * status, double * tinv, cudaStream_t st )
{
    if( count <= 0 ) { return; }
    switch( threads )
    {
        case 128: launch_pdl( front_kernel<128>, count, 128, smem, st, tasks, segs, lut, arena, status, tinv ); break;
        case 256: launch_pdl( front_kernel<256>, count, 256, smem, st, tasks, segs, lut, arena, status, tinv ); break;
        default:  launch_pdl( front_kernel<384>, count, 384, smem, st, tasks, segs, lut, arena, status, tinv ); break;
    }
}

template<typename T>
void launch_potrf( const PanelTask * tasks, int count, T * arena, int * status, const double * pivot_floor, double * tinv,
                   cudaStream_t st, bool pending )
{
    if constexpr ( sizeof(T) == 8 )
    {
        if( count > 0 && pending ) { launch_pdl( potrf_kernel<T, true>, count, kPotrfThreads, kPotrfSmemBytes, st, tasks, arena, status, pivot_floor, tinv ); return; }
    }
    if( count > 0 ) { launch_pdl( potrf_kernel<T, false>, count, kPotrfThreads, kPotrfSmemBytes, st, tasks, arena, status, pivot_floor, tinv ); }
}

// floor[i] = rel * |diagonal entry of row i| after assembly (FP32 storage).
// out[1 + i] = rel * |a_ii|; out[0] = max_i |a_ii| (cleared by the caller),
// by an integer maximum over the bit patterns of non-negative doubles.
__global__ void pivot_floor_kernel( const std::int64_t * __restrict__ offsets, const float * __restrict__ arena, double rel,
                                    double * __restrict__ out, int n )
{
    unsigned long long mx = 0ull;
    for( std::int64_t i = blockIdx.x * (std::int64_t)blockDim.x + threadIdx.x; i < n; i += (std::int64_t)gridDim.x * blockDim.x )
    {
        const double a = fabs( static_cast<double>( arena[offsets[i]] ) );
        out[1 + i] = rel * a;
        const unsigned long long bits = static_cast<unsigned long long>( __double_as_longlong( a ) );
        mx = bits > mx ? bits : mx;
    }
#pragma unroll
    for( int o = 16; o > 0; o >>= 1 )
    {
        const unsigned long long v = __shfl_xor_sync( 0xffffffffu, mx, o );
        mx = v > mx ? v : mx;
    }
    if( (threadIdx.x & 31) == 0 && mx != 0ull ) { atomicMax( reinterpret_cast<unsigned long long *>( out ), mx ); }
}

void launch_pivot_floor( const std::int64_t * offsets, const float * arena, double rel, double * out, int n, cudaStream_t st )
{
    cudaMemsetAsync( out, 0, sizeof(double), st );
    pivot_floor_kernel<<<grid_for( n, 256 ), 256, 0, st>>>( offsets, arena, rel, out, n );
}

template<typename T>
void launch_trsm( const PanelTask * tasks, int count, T * arena, const double * tinv, cudaStream_t st, float * img, bool after_potrf )
{
    if( count <= 0 ) { return; }
    if( after_potrf ) { launch_pdl( trsm_kernel<T, true>, count, kTrsmThreads, kTrsmSmemBytes, st, tasks, arena, tinv, img ); }
    else { launch_pdl( trsm_kernel<T, false>, count, kTrsmThreads, kTrsmSmemBytes, st, tasks, arena, tinv, img ); }
}

template<typename T>
void launch_gemm( const GemmTask * tasks, int count, T * arena, int * status, cudaStream_t st, bool programmatic )
{
    if( count <= 0 ) { return; }
    if constexpr ( sizeof(T) == 8 )
    {
        (void)status;
        launch( programmatic, gemm_tn_kernel, count, kGemmThreads, kGemmSmemBytes, st, tasks, arena );
    }
    else
    {
        int dev = 0, sms = 0;
        cudaGetDevice( &dev );
        cudaDeviceGetAttribute( &sms, cudaDevAttrMultiProcessorCount, dev );
        const int grid = std::min( count, 3 * std::max( sms, 1 ) );
        launch( programmatic, gemm_tc_kernel, grid, kGemmThreads, kGemmSmemBytesF, st, tasks, count, arena, status );
    }
}

template<typename T>
void launch_factor_dag( const DagArgs & args, int grid, cudaStream_t st )
{
    if( args.ntasks > 0 && grid > 0 ) { factor_dag_kernel<T><<<grid, kDagThreads, kDagSmemBytes, st>>>( args ); }
}

// The occupancy query answers 1 for the FP32 instance, which allocates tensor
// memory, although 3 such CTAs (64 KB of shared memory and 64 TMEM columns
// each) were measured co-resident on one SM; both instances have the same
// shared memory and launch bounds, so the FP64 instance's answer is used for
// both.  Correctness does not depend on residency: tasks are taken by running
// CTAs in a topological order.
int factor_dag_blocks_per_sm()
{
    int b = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor( &b, factor_dag_kernel<double>, kDagThreads, kDagSmemBytes );
    return e == cudaSuccess ? b : 0;
}


static int solve_lkp( int k )
{
    int l = 3;
    while( (1 << l) < k ) { ++l; }
    return l;
}

template<typename T>
static size_t solve_smem_bytes( int k )
{
    return sizeof(double) * (kPanel * kTld + 2 * kPanel * ((1 << solve_lkp( k )) + 4));
}

template<typename T>
void launch_solve_dag( const SolveDagArgs & args, int grid, const T * arena, double * in, double * out, int ld, int k,
                       cudaStream_t st )
{
    if( args.ntasks <= 0 || grid <= 0 ) { return; }
    const size_t sm = solve_smem_bytes<T>( k );
    switch( solve_lkp( k ) )
    {
        case 3:  solve_dag_kernel<T, 8><<<grid, kSolveThreads, sm, st>>>( args, arena, in, out, ld, k ); break;
        case 4:  solve_dag_kernel<T, 16><<<grid, kSolveThreads, sm, st>>>( args, arena, in, out, ld, k ); break;
        case 5:  solve_dag_kernel<T, 32><<<grid, kSolveThreads, sm, st>>>( args, arena, in, out, ld, k ); break;
        default: solve_dag_kernel<T, 64><<<grid, kSolveThreads, sm, st>>>( args, arena, in, out, ld, k ); break;
    }
}

template<typename T>
int solve_dag_occupancy( int k )
{
    const size_t sm = solve_smem_bytes<T>( k );
    int n = 0;
    cudaError_t e = cudaSuccess;
    switch( solve_lkp( k ) )
    {
        case 3:  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor( &n, solve_dag_kernel<T, 8>, kSolveThreads, sm ); break;
        case 4:  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor( &n, solve_dag_kernel<T, 16>, kSolveThreads, sm ); break;
        case 5:  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor( &n, solve_dag_kernel<T, 32>, kSolveThreads, sm ); break;
        default: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor( &n, solve_dag_kernel<T, 64>, kSolveThreads, sm ); break;
    }
    return e == cudaSuccess ? n : 0;
}

int solve_dag_blocks_per_sm( int k )
{
    return std::min( solve_dag_occupancy<double>( k ), solve_dag_occupancy<float>( k ) );
}

template<typename T>
void launch_solve_step( const SolveRestTask * tasks, int count, int small_count, bool upper, const T * arena, const double * tinv,
                        const std::int32_t * sn_inner, double * in, double * out, int ld, int k, cudaStream_t st )
{
    if( count <= 0 ) { return; }
    const size_t sm = small_count < count ? solve_smem_bytes<T>( k ) : 0;
    constexpr int kWarps = kSolveThreads / 32;
    const int u = upper ? 1 : 0, ctas = count - small_count, grid = ctas + (small_count + kWarps - 1) / kWarps;
    switch( solve_lkp( k ) )
    {
        case 3:  launch_pdl( solve_step_kernel<T, 8>, grid, kSolveThreads, sm, st, tasks, ctas, count, u, arena, tinv, sn_inner, in, out, ld, k ); break;
        case 4:  launch_pdl( solve_step_kernel<T, 16>, grid, kSolveThreads, sm, st, tasks, ctas, count, u, arena, tinv, sn_inner, in, out, ld, k ); break;
        case 5:  launch_pdl( solve_step_kernel<T, 32>, grid, kSolveThreads, sm, st, tasks, ctas, count, u, arena, tinv, sn_inner, in, out, ld, k ); break;
        default: launch_pdl( solve_step_kernel<T, 64>, grid, kSolveThreads, sm, st, tasks, ctas, count, u, arena, tinv, sn_inner, in, out, ld, k ); break;
    }
}

template<typename T>
void launch_super_inv( const SuperInvTask * tasks, int count, int part, const SuperPanel * sps, const T * arena, const double * tinv,
                       double * tbuf, int * grown, cudaStream_t st )
{
    if( count > 0 ) { launch_pdl( super_inv_kernel<T>, count, 256, kSuperInvSmem, st, tasks, part, sps, arena, tinv, tbuf, grown ); }
}

template<typename T>
static size_t super_diag_smem( int k )
{
    return std::max( solve_smem_bytes<T>( k ), sizeof(double) * (kPanel * kPld + 2 * kPanel * ((1 << solve_lkp( k )) + 4)) );
}

template<typename T>
static size_t super_rest_smem( int k )
{
    return sizeof(double) * (super_block_doubles<T>() + kPanel * ((1 << solve_lkp( k )) + 4));
}

template<typename T>
void launch_super_diag( const SuperSolveTask * tasks, int count, const SolveRestTask * steps, int nsteps, const SuperPanel * sps,
                        const double * tbuf, const int * grown, const T * arena, const double * tinv, const std::int32_t * sn_inner,
                        bool upper, double * in, const double * zbuf, double * out, int ld, int k, cudaStream_t st )
{
    if( count + nsteps <= 0 ) { return; }
    const size_t sm = super_diag_smem<T>( k );
    const int u = upper ? 1 : 0, n = count + nsteps;
    switch( solve_lkp( k ) )
    {
        case 3:  launch_pdl( super_diag_kernel<T, 8>, n, 256, sm, st, tasks, count, steps, sps, tbuf, grown, arena, tinv, sn_inner, u, in, zbuf, out, ld, k ); break;
        case 4:  launch_pdl( super_diag_kernel<T, 16>, n, 256, sm, st, tasks, count, steps, sps, tbuf, grown, arena, tinv, sn_inner, u, in, zbuf, out, ld, k ); break;
        case 5:  launch_pdl( super_diag_kernel<T, 32>, n, 256, sm, st, tasks, count, steps, sps, tbuf, grown, arena, tinv, sn_inner, u, in, zbuf, out, ld, k ); break;
        default: launch_pdl( super_diag_kernel<T, 64>, n, 256, sm, st, tasks, count, steps, sps, tbuf, grown, arena, tinv, sn_inner, u, in, zbuf, out, ld, k ); break;
    }
}

template<typename T>
void launch_super_rest( const SuperSolveTask * tasks, int count, const SuperPanel * sps, const T * arena,
                        const std::int32_t * sn_inner, bool upper, double * in, double * zbuf, const double * out, int ld, int k,
                        cudaStream_t st )
{
    if( count <= 0 ) { return; }
    const size_t sm = super_rest_smem<T>( k );
    const int u = upper ? 1 : 0;
    switch( solve_lkp( k ) )
    {
        case 3:  launch_pdl( super_rest_kernel<T, 8>, count, 256, sm, st, tasks, sps, arena, sn_inner, u, in, zbuf, out, ld, k ); break;
        case 4:  launch_pdl( super_rest_kernel<T, 16>, count, 256, sm, st, tasks, sps, arena, sn_inner, u, in, zbuf, out, ld, k ); break;
        case 5:  launch_pdl( super_rest_kernel<T, 32>, count, 256, sm, st, tasks, sps, arena, sn_inner, u, in, zbuf, out, ld, k ); break;
        default: launch_pdl( super_rest_kernel<T, 64>, count, 256, sm, st, tasks, sps, arena, sn_inner, u, in, zbuf, out, ld, k ); break;
    }
}

template<typename T>
void launch_gather_diag( const std::int64_t * offsets, const T * arena, double * out, int n, cudaStream_t st )
{
    gather_diag_kernel<<<grid_for( n, 256 ), 256, 0, st>>>( offsets, arena, out, n );
}

#define TB_INSTANTIATE( T )                                                                                          \
    template void launch_assemble<T>( const double *, const std::int64_t *, const std::int64_t *, std::int64_t,      \
                                      const double *, T *, cudaStream_t );                                         \
    template void launch_zero<T>( const ZeroTask *, int, T *, cudaStream_t );                                        \
    template void launch_export<T>( const ExportTask *, int, const std::int32_t *, const T *, double *, double *,    \
                                    cudaStream_t );                                                                \
    template void launch_extend<T>( const ExtendTask *, int, const std::int32_t *, T *, cudaStream_t );             \
    template void launch_extend_pull<T>( const ExtendPullTask *, int, const ExtendTask *, const std::int32_t *, T *, cudaStream_t ); \
    template void launch_potrf<T>( const PanelTask *, int, T *, int *, const double *, double *, cudaStream_t, bool );     \
    template void launch_trsm<T>( const PanelTask *, int, T *, const double *, cudaStream_t, float *, bool );              \
    template void launch_gemm<T>( const GemmTask *, int, T *, int *, cudaStream_t, bool );                                 \
    template void launch_solve_dag<T>( const SolveDagArgs &, int, const T *, double *, double *, int, int, cudaStream_t );                                        \
    template void launch_factor_dag<T>( const DagArgs &, int, cudaStream_t );                                        \
    template void launch_solve_step<T>( const SolveRestTask *, int, int, bool, const T *, const double *,                \
                                        const std::int32_t *, double *, double *, int, int, cudaStream_t );         \
    template void launch_gather_diag<T>( const std::int64_t *, const T *, double *, int, cudaStream_t );          \
    template void launch_super_inv<T>( const SuperInvTask *, int, int, const SuperPanel *, const T *, const double *,      \
                                       double *, int *, cudaStream_t );                                             \
    template void launch_super_diag<T>( const SuperSolveTask *, int, const SolveRestTask *, int, const SuperPanel *, const double *, const int *, const T *, \
                                        const double *, const std::int32_t *, bool, double *, const double *, double *, int, int, cudaStream_t ); \
    template void launch_super_rest<T>( const SuperSolveTask *, int, const SuperPanel *, const T *,                 \
                                        const std::int32_t *, bool, double *, double *, const double *, int, int,   \
                                        cudaStream_t );
TB_INSTANTIATE( double )
TB_INSTANTIATE( float )
#undef TB_INSTANTIATE

void launch_gather_rows( const double * B, int ldB, const std::int32_t * p, double * W, int ldw,
                         int n, int k, cudaStream_t st, int kw )
{
    kw = std::max( kw, k );
    gather_rows_kernel<<<grid_for( (std::int64_t)n * kw, 256 ), 256, 0, st>>>( B, ldB, p, W, ldw, n, k, kw );
}

void launch_scatter_rows( const double * W, int ldw, const std::int32_t * p_inv, double alpha, double beta,
                          double * Y, int ldY, int n, int k, cudaStream_t st )
{
    scatter_rows_kernel<<<grid_for( (std::int64_t)n * k, 256 ), 256, 0, st>>>( W, ldw, p_inv, alpha, beta, Y, ldY, n, k );
}

template<typename Launch>
static void by_column_width( int k, Launch launch )
{
    if( k <= 1 ) { launch( std::integral_constant<int, 1>{} ); }
    else if( k <= 2 ) { launch( std::integral_constant<int, 2>{} ); }
    else if( k <= 4 ) { launch( std::integral_constant<int, 4>{} ); }
    else if( k <= 8 ) { launch( std::integral_constant<int, 8>{} ); }
    else if( k <= 16 ) { launch( std::integral_constant<int, 16>{} ); }
    else { launch( std::integral_constant<int, 32>{} ); }
}

void launch_residual( int n, const std::int64_t * outer, const std::int32_t * inner, const double * vals,
                      const double * X, const double * B, double * R, int k, cudaStream_t st )
{
    launch_apply_shifted( n, outer, inner, vals, 0.0, X, k, B, k, R, k, k, st );
}

cudaError_t configure_kernels()
{
    const struct { const void * fn; size_t bytes; } attrs[] = {
        { reinterpret_cast<const void *>( front_kernel<128> ), kFrontSmemSmall },
        { reinterpret_cast<const void *>( front_kernel<256> ), kFrontSmemMid },
        { reinterpret_cast<const void *>( front_kernel<384> ), kFrontSmemMax },
        { reinterpret_cast<const void *>( potrf_kernel<double, false> ), kPotrfSmemBytes },
        { reinterpret_cast<const void *>( potrf_kernel<double, true> ), kPotrfSmemBytes },
        { reinterpret_cast<const void *>( potrf_kernel<float, false> ), kPotrfSmemBytes },
        { reinterpret_cast<const void *>( trsm_kernel<double, false> ), kTrsmSmemBytes },
        { reinterpret_cast<const void *>( trsm_kernel<double, true> ), kTrsmSmemBytes },
        { reinterpret_cast<const void *>( trsm_kernel<float, false> ), kTrsmSmemBytes },
        { reinterpret_cast<const void *>( trsm_kernel<float, true> ), kTrsmSmemBytes },
        { reinterpret_cast<const void *>( gemm_tn_kernel ), kGemmSmemBytes },
        { reinterpret_cast<const void *>( gemm_tc_kernel ), kGemmSmemBytesF },
        { reinterpret_cast<const void *>( factor_dag_kernel<double> ), kDagSmemBytes },
        { reinterpret_cast<const void *>( factor_dag_kernel<float> ), kDagSmemBytes },
        { reinterpret_cast<const void *>( solve_step_kernel<double, 8> ), solve_smem_bytes<double>( 8 ) },
        { reinterpret_cast<const void *>( solve_step_kernel<double, 16> ), solve_smem_bytes<double>( 16 ) },
        { reinterpret_cast<const void *>( solve_step_kernel<double, 32> ), solve_smem_bytes<double>( 32 ) },
        { reinterpret_cast<const void *>( solve_step_kernel<double, 64> ), solve_smem_bytes<double>( 64 ) },
        { reinterpret_cast<const void *>( solve_step_kernel<float, 8> ), solve_smem_bytes<float>( 8 ) },
        { reinterpret_cast<const void *>( solve_step_kernel<float, 16> ), solve_smem_bytes<float>( 16 ) },
        { reinterpret_cast<const void *>( solve_step_kernel<float, 32> ), solve_smem_bytes<float>( 32 ) },
        { reinterpret_cast<const void *>( solve_step_kernel<float, 64> ), solve_smem_bytes<float>( 64 ) },
        { reinterpret_cast<const void *>( solve_dag_kernel<double, 8> ), solve_smem_bytes<double>( 8 ) },
        { reinterpret_cast<const void *>( solve_dag_kernel<double, 16> ), solve_smem_bytes<double>( 16 ) },
        { reinterpret_cast<const void *>( solve_dag_kernel<double, 32> ), solve_smem_bytes<double>( 32 ) },
        { reinterpret_cast<const void *>( solve_dag_kernel<double, 64> ), solve_smem_bytes<double>( 64 ) },
        { reinterpret_cast<const void *>( solve_dag_kernel<float, 8> ), solve_smem_bytes<float>( 8 ) },
        { reinterpret_cast<const void *>( solve_dag_kernel<float, 16> ), solve_smem_bytes<float>( 16 ) },
        { reinterpret_cast<const void *>( solve_dag_kernel<float, 32> ), solve_smem_bytes<float>( 32 ) },
        { reinterpret_cast<const void *>( solve_dag_kernel<float, 64> ), solve_smem_bytes<float>( 64 ) },
        { reinterpret_cast<const void *>( super_inv_kernel<double> ), kSuperInvSmem },
        { reinterpret_cast<const void *>( super_inv_kernel<float> ), kSuperInvSmem },
        { reinterpret_cast<const void *>( super_diag_kernel<double, 8> ), super_diag_smem<double>( 8 ) },
        { reinterpret_cast<const void *>( super_diag_kernel<float, 8> ), super_diag_smem<float>( 8 ) },
        { reinterpret_cast<const void *>( super_diag_kernel<double, 16> ), super_diag_smem<double>( 16 ) },
        { reinterpret_cast<const void *>( super_diag_kernel<float, 16> ), super_diag_smem<float>( 16 ) },
        { reinterpret_cast<const void *>( super_diag_kernel<double, 32> ), super_diag_smem<double>( 32 ) },
        { reinterpret_cast<const void *>( super_diag_kernel<float, 32> ), super_diag_smem<float>( 32 ) },
        { reinterpret_cast<const void *>( super_diag_kernel<double, 64> ), super_diag_smem<double>( 64 ) },
        { reinterpret_cast<const void *>( super_diag_kernel<float, 64> ), super_diag_smem<float>( 64 ) },
        { reinterpret_cast<const void *>( super_rest_kernel<double, 8> ), super_rest_smem<double>( 8 ) },
        { reinterpret_cast<const void *>( super_rest_kernel<double, 16> ), super_rest_smem<double>( 16 ) },
        { reinterpret_cast<const void *>( super_rest_kernel<double, 32> ), super_rest_smem<double>( 32 ) },
        { reinterpret_cast<const void *>( super_rest_kernel<double, 64> ), super_rest_smem<double>( 64 ) },
        { reinterpret_cast<const void *>( super_rest_kernel<float, 8> ), super_rest_smem<float>( 8 ) },
        { reinterpret_cast<const void *>( super_rest_kernel<float, 16> ), super_rest_smem<float>( 16 ) },
        { reinterpret_cast<const void *>( super_rest_kernel<float, 32> ), super_rest_smem<float>( 32 ) },
        { reinterpret_cast<const void *>( super_rest_kernel<float, 64> ), super_rest_smem<float>( 64 ) },
    };
    for( const auto & a : attrs )
    {
        const cudaError_t e = cudaFuncSetAttribute( a.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)a.bytes );
        if( e != cudaSuccess ) { return e; }
    }
    return cudaSuccess;
}

void launch_apply_shifted( int n, const std::int64_t * outer, const std::int32_t * inner, const double * vals,
                           double shift, const double * X, int ldx, const double * B, int ldb, double * R, int ldr,
                           int k, cudaStream_t st )
{
    if( n <= 0 ) { return; }
    if( k >= 3 )
    {
        // one warp per 32 / KP rows, up to 32 blocks per SM (measured best on a 3-dof 27-point stencil)
        const int grid = grid_for( (std::int64_t)n * 32, 256 );
        by_column_width( k, [&]( auto kp ) {
            if constexpr ( decltype( kp )::value >= 4 )
            {
                spmv_group_kernel<decltype( kp )::value><<<grid, 256, 0, st>>>( n, outer, inner, vals, shift, X, ldx, B, ldb, R, ldr, k );
            }
        } );
        return;
    }
    const int grid = grid_for( (std::int64_t)n * 32, 256 );
    by_column_width( k, [&]( auto kp ) {
        spmv_rows_kernel<decltype( kp )::value><<<grid, 256, 0, st>>>( n, outer, inner, vals, shift, X, ldx, B, ldb, R, ldr, k );
    } );
}

void launch_column_dots( const double * X, int ldx, const double * Y, int ldy, int n, int k, double * out, cudaStream_t st )
{
    if( n <= 0 ) { return; }
    // two blocks per SM: few atomics per column, every row read once
    const int grid = static_cast<int>( std::min<std::int64_t>( 296, ((std::int64_t)n + 255) / 256 ) );
    by_column_width( k, [&]( auto kp ) {
        column_dots_kernel<decltype( kp )::value><<<grid, 256, 0, st>>>( X, ldx, Y, ldy, n, k, out );
    } );
}

void launch_cg_update_xr( int n, int k, const double * rz, const double * pq, const double * p, const double * q,
                          double * x, double * r, cudaStream_t st )
{
    cg_update_xr_kernel<<<grid_for( (std::int64_t)n * k, 256 ), 256, 0, st>>>( n, k, rz, pq, p, q, x, r );
}

void launch_cg_update_p( int n, int k, const double * rz_new, const double * rz_old, const double * z, double * p,
                         cudaStream_t st )
{
    cg_update_p_kernel<<<grid_for( (std::int64_t)n * k, 256 ), 256, 0, st>>>( n, k, rz_new, rz_old, z, p );
}

void launch_multi_dots( const double * Q, std::int64_t nk, int nq, const double * q, int n, int k, double * out, cudaStream_t st )
{
    if( nq <= 0 ) { return; }
    multi_dots_kernel<<<dim3( static_cast<unsigned>( grid_for( n, 256 ) ), static_cast<unsigned>( nq ) ), 256, 0, st>>>( Q, nk, q, n, k, out );
}

void launch_multi_axpy( const double * Q, std::int64_t nk, int nq, const double * coef, double sign, double * q, int n, int k,
                        cudaStream_t st )
{
    if( nq <= 0 ) { return; }
    multi_axpy_kernel<<<grid_for( (std::int64_t)n * k, 256 ), 256, 0, st>>>( Q, nk, nq, coef, sign, q, n, k );
}

void launch_col_normalize( double * x, int n, int k, const double * sq, cudaStream_t st )
{
    col_normalize_kernel<<<grid_for( (std::int64_t)n * k, 256 ), 256, 0, st>>>( x, n, k, sq );
}

void launch_axpy( std::int64_t n, double a, const double * x, double * y, cudaStream_t st )
{
    axpy_kernel<<<grid_for( n, 256 ), 256, 0, st>>>( n, a, x, y );
}

void launch_combine( int n, int k, double alpha, const double * X, int ldx, double beta, double * Y, int ldy, cudaStream_t st )
{
    combine_kernel<<<grid_for( (std::int64_t)n * k, 256 ), 256, 0, st>>>( n, k, alpha, X, ldx, beta, Y, ldy );
}

// Row-major n x k blocks between the two scalar types (the reference casts
// right-hand sides and solutions on copy, Solve.hpp:20-27).
template<typename S, typename D>
__global__ void convert_rows_kernel( const S * __restrict__ src, int lds, D * __restrict__ dst, int ldd, std::int64_t n, int k )
{
    const std::int64_t total = n * k;
    for( std::int64_t i = blockIdx.x * static_cast<std::int64_t>( blockDim.x ) + threadIdx.x; i < total;
         i += static_cast<std::int64_t>( gridDim.x ) * blockDim.x )
    {
        const std::int64_t r = i / k;
        const int c = static_cast<int>( i - r * k );
        dst[r * ldd + c] = static_cast<D>( src[r * lds + c] );
    }
}

void launch_widen( const float * src, int lds, double * dst, int ldd, std::int64_t n, int k, cudaStream_t st )
{
    if( n * k > 0 ) { convert_rows_kernel<float, double><<<grid_for( std::min<std::int64_t>( n * k, std::int64_t( 1 ) << 24 ), 256 ), 256, 0, st>>>( src, lds, dst, ldd, n, k ); }
}

void launch_narrow( const double * src, int lds, float * dst, int ldd, std::int64_t n, int k, cudaStream_t st )
{
    if( n * k > 0 ) { convert_rows_kernel<double, float><<<grid_for( std::min<std::int64_t>( n * k, std::int64_t( 1 ) << 24 ), 256 ), 256, 0, st>>>( src, lds, dst, ldd, n, k ); }
}

void launch_init_status( int * status, cudaStream_t st )
{
    init_status_kernel<<<1, 1, 0, st>>>( status );
}

} // namespace tb
