// Operators whose wedge matrices separate into a lateral and a radial factor:
// Laplace and VectorLaplace (constant coefficient, 3x2 rule) and the plain
// mass matrix.
//
// With the factored wedge stiffness of laplace.cu, every entry between node
// (m_i, l_i) and node (m_j, l_j) of a wedge (m lateral vertex, l = 0 bottom,
// 1 top) is a sum of K lateral factors times radial ones, and the radial ones
// are the same for every wedge of a layer.  Summing the lateral factors over
// the (up to six) triangles around a lateral point first gives K lateral 7-point
// stencils per point, so a node needs K lateral sums per radial level,
//     s_k(r) = sum over the 7 columns Y of C_k(X, Y) u(Y, r),
// and combines those of the levels r - 1, r, r + 1 with the two layers' radial
// factors: about 50 multiply-adds per node for the Laplacian (480 in the
// wedge-by-wedge form), no atomics and no zero fill, each node written once.
// The first S stencils are summed per level, on the differences to the column
// itself where their rows sum to zero (kDiff); the other D enter only through
// the difference of a layer's two levels and are summed on that difference: the
// rounding error then scales with the differences of u and not with u (level 5,
// a smooth u: 5e-15 against 1e-13 without the differences and 1e-14 for the
// quadrature point by point).
//
// Interior columns (tile blocks): one thread per column marches up a run of
// levels with the column's 7 K stencil values in registers and the sums of the
// level below carried, so neither is read again and no sum crosses a thread.
// Its operands come from shared memory, where the block stages the levels of
// its 8 x 16 columns and their neighbours (odd column stride: the lanes of a
// warp, consecutive columns, hit distinct banks) and from where the results go
// out along r: both sides of global memory see runs of consecutive levels.
// Measured for the level-6 FP64 Laplacian: one thread per node with the
// stencil read for every node 58 us, four levels per thread 56 us (bound by
// instruction issue and the latency of those reads), runs of 22 levels staged
// by whole warps 41 us, runs of 14 staged by half-warps 29 us, and 33 us with the
// sums on differences.  What is left is instruction issue (44 % of the slots).
//
// Columns on the edge of a diamond have copies in other diamonds.  With
// additive communication their sums run over the columns of all copies (each
// diamond contributes its own triangles with its own values) and go to every
// copy: the halo sum without a second pass.  These columns (1/16 of all at
// N = 64) are computed one node per thread over the flat (column, r) index.
#pragma once

#include <cuda_pipeline.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "reduce.cuh"
#include "wedge.cuh"

namespace tn {

constexpr int kStencil        = 7;
constexpr int kLateralThreads = 128;
constexpr int kTileX = 8, kTileY = 16;                        // columns of a tile block
constexpr int kTileCols = ( kTileX + 2 ) * ( kTileY + 2 );    // with their neighbours
constexpr int kMaxRun   = 14; // levels of a run: with the two around them they are the 16 lanes of a half-warp
constexpr int kStride   = ( kMaxRun + 2 ) | 1; // words per staged column

// neighbour columns: the point itself and the six edges of the triangulation
// (wedge 0 = (0,0), (1,0), (0,1); wedge 1 = (1,1), (0,1), (1,0))
__host__ __device__ constexpr int stencil_dx( int i ) { return i == 1 || i == 5 ? 1 : ( i == 2 || i == 6 ? -1 : 0 ); }
__host__ __device__ constexpr int stencil_dy( int i ) { return i == 3 || i == 6 ? 1 : ( i == 4 || i == 5 ? -1 : 0 ); }

__host__ __device__ constexpr int stencil_entry( int dx, int dy )
{
    for ( int i = 0; i < kStencil; ++i )
        if ( stencil_dx( i ) == dx && stencil_dy( i ) == dy )
            return i;
    return -1;
}

// Coupling of a cell's wedge nodes: all (kNeu), CMB-side nodes decoupled
// keeping their diagonal (kBot), SURFACE-side ones likewise (kTop), or the
// diagonal alone (kDiag).  It depends on the cell's radial layer only.
enum : int
{
    kNeu  = 0,
    kBot  = 1,
    kTop  = 2,
    kDiag = 3
};

__device__ __forceinline__ int layer_mode( int r, int N, int first, int inner, int last )
{
    return r == 0 ? first : ( r == N - 1 ? last : inner );
}

template < typename T >
struct LateralParams
{
    int             N, n1;
    size_t          columns;                 // stored columns
    int             run, runs;               // levels per run, runs per column
    int             tiles_x, tiles_y;        // tile blocks per diamond
    unsigned        edge_blocks, edge_nodes; // blocks of edge columns (they come first), nodes they write
    const T*        lat;                     // [7 K][column]
    const T*        rad;                     // [factor][layer]
    const int*      offsets;                 // copies of edge entry e: members[offsets[e] .. offsets[e + 1]); NULL: the
    const int*      members;                 // entries are the members themselves (every column on its own)
    Ptr3< const T > src;
    Ptr3< T >       dst;
    int             add;
    int             mode_first, mode_inner, mode_last; // coupling of the layers, kNeu .. kDiag
};

// What a CG step adds to the apply (lateral_cg.cuh): the operand is the new direction p = r + beta p_old, formed
// while it is read and written to p_new, and <p, A p> is summed over the owned nodes.
struct LateralCG
{
    const double* r;
    const double* p_old;
    double*       p_new;
    double*       state; // tn_pcg_* layout
    double*       partials;
    unsigned int* counter;
};

// a column's sums at one level: of the first S stencils, of the other D on the level's own values (used by the layers
// that do not couple their two levels), and the products of all K self entries
template < typename OP, typename T >
struct LevelSums
{
    T s[OP::S], side[OP::D + 1], self[OP::K];
};

// A layer's contributions to its lower and upper node: OP::layer where both levels are coupled, else each coupled
// side with itself (OP::side_*) and the diagonal (OP::self_*) at the decoupled nodes.
template < typename OP, typename T >
__device__ __forceinline__ void lateral_layer( int mode, const T ( &rad )[OP::R], const LevelSums< OP, T >& b,
                                               const LevelSums< OP, T >& t, const T ( &diff )[OP::D + 1], T& low, T& high )
{
    if ( mode == kNeu )
        OP::layer( rad, b.s, t.s, diff, low, high );
    else
    {
        low  = mode == kTop ? OP::side_low( rad, b.s, b.side ) : OP::self_low( rad, b.self );
        high = mode == kBot ? OP::side_high( rad, t.s, t.side ) : OP::self_high( rad, t.self );
    }
}

// *p = v, or added to *p: as one atomic, so that applies on several streams may add into the same field
template < typename T >
__device__ __forceinline__ void lateral_store( T* p, T v, int add )
{
    if ( add )
        atomicAdd( p, v );
    else
        *p = v;
}

template < typename OP, bool CG, typename T >
__device__ __forceinline__ void lateral_tile( const LateralParams< T >& P, const LateralCG& cg, T beta, unsigned block, T* smem,
                                              Neumaier& dot )
{
    constexpr int  K = OP::K, R = OP::R;
    constexpr bool exact_dot = CG && OP::kExactDot;
    const int     n1 = P.n1, tid = int( threadIdx.x ), lane = tid & 31, warp = tid >> 5;
    const int     chunk = int( block % unsigned( P.runs ) );
    const unsigned tile = block / unsigned( P.runs );
    const int     x0 = int( tile / unsigned( P.tiles_y ) % unsigned( P.tiles_x ) ) * kTileX;
    const int     y0 = int( tile % unsigned( P.tiles_y ) ) * kTileY;
    const int     d  = int( tile / unsigned( P.tiles_x * P.tiles_y ) );
    const int     ra = chunk * P.run, rb = min( ra + P.run, n1 ); // levels [ra, rb) are written
    T*            in  = smem;                       // [column of the tile with neighbours][level ra - 1 ..]
    T*            out = in + kTileCols * kStride;   // [column of the tile][level ra ..]
    T*            rad = out + kTileX * kTileY * kStride;
    const T*      src = P.src.at( blockIdx.y ) + ( ( size_t( d ) * n1 + x0 ) * n1 + y0 ) * n1;
    // a half-warp copies one column's levels; the block's eight take the rows of the tile in turn
    const int hl = lane & 15, half = warp * 2 + ( lane >> 4 ), r = ra - 1 + hl;
    if ( hl < P.run + 2 && r >= 0 && r < n1 )
    {
        const int ymax = min( kTileY + 2, n1 - y0 );
        for ( int x = half; x < min( kTileX + 2, n1 - x0 ); x += kLateralThreads / 16 )
        {
            const T* g = src + size_t( x ) * n1 * n1 + r;
            T*       c = in + x * ( kTileY + 2 ) * kStride + hl;
            if constexpr ( CG )
            {
                const T* q = cg.r + ( g - P.src.p[0] );
#pragma unroll
                for ( int y = 0; y < kTileY + 2; ++y )
                    if ( y < ymax )
                        c[y * kStride] = q[size_t( y ) * n1] + beta * g[size_t( y ) * n1];
            }
            else
            {
#pragma unroll
                for ( int y = 0; y < kTileY + 2; ++y, g += n1 )
                    if ( y < ymax )
                        __pipeline_memcpy_async( c + y * kStride, g, sizeof( T ) );
            }
        }
    }
    for ( int i = tid; i < R * ( P.run + 1 ); i += kLateralThreads )
    {
        const int l = ra - 1 + i / R; // the layer
        rad[i]      = l >= 0 && l < P.N ? P.rad[( i % R ) * P.N + l] : T( 0 );
    }
    // this thread's column, 1 <= x, y <= N - 1, and its stencil
    const int  tx = tid / kTileY, ty = tid % kTileY, x = x0 + 1 + tx, y = y0 + 1 + ty;
    const bool mine = x < P.N && y < P.N;
    T          f[kStencil][K];
#pragma unroll
    for ( int i = 0; i < kStencil; ++i )
#pragma unroll
        for ( int k = 0; k < K; ++k )
            f[i][k] = mine ? P.lat[size_t( i * K + k ) * P.columns + ( size_t( d ) * n1 + x ) * n1 + y] : T( 0 );
    __pipeline_commit();
    __pipeline_wait_prior( 0 );
    __syncthreads();
    if ( mine )
    {
        const T* u = in + ( ( tx + 1 ) * ( kTileY + 2 ) + ty + 1 ) * kStride - ( ra - 1 ); // u[r] = level r
        T*       o = out + tid * kStride - ra;
        T                  high = T( 0 );
        LevelSums< OP, T > b{};
        // sums of level l, which close the layer l - 1 below it (the level below is read again for the difference:
        // held in registers it made them spill, 39 instead of 33 us)
        int below = kNeu;
        for ( int l = max( ra - 1, 0 ); l <= min( rb, P.N ); ++l )
        {
            const int          above = l < P.N ? layer_mode( l, P.N, P.mode_first, P.mode_inner, P.mode_last ) : kNeu;
            LevelSums< OP, T > t;
            T                  v[kStencil], diff[OP::D + 1];
#pragma unroll
            for ( int i = 0; i < kStencil; ++i )
                v[i] = u[( stencil_dx( i ) * ( kTileY + 2 ) + stencil_dy( i ) ) * kStride + l];
#pragma unroll
            for ( int k = 0; k < OP::S; ++k )
            {
                t.s[k] = OP::kDiff ? T( 0 ) : f[0][k] * v[0];
#pragma unroll
                for ( int i = 1; i < kStencil; ++i )
                    t.s[k] += f[i][k] * ( OP::kDiff ? v[i] - v[0] : v[i] );
            }
#pragma unroll
            for ( int k = 0; k < OP::D; ++k )
            {
                diff[k] = T( 0 );
#pragma unroll
                for ( int i = 0; i < kStencil; ++i )
                    diff[k] += f[i][OP::S + k] * ( v[i] - u[( stencil_dx( i ) * ( kTileY + 2 ) + stencil_dy( i ) ) * kStride + l - 1] );
            }
            if ( above != kNeu || below != kNeu ) // a layer next to this level that does not couple its levels
            {
#pragma unroll
                for ( int k = 0; k < OP::D; ++k )
                {
                    t.side[k] = T( 0 );
#pragma unroll
                    for ( int i = 0; i < kStencil; ++i )
                        t.side[k] += f[i][OP::S + k] * v[i];
                }
#pragma unroll
                for ( int k = 0; k < K; ++k )
                    t.self[k] = f[0][k] * v[0];
            }
            if ( l > 0 && l > ra - 1 )
            {
                T low, up, fr[R];
#pragma unroll
                for ( int i = 0; i < R; ++i )
                    fr[i] = rad[( l - ra ) * R + i];
                lateral_layer< OP >( below, fr, b, t, diff, low, up );
                if ( l - 1 >= ra )
                    o[l - 1] = high + low;
                high = up;
            }
            b     = t;
            below = above;
        }
        if ( rb == n1 )
            o[P.N] = high;
    }
    __syncthreads();
    T* dst = P.dst.at( blockIdx.y ) + ( ( size_t( d ) * n1 + x0 + 1 ) * n1 + y0 + 1 ) * n1;
    if ( hl < rb - ra )
    {
        const int ymax = min( kTileY, P.N - 1 - y0 );
        for ( int cx = half; cx < min( kTileX, P.N - 1 - x0 ); cx += kLateralThreads / 16 )
        {
            T*       g = dst + size_t( cx ) * n1 * n1 + ra + hl;
            const T* c = out + cx * kTileY * kStride + hl;
            if constexpr ( CG ) // interior columns are owned
            {
                T*       q = cg.p_new + ( g - P.dst.p[0] );
                const T* v = in + ( ( cx + 1 ) * ( kTileY + 2 ) + 1 ) * kStride + hl + 1;
                double   part[2] = { 0.0, 0.0 }; // plain sums per thread: two chains, compensated across threads
#pragma unroll
                for ( int cy = 0; cy < kTileY; ++cy, g += n1, q += n1 )
                    if ( cy < ymax )
                    {
                        *g = c[cy * kStride];
                        *q = v[cy * kStride];
                        if constexpr ( exact_dot )
                            dot.add( __dmul_rn( c[cy * kStride], v[cy * kStride] ) );
                        else
                            part[cy & 1] += c[cy * kStride] * v[cy * kStride];
                    }
                dot.add( part[0] + part[1] );
            }
            else
            {
#pragma unroll
                for ( int cy = 0; cy < kTileY; ++cy, g += n1 )
                    if ( cy < ymax )
                        lateral_store( g, c[cy * kStride], P.add );
            }
        }
    }
}

template < typename OP, bool CG, typename T >
__device__ __forceinline__ void lateral_edge( const LateralParams< T >& P, const LateralCG& cg, T beta, unsigned block, Neumaier& dot )
{
    constexpr int  K = OP::K, R = OP::R;
    const int      n1 = P.n1, N = P.N;
    const unsigned t = block * unsigned( kLateralThreads ) + threadIdx.x; // node (entry, level)
    if ( t >= P.edge_nodes )
        return;
    const int e = int( t / unsigned( n1 ) ), r = int( t - unsigned( e ) * unsigned( n1 ) );
    const int m0 = P.offsets ? P.offsets[e] : e, m1 = P.offsets ? P.offsets[e + 1] : e + 1;
    const T*  src = P.src.at( blockIdx.y );
    const int rd = max( r - 1, 0 ) - r, ru = min( r + 1, N ) - r; // levels past the ends are not used below
    LevelSums< OP, T > s[3]; // of the level below, the node's and the one above
    T                  diff[2][OP::D + 1];
#pragma unroll
    for ( int k = 0; k < OP::S; ++k )
        s[0].s[k] = s[1].s[k] = s[2].s[k] = T( 0 );
#pragma unroll
    for ( int k = 0; k < OP::D; ++k )
        diff[0][k] = diff[1][k] = s[1].side[k] = T( 0 );
#pragma unroll
    for ( int k = 0; k < K; ++k )
        s[1].self[k] = T( 0 );
    T owner = T( 0 ); // the direction at the owning (first) copy
    // value of stored node i: of the field, or of the new direction
    const auto value = [&]( ptrdiff_t i ) {
        if constexpr ( CG )
            return cg.r[i] + beta * src[i];
        else
            return src[i];
    };
    for ( int m = m0; m < m1; ++m )
    {
        const int       col = P.members[m], y = col % n1, x = col / n1 % n1;
        const ptrdiff_t u = ptrdiff_t( col ) * n1 + r;
        const T         v0[3] = { value( u + rd ), value( u ), value( u + ru ) };
        if constexpr ( CG )
        {
            cg.p_new[u] = v0[1];
            owner = m == m0 ? v0[1] : owner;
        }
#pragma unroll
        for ( int i = 0; i < kStencil; ++i )
        {
            const int dx = stencil_dx( i ), dy = stencil_dy( i );
            if ( x + dx < 0 || x + dx > N || y + dy < 0 || y + dy > N )
                continue; // no triangle of this diamond there
            const ptrdiff_t q = u + ptrdiff_t( dx * n1 + dy ) * n1;
            const T         v[3] = { i ? value( q + rd ) : v0[0], i ? value( q ) : v0[1], i ? value( q + ru ) : v0[2] };
#pragma unroll
            for ( int k = 0; k < K; ++k )
            {
                const T f = P.lat[size_t( i * K + k ) * P.columns + col];
                if ( k < OP::S )
                {
                    if ( i > 0 || !OP::kDiff )
#pragma unroll
                        for ( int l = 0; l < 3; ++l )
                            s[l].s[k] += f * ( OP::kDiff ? v[l] - v0[l] : v[l] );
                }
                else
                {
                    diff[0][k - OP::S] += f * ( v[1] - v[0] );
                    diff[1][k - OP::S] += f * ( v[2] - v[1] );
                    s[1].side[k - OP::S] += f * v[1];
                }
                if ( i == 0 )
                    s[1].self[k] += f * v[1];
            }
        }
    }
    T v = T( 0 ), low, high, fr[R];
    if ( r < N )
    {
#pragma unroll
        for ( int i = 0; i < R; ++i )
            fr[i] = P.rad[i * N + r];
        lateral_layer< OP >( layer_mode( r, N, P.mode_first, P.mode_inner, P.mode_last ), fr, s[1], s[2], diff[1], low, high );
        v += low;
    }
    if ( r > 0 )
    {
#pragma unroll
        for ( int i = 0; i < R; ++i )
            fr[i] = P.rad[i * N + r - 1];
        lateral_layer< OP >( layer_mode( r - 1, N, P.mode_first, P.mode_inner, P.mode_last ), fr, s[0], s[1], diff[0], low, high );
        v += high;
    }
    if constexpr ( CG )
        dot.add( owner * v );
    T* dst = P.dst.at( blockIdx.y );
    for ( int m = m0; m < m1; ++m )
        lateral_store( dst + size_t( P.members[m] ) * n1 + r, v, P.add );
}

// shared memory of a tile block: operands, results and radial factors
template < typename OP >
constexpr size_t lateral_words()
{
    return size_t( kTileCols + kTileX * kTileY ) * kStride + size_t( OP::R ) * ( kMaxRun + 1 );
}

template < typename OP, typename T >
__global__ void __launch_bounds__( kLateralThreads, 4 ) lateral_kernel( LateralParams< T > P )
{
    extern __shared__ double lateral_smem[];
    T*                       smem = reinterpret_cast< T* >( lateral_smem );
    Neumaier                 none;
    if ( blockIdx.x < P.edge_blocks )
        lateral_edge< OP, false >( P, LateralCG{}, T( 0 ), blockIdx.x, none );
    else
        lateral_tile< OP, false >( P, LateralCG{}, T( 0 ), blockIdx.x - P.edge_blocks, smem, none );
}

// Launches lateral_kernel for every node of nc fields; Replace with additive communication merges the copies, Add
// with additive communication adds this call's own sums first and then sums the copies (halo_sum).
template < typename T >
int halo_sum( const tn_mesh* m, T* const* fields, int nfields, cudaStream_t st );

// fills the launch shape of P (merge: the copies of a column are summed and all written) and returns its blocks
template < typename T >
unsigned lateral_shape( const tn_mesh* m, bool merge, LateralParams< T >& P )
{
    P.N = m->N, P.n1 = m->n1, P.columns = m->nlat;
    P.tiles_x = ( m->N - 1 + kTileX - 1 ) / kTileX, P.tiles_y = ( m->N - 1 + kTileY - 1 ) / kTileY;
    const unsigned tiles = unsigned( m->nd ) * unsigned( P.tiles_x * P.tiles_y );
    // runs of at most kMaxRun levels; shorter ones (down to 8) while they leave SMs without a block
    P.runs = ( m->n1 + kMaxRun - 1 ) / kMaxRun;
    while ( tiles * unsigned( P.runs ) < 2u * 148u && m->n1 > 8 * P.runs )
        ++P.runs;
    P.run         = ( m->n1 + P.runs - 1 ) / P.runs;
    P.runs        = ( m->n1 + P.run - 1 ) / P.run;
    P.members     = m->d_halo_members;
    P.offsets     = merge ? m->d_halo_offsets : nullptr;
    P.edge_nodes  = unsigned( merge ? m->n_halo_groups : m->n_halo_members ) * unsigned( m->n1 );
    P.edge_blocks = ( P.edge_nodes + kLateralThreads - 1 ) / kLateralThreads;
    return P.edge_blocks + tiles * unsigned( P.runs );
}

// allows `kernel` the shared memory of a tile block, once per device
template < typename OP, typename T, typename F >
int lateral_opt_in( std::atomic< bool > ( &done )[kMaxDevices], F* kernel )
{
    const int dev = current_device();
    if ( !done[dev].load( std::memory_order_acquire ) )
    {
        TN_CUDA_TRY( cudaFuncSetAttribute( kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           int( sizeof( T ) * lateral_words< OP >() ) ) );
        done[dev].store( true, std::memory_order_release );
    }
    return TN_OK;
}

template < typename OP, typename T >
int launch_lateral( const tn_mesh* m, LateralParams< T > P, int nc, int apply_mode, int comm_mode, cudaStream_t st )
{
    P.add = apply_mode == TN_APPLY_ADD;
    const bool     merge  = !P.add && comm_mode == TN_COMM_ADDITIVE;
    const unsigned blocks = lateral_shape( m, merge, P );
    static std::atomic< bool > opted_in[kMaxDevices];
    if ( const int rc = lateral_opt_in< OP, T >( opted_in, lateral_kernel< OP, T > ) )
        return rc;
    lateral_kernel< OP, T ><<< dim3( blocks, unsigned( nc ) ), kLateralThreads, sizeof( T ) * lateral_words< OP >(), st >>>( P );
    TN_LAUNCH_CHECK();
    if ( !merge && comm_mode == TN_COMM_ADDITIVE )
        return halo_sum< T >( m, P.dst.p, nc, st );
    return TN_OK;
}

// Unevaluated sum of two doubles (v the rounded sum), for tables whose entries are to carry no more than their own
// rounding: error-free sums (Knuth's two-sum) and products (fused multiply-add).
struct Pair
{
    double v = 0.0, e = 0.0;
};
__device__ __forceinline__ Pair pair_sum( double a, double b )
{
    const double s = a + b, z = s - a;
    return { s, ( a - ( s - z ) ) + ( b - z ) };
}
__device__ __forceinline__ Pair operator+( const Pair& a, const Pair& b )
{
    const Pair s = pair_sum( a.v, b.v );
    return pair_sum( s.v, s.e + ( a.e + b.e ) );
}
__device__ __forceinline__ Pair operator-( const Pair& a )
{
    return { -a.v, -a.e };
}
__device__ __forceinline__ Pair operator*( const Pair& a, const Pair& b )
{
    const double p = __dmul_rn( a.v, b.v );
    return pair_sum( p, fma( a.v, b.v, -p ) + ( a.v * b.e + a.e * b.v ) );
}
// a / d rounded once (but for ties)
__device__ __forceinline__ double quotient( const Pair& a, double d )
{
    const double q = a.v / d;
    return q + ( fma( -q, d, a.v ) + a.e ) / d;
}

// Tabulates an operator's stencils ([7 K][column], thread per column: OP::triangle adds the factors between vertex i of
// a triangle and its three to their entries, OP::entry is the value of such a sum) and radial factors ([R][layer],
// OP::radial), in the precisions that are given an array.
struct LateralTables
{
    double *lat, *rad;
    float * lat32, *rad32;
};
template < typename OP >
__global__ void __launch_bounds__( 128 ) lateral_table_kernel( int N, size_t columns, const double* __restrict__ coords,
                                                              const double* __restrict__ radii, LateralTables t )
{
    const auto put = []( double* d, float* f, size_t i, double v ) {
        if ( d )
            d[i] = v;
        if ( f )
            f[i] = float( v );
    };
    const size_t col = blockIdx.x * size_t( blockDim.x ) + threadIdx.x;
    const int    n1  = N + 1;
    if ( col < size_t( N ) )
    {
        double f[OP::R];
        OP::radial( radii[col], radii[col + 1], f );
#pragma unroll
        for ( int i = 0; i < OP::R; ++i )
            put( t.rad, t.rad32, size_t( i ) * N + col, f[i] );
    }
    if ( col >= columns )
        return;
    const int y = int( col % n1 ), x = int( col / n1 % n1 );
    typename OP::Sum A[kStencil][OP::K] = {};
#pragma unroll
    for ( int w = 0; w < 2; ++w )
#pragma unroll
        for ( int i = 0; i < 3; ++i )
        {
            // the triangle w whose vertex i is this column
            const int cx = x - wedge_node( w, i, 0 ), cy = y - wedge_node( w, i, 1 );
            if ( cx < 0 || cy < 0 || cx >= N || cy >= N )
                continue;
            const double* p[3];
            int           e[3];
#pragma unroll
            for ( int j = 0; j < 3; ++j )
            {
                const int dx = wedge_node( w, j, 0 ) - wedge_node( w, i, 0 ), dy = wedge_node( w, j, 1 ) - wedge_node( w, i, 1 );
                p[j] = coords + ( col + ptrdiff_t( dx ) * n1 + dy ) * 3;
                e[j] = stencil_entry( dx, dy );
            }
            OP::triangle( p[0], p[1], p[2], i, e, A );
        }
#pragma unroll
    for ( int e = 0; e < kStencil; ++e )
#pragma unroll
        for ( int k = 0; k < OP::K; ++k )
            put( t.lat, t.lat32, size_t( e * OP::K + k ) * columns + col, OP::entry( A[e][k], e ) );
}

// the double or single precision member of a table pair
template < typename T >
T*& lateral_slot( double*& d, float*& f )
{
    if constexpr ( sizeof( T ) == 8 )
        return d;
    else
        return f;
}

// values of an operator's stencil and radial tables on mesh m, and the launch that fills them
template < typename OP >
size_t lateral_table_words( const tn_mesh* m, bool radial )
{
    return radial ? size_t( OP::R ) * m->N : size_t( kStencil * OP::K ) * m->nlat;
}
template < typename OP >
bool lateral_fill( const tn_mesh* m, const LateralTables& t, cudaStream_t st )
{
    const size_t n = std::max( m->nlat, size_t( m->N ) );
    lateral_table_kernel< OP ><<< unsigned( ( n + 127 ) / 128 ), 128, 0, st >>>( m->N, m->nlat, m->d_coords, m->d_radii, t );
    return cudaGetLastError() == cudaSuccess;
}

// An operator's tables in the precision of T, built on the mesh's first use of them and complete for every stream when
// this returns; false when that fails.  The first use may lie in a stream capture (that of another precision or of an
// operator that shares no table may have come before it): the fill runs on a stream of its own, and allocating is allowed
// to this thread meanwhile.
template < typename OP, typename T >
bool lateral_tables( const tn_mesh* m, tn_lateral_tables tn_mesh::*which, LateralParams< T >& P )
{
    struct AllowAllocation
    {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        AllowAllocation() { cudaThreadExchangeStreamCaptureMode( &mode ); }
        ~AllowAllocation() { cudaThreadExchangeStreamCaptureMode( &mode ); }
    };
    tn_mesh*                      mm = const_cast< tn_mesh* >( m );
    std::lock_guard< std::mutex > lock( mm->geom_mutex );
    tn_lateral_tables&            t    = mm->*which;
    T *&                          dlat = lateral_slot< T >( t.lat, t.lat32 ), *&drad = lateral_slot< T >( t.rad, t.rad32 );
    if ( !dlat )
    {
        const AllowAllocation allow;
        const size_t          words = lateral_table_words< OP >( m, false );
        T*                    l     = nullptr; // the stencils, then the radial factors
        cudaStream_t          st    = nullptr;
        LateralTables         out{};
        bool ok = cudaMalloc( &l, ( words + lateral_table_words< OP >( m, true ) ) * sizeof( T ) ) == cudaSuccess &&
                  cudaStreamCreateWithFlags( &st, cudaStreamNonBlocking ) == cudaSuccess;
        if ( ok )
        {
            lateral_slot< T >( out.lat, out.lat32 ) = l, lateral_slot< T >( out.rad, out.rad32 ) = l + words;
            ok = lateral_fill< OP >( m, out, st ) && cudaStreamSynchronize( st ) == cudaSuccess;
        }
        if ( st )
            cudaStreamDestroy( st );
        if ( !ok )
        {
            (void) cudaGetLastError();
            cudaFree( l );
            return false;
        }
        dlat = l, drad = l + words;
    }
    P.lat = dlat, P.rad = drad;
    return true;
}

}  // namespace tn
