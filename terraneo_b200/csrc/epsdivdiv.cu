// EpsilonDivDiv with the 3x2 Felippa rule (fe/wedge/operators/shell/
// epsilon_divdiv.hpp:218-600): int k (2 eps(u):eps(v) - 2/3 div u div v) with
// k interpolated by the wedge shape functions at each of the six quadrature
// points.  treat_boundary eliminates the CMB nodes of layer 0 (otherwise the
// SURFACE nodes of layer N-1) keeping their diagonal; diagonal mode keeps only
// the diagonal.  The reference runs nine (dim_i, dim_j) passes per cell; here
// one pass per quadrature point forms grad u over the coupled nodes and tests
// it with every node at once.
//
// Factored form (cell.cuh).  At a point the scaled gradient matrix D r G =
// beta_1 (x) S_1 + beta_2 (x) S_2 + v (x) Z has edge differences S_i of u that
// depend on zeta only and Z = rho T - xi S_1 - eta S_2 (T = sum_m lat_m (u_top -
// u_bottom) / 2 of vertex m).  So only Z changes over the three lateral points of
// a zeta; the stress of beta (x) S is formed once, v (x) Z adds
//     omega (sym(v (x) Z)) v = omega (|v|^2 Z + (v . Z) v / 3),
// and the test side needs the zeta's summed stress M against beta_1 and beta_2 and
// the moments of (stress v) over the points: about 480 multiply-adds per wedge
// instead of 2,100 (Jacobian, inverse and six gradients at every point).
//
// One thread per cell (r fastest), contributions added by add_column: the upper
// nodes are handed to the lane above, 12 atomics per cell.  Nodes that the
// boundary treatment decouples enter with zero; their diagonal comes from
// further blocks of the launch (one thread per lateral cell, wedge and side).
// Level-6 apply with its halo: FP64 1,067 -> 246 us, FP32 577 -> 153 us, bound by
// instruction issue.
#include "cell.cuh"
#include "common.cuh"
#include "wedge.cuh"

namespace tn {

template < typename T >
int halo_sum( const tn_mesh* m, T* const* fields, int nfields, cudaStream_t st );

namespace {

template < typename T >
struct E32Params
{
    int             N, n1;
    const T*        table;
    const T*        k;
    Ptr3< const T > src;
    Ptr3< T >       dst;
    int             treat;
    unsigned        cell_blocks; // blocks of cells; those after them add diagonals
};

// one wedge from the values s of its six nodes (bottom 0-2, top 3-5) and k there; out[n][c] = its row of node n
template < typename T >
__device__ __forceinline__ void epsdivdiv_wedge( const Triangle< T >& G, T h, T rho_b, T rho_t, const T ( &s )[6][3],
                                                 const T ( &kn )[6], T ( &out )[6][3] )
{
    // omega = k h / (6 |D|) at the lateral points, bottom and top: k there is (the sum + 3 the near vertex) / 6, and both
    // sixths are one rounded factor
    const T scale = T( 1.0 / 36.0 ) * h * fabs( G.iD );
    T       kb[3], kt[3];
    {
        const T sb = kn[0] + kn[1] + kn[2], st = kn[3] + kn[4] + kn[5];
#pragma unroll
        for ( int q = 0; q < 3; ++q )
        {
            const int m = ( q + 1 ) % 3; // point q lies next to vertex m
            kb[q] = scale * ( sb + T( 3 ) * kn[m] ), kt[q] = scale * ( st + T( 3 ) * kn[3 + m] );
        }
    }
    const T vv = dot3( G.v, G.v );
    T       t[3][3], ts[3], L[3][3];
#pragma unroll
    for ( int c = 0; c < 3; ++c )
    {
#pragma unroll
        for ( int m = 0; m < 3; ++m )
            t[m][c] = T( 0.5 ) * ( s[3 + m][c] - s[m][c] ), L[m][c] = T( 0 );
        ts[c] = ( t[0][c] + t[1][c] + t[2][c] ) * T( 1.0 / 6.0 );
    }
#pragma unroll
    for ( int n = 0; n < 6; ++n )
        out[n][0] = out[n][1] = out[n][2] = T( 0 );
#pragma unroll
    for ( int zq = 0; zq < 2; ++zq )
    {
        const T nb = T( zq ? 0.5 * ( 1.0 - kFelippaZ ) : 0.5 * ( 1.0 + kFelippaZ ) );
        const T nt = T( zq ? 0.5 * ( 1.0 + kFelippaZ ) : 0.5 * ( 1.0 - kFelippaZ ) );
        const T rho = zq ? rho_t : rho_b;
        T       S1[3], S2[3], Z0[3];
#pragma unroll
        for ( int c = 0; c < 3; ++c )
        {
            S1[c] = nb * ( s[1][c] - s[0][c] ) + nt * ( s[4][c] - s[3][c] );
            S2[c] = nb * ( s[2][c] - s[0][c] ) + nt * ( s[5][c] - s[3][c] );
            Z0[c] = rho * ts[c] - T( 1.0 / 6.0 ) * ( S1[c] + S2[c] );
        }
        // E = B + B^T - 2/3 tr B of B = beta_1 (x) S_1 + beta_2 (x) S_2, and E v
        T B[3][3];
#pragma unroll
        for ( int a = 0; a < 3; ++a )
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                B[a][c] = G.b1[a] * S1[c] + G.b2[a] * S2[c];
        const T tr = T( 2.0 / 3.0 ) * ( B[0][0] + B[1][1] + B[2][2] );
        const T E00 = T( 2 ) * B[0][0] - tr, E11 = T( 2 ) * B[1][1] - tr, E22 = T( 2 ) * B[2][2] - tr;
        const T E01 = B[0][1] + B[1][0], E02 = B[0][2] + B[2][0], E12 = B[1][2] + B[2][1];
        const T e[3] = { E00 * G.v[0] + E01 * G.v[1] + E02 * G.v[2], E01 * G.v[0] + E11 * G.v[1] + E12 * G.v[2],
                         E02 * G.v[0] + E12 * G.v[1] + E22 * G.v[2] };
        T om = T( 0 ), Zs[3] = { T( 0 ), T( 0 ), T( 0 ) }, ev[2][3];
#pragma unroll
        for ( int q = 0; q < 3; ++q )
        {
            const T w = nb * kb[q] + nt * kt[q];
            T       Z[3];
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                Z[c] = Z0[c] + T( 0.5 ) * ( q == 0 ? rho * t[1][c] - S1[c] : ( q == 1 ? rho * t[2][c] - S2[c] : rho * t[0][c] ) );
            om += w;
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                Zs[c] += w * Z[c];
            if ( q < 2 )
            {
                const T vz = T( 1.0 / 3.0 ) * dot3( G.v, Z );
#pragma unroll
                for ( int c = 0; c < 3; ++c )
                    ev[q][c] = w * ( e[c] + vv * Z[c] + vz * G.v[c] );
            }
        }
        // M = sum omega (E + v (x) Z + Z (x) v - 2/3 (v . Z))
        const T vz  = T( 2.0 / 3.0 ) * dot3( G.v, Zs );
        const T M00 = om * E00 + T( 2 ) * G.v[0] * Zs[0] - vz, M11 = om * E11 + T( 2 ) * G.v[1] * Zs[1] - vz;
        const T M22 = om * E22 + T( 2 ) * G.v[2] * Zs[2] - vz, M01 = om * E01 + G.v[0] * Zs[1] + G.v[1] * Zs[0];
        const T M02 = om * E02 + G.v[0] * Zs[2] + G.v[2] * Zs[0], M12 = om * E12 + G.v[1] * Zs[2] + G.v[2] * Zs[1];
        const T F1[3] = { M00 * G.b1[0] + M01 * G.b1[1] + M02 * G.b1[2], M01 * G.b1[0] + M11 * G.b1[1] + M12 * G.b1[2],
                          M02 * G.b1[0] + M12 * G.b1[1] + M22 * G.b1[2] };
        const T F2[3] = { M00 * G.b2[0] + M01 * G.b2[1] + M02 * G.b2[2], M01 * G.b2[0] + M11 * G.b2[1] + M12 * G.b2[2],
                          M02 * G.b2[0] + M12 * G.b2[1] + M22 * G.b2[2] };
        const T V[3]  = { M00 * G.v[0] + M01 * G.v[1] + M02 * G.v[2], M01 * G.v[0] + M11 * G.v[1] + M12 * G.v[2],
                          M02 * G.v[0] + M12 * G.v[1] + M22 * G.v[2] };
#pragma unroll
        for ( int c = 0; c < 3; ++c )
        {
            // moments of (stress v) with xi, eta
            const T X = T( 1.0 / 6.0 ) * V[c] + T( 0.5 ) * ev[0][c], Y = T( 1.0 / 6.0 ) * V[c] + T( 0.5 ) * ev[1][c];
            const T f1 = F1[c] - X, f2 = F2[c] - Y, f0 = -( f1 + f2 );
            out[0][c] += nb * f0, out[1][c] += nb * f1, out[2][c] += nb * f2;
            out[3][c] += nt * f0, out[4][c] += nt * f1, out[5][c] += nt * f2;
            L[0][c] += rho * ( V[c] - X - Y ), L[1][c] += rho * X, L[2][c] += rho * Y;
        }
    }
#pragma unroll
    for ( int m = 0; m < 3; ++m )
#pragma unroll
        for ( int c = 0; c < 3; ++c )
            out[m][c] -= T( 0.5 ) * L[m][c], out[3 + m][c] += T( 0.5 ) * L[m][c];
}

// adds the diagonal entries of the three lower (top false) or upper nodes of a wedge times their values
template < typename T >
__device__ __forceinline__ void epsdivdiv_diagonal( const E32Params< T >& P, int d, int x, int y, int r, int w, bool top )
{
    const T             h = layer_h( P.table, P.N, r ), rq = layer_q( P.table, P.N, r ), side = top ? T( 1 ) : T( -1 );
    const Triangle< T > G( P.table, P.N, d, x, y, w );
    unsigned            node[4], id[3];
    T                   kn[6], o[3][3];
    cell_nodes( P.n1, d, x, y, r, node );
    wedge_columns( node, w, id );
#pragma unroll
    for ( int n = 0; n < 6; ++n )
        kn[n] = P.k[id[n % 3] + n / 3];
#pragma unroll
    for ( int m = 0; m < 3; ++m )
        o[m][0] = o[m][1] = o[m][2] = T( 0 );
#pragma unroll
    for ( int q = 0; q < 6; ++q )
    {
        const T xi = T( felippa_xi( q ) ), eta = T( felippa_eta( q ) ), zeta = T( q < 3 ? -kFelippaZ : kFelippaZ );
        const T lat[3] = { T( 1 ) - xi - eta, xi, eta };
        T       k = T( 0 );
#pragma unroll
        for ( int n = 0; n < 6; ++n )
            k += lat[n % 3] * T( 0.5 ) * ( n < 3 ? T( 1 ) - zeta : T( 1 ) + zeta ) * kn[n];
        const T om = T( kFelippaW ) * k * h * fabs( G.iD ), rho = rq + T( 1 ) + zeta;
#pragma unroll
        for ( int m = 0; m < 3; ++m )
        {
            T g[3];
            scaled_gradient( G, m, side, xi, eta, zeta, rho, g );
            const T gg = dot3( g, g );
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                o[m][c] += om * ( gg + g[c] * g[c] * T( 1.0 / 3.0 ) );
        }
    }
#pragma unroll
    for ( int m = 0; m < 3; ++m )
#pragma unroll
        for ( int c = 0; c < 3; ++c )
            atomicAdd( P.dst.p[c] + id[m] + top, o[m][c] * P.src.p[c][id[m] + top] );
}

// Blocks per SM, level 6: FP64 at 3 / 4 / 5 blocks 248 / 252 / 319 us (36 bytes spilled at 3, more above), FP32 at 4 / 5 /
// 6 165 / 155 / 153 us (24 bytes at 6).
template < typename T >
__global__ void __launch_bounds__( 128, sizeof( T ) == 8 ? 3 : 6 ) epsdivdiv3x2_kernel( E32Params< T > P )
{
    const int N = P.N, n1 = P.n1;
    int       d, x, y, r;
    if ( blockIdx.x >= P.cell_blocks )
    {
        // the kept diagonal of the CMB side of layer 0 and of the SURFACE side of layer N - 1
        int  w;
        bool top;
        if ( boundary_item( ( blockIdx.x - P.cell_blocks ) * blockDim.x + threadIdx.x, N, d, x, y, r, w, top ) )
            epsdivdiv_diagonal( P, d, x, y, r, w, top );
        return;
    }
    const bool in  = cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, N, d, x, y, r );
    const bool bot = P.treat && r == 0, top = P.treat && !bot && r == N - 1;
    const T    h = layer_h( P.table, N, r ), rq = layer_q( P.table, N, r );
    const T    rho_b = rq + T( 1.0 - kFelippaZ ), rho_t = rq + T( 1.0 + kFelippaZ );
    T* const   dst[3] = { P.dst.p[0], P.dst.p[1], P.dst.p[2] };
    unsigned   node[4];
    T          s[4][2][3], k[4][2];
    cell_nodes( n1, d, x, y, r, node );
#pragma unroll
    for ( int i = 0; i < 4; ++i )
    {
#pragma unroll
        for ( int l = 0; l < 2; ++l )
        {
            k[i][l] = P.k[node[i] + l];
#pragma unroll
            for ( int c = 0; c < 3; ++c )
            {
                const T v  = P.src.p[c][node[i] + l];
                s[i][l][c] = ( l ? top : bot ) ? T( 0 ) : v;
            }
        }
    }
    T acc[2][2][3]; // columns 1 and 2 get both wedges
#pragma unroll
    for ( int w = 0; w < 2; ++w )
    {
        const Triangle< T > G( P.table, N, d, x, y, w );
        T                   sw[6][3], kw[6], out[6][3];
#pragma unroll
        for ( int n = 0; n < 6; ++n )
        {
            const int i = wedge_node( w, n, 0 ) + 2 * wedge_node( w, n, 1 ), l = n / 3;
            kw[n]       = k[i][l];
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                sw[n][c] = s[i][l][c];
        }
        epsdivdiv_wedge( G, h, rho_b, rho_t, sw, kw, out );
        // wedge 0: vertices columns 0, 1, 2; wedge 1: columns 3, 2, 1
        add_column< T, 3 >( dst, node[w ? 3 : 0], r, N, in, !bot, !top, out[0], out[3] );
#pragma unroll
        for ( int m = 1; m < 3; ++m )
        {
            const int a = w ? 2 - m : m - 1; // column m of wedge 0, 3 - m of wedge 1
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                if ( w == 0 )
                    acc[a][0][c] = out[m][c], acc[a][1][c] = out[3 + m][c];
                else
                    acc[a][0][c] += out[m][c], acc[a][1][c] += out[3 + m][c];
        }
    }
    add_column< T, 3 >( dst, node[1], r, N, in, !bot, !top, acc[0][0], acc[0][1] );
    add_column< T, 3 >( dst, node[2], r, N, in, !bot, !top, acc[1][0], acc[1][1] );
}

// the diagonal alone: one thread per cell, wedge and side (blockIdx.y)
template < typename T >
__global__ void __launch_bounds__( 128 ) epsdivdiv3x2_diagonal_kernel( E32Params< T > P )
{
    int d, x, y, r;
    if ( cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, P.N, d, x, y, r ) )
        epsdivdiv_diagonal( P, d, x, y, r, int( blockIdx.y & 1 ), blockIdx.y >= 2 );
}

}  // namespace

template < typename T >
int epsdivdiv3x2_apply( const tn_mesh* m, const T* k, int treat, int diag, int apply_mode, int comm_mode,
                        const T* const* src, T* const* dst, cudaStream_t st )
{
    TN_CHECK_ARG( m && k && src && dst, "epsdivdiv3x2_apply: null argument" );
    TN_CHECK_ARG( apply_mode == TN_APPLY_REPLACE || apply_mode == TN_APPLY_ADD, "epsdivdiv3x2_apply: bad apply mode" );
    E32Params< T > P{};
    for ( int c = 0; c < 3; ++c )
    {
        TN_CHECK_ARG( src[c] && dst[c], "epsdivdiv3x2_apply: null vector component" );
        P.src.p[c] = src[c];
        P.dst.p[c] = dst[c];
    }
    if ( apply_mode == TN_APPLY_REPLACE )
        TN_CUDA_TRY( zero_fields( dst, 3, m->ns, st ) );
    P.N = m->N, P.n1 = m->n1, P.k = k, P.treat = treat != 0, P.table = triangle_table< T >( m );
    const long long cells = (long long) kDiamonds * m->N * m->N * m->N;
    P.cell_blocks         = unsigned( ( cells + 127 ) / 128 );
    const unsigned edge   = treat ? ( boundary_items( m->N ) + 127u ) / 128u : 0u;
    if ( diag )
        epsdivdiv3x2_diagonal_kernel< T ><<< dim3( P.cell_blocks, 4 ), 128, 0, st >>>( P );
    else
        epsdivdiv3x2_kernel< T ><<< P.cell_blocks + edge, 128, 0, st >>>( P );
    TN_LAUNCH_CHECK();
    if ( comm_mode == TN_COMM_ADDITIVE )
        return halo_sum< T >( m, dst, 3, st );
    return TN_OK;
}

}  // namespace tn

using namespace tn;

extern "C" int tn_epsdivdiv3x2_apply_f64( const tn_mesh* m, const double* k, int treat_boundary, int diagonal,
                                          int apply_mode, int comm_mode, const double* const* src, double* const* dst,
                                          void* s )
{
    return epsdivdiv3x2_apply< double >( m, k, treat_boundary, diagonal, apply_mode, comm_mode, src, dst,
                                         as_stream( s ) );
}
extern "C" int tn_epsdivdiv3x2_apply_f32( const tn_mesh* m, const float* k, int treat_boundary, int diagonal,
                                          int apply_mode, int comm_mode, const float* const* src, float* const* dst,
                                          void* s )
{
    return epsdivdiv3x2_apply< float >( m, k, treat_boundary, diagonal, apply_mode, comm_mode, src, dst,
                                        as_stream( s ) );
}
