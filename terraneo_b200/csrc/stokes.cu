// Stokes coupling blocks: Divergence B (fine P1 velocity -> coarse P1
// pressure, fe/wedge/operators/shell/divergence.hpp) and Gradient B^T
// (gradient.hpp), Q1-iso-Q2 / Q1 with the 3x2 Felippa rule.
//
// B_{i,(d,j)} = -int (J^{-T} grad N_j)_d N^c_i |det J| over each fine wedge,
// N^c_i the coarse shape functions of the coarse wedge containing it
// (shape_coarse, integrands.hpp:266-400).  The coarse node each wedge-local
// coarse slot is added to follows the reference's wedge map
// (atomically_add_local_wedge_scalar_coefficients, kernel_helpers.hpp:407):
// fine wedge w always scatters to coarse wedge w's node positions, also for
// the two middle fine triangles whose shape functions belong to the other
// coarse wedge.  Kept as is for parity; Gradient uses the same map, so B^T is
// the exact transpose.
//
// Boundary conditions act on the velocity side: Dirichlet nodes are dropped,
// free-slip nodes are projected onto the tangent plane (the reference's
// rotate / eliminate-normal / rotate-back sequence, :226-290).
//
// Factored form (cell.cuh).  Every quadrature point has
//     |det J| grad N_n = sign(D) ( r h nr_n(zeta) u_m + r^2 s_n lat_m v ),  u_m = beta_m - lat_m v
// (m the lateral vertex of node n), and the coarse shape function is a lateral
// factor latc_i times a radial one.  On the tensor-product 3x2 rule the lateral
// and radial sums separate, and the lateral ones are numbers of the fine
// triangle's position in the coarse one alone,
//     C0_i = sum_q w latc_i,  C1_im = sum_q w latc_i lat_m,
// so a wedge needs only beta_1, beta_2 and v of its triangle:
//     B_{i,(n,:)} = -sign(D) ( Ra[i/3][n/3] (C0_i beta_m - C1_im v) + s_n Rb[i/3] C1_im v )
// with the radial sums Ra = sum_zeta radc_i r h nr_n, Rb = sum_zeta radc_i r^2
// formed per cell: the same integrals as the per-point Jacobian of
// fe/wedge/integrands.hpp, about 90 multiply-adds per wedge and direction (200
// and a table of 39 values per wedge when U_im = C0_i beta_m - C1_im v was
// tabulated).
//
// One thread per fine cell, r fastest.  In B the two fine cells of one coarse
// cell (neighbouring lanes) add together and hand their upper coarse nodes to
// the next pair; in B^T the upper fine nodes go to the lane above (add_column).
// Free-slip applies, FP64: B 288 -> 109 us and B^T 208 -> 127 us at level 6, 1,778 ->
// 719 and 1,479 -> 968 us at level 7; bound by instruction issue (53 and 59 % of the
// slots), B^T also by its 12 atomics per cell.
#include <cmath>

#include "cell.cuh"
#include "common.cuh"
#include "wedge.cuh"

namespace tn {

template < typename T >
int halo_sum( const tn_mesh* m, T* const* fields, int nfields, cudaStream_t st );

namespace {

// coarse lateral shape coefficients (a, b xi, c eta) per [node % 3][fine lateral wedge index]
// (shape_coarse, integrands.hpp:266-400)
__device__ constexpr double kCoarseLat[3][4][3] = {
    { { 1.0, -0.5, -0.5 }, { 0.5, -0.5, -0.5 }, { 0.5, -0.5, -0.5 }, { 0.0, 0.5, 0.5 } },
    { { 0.0, 0.5, 0.0 }, { 0.5, 0.5, 0.0 }, { 0.0, 0.5, 0.0 }, { 0.5, -0.5, 0.0 } },
    { { 0.0, 0.0, 0.5 }, { 0.0, 0.0, 0.5 }, { 0.5, 0.0, 0.5 }, { 0.5, 0.0, -0.5 } } };

__device__ __forceinline__ int fine_lateral_wedge( int x, int y, int w )
{
    // fine_lateral_wedge_idx (kernel_helpers.hpp:601)
    const int xm = x & 1, ym = y & 1;
    return w == 0 ? ( ym * 2 + xm ) : ( 3 - ( ym * 2 + xm ) );
}

// C0_i and C1_im of fine triangle `flat`: with the weight 1/6 the rule's sums of 1, xi (or eta), xi^2 (eta^2) and
// xi eta are 1/2, 1/6, 1/12 and 1/24
template < typename T >
struct CoarseMoments
{
    T c0[3], c1[3][3];
    __device__ __forceinline__ explicit CoarseMoments( int flat )
    {
#pragma unroll
        for ( int i = 0; i < 3; ++i )
        {
            const T a = T( kCoarseLat[i][flat][0] ), b = T( kCoarseLat[i][flat][1] ), c = T( kCoarseLat[i][flat][2] );
            c0[i]    = T( 0.5 ) * a + T( 1.0 / 6.0 ) * ( b + c );
            c1[i][1] = T( 1.0 / 6.0 ) * a + T( 1.0 / 12.0 ) * b + T( 1.0 / 24.0 ) * c;
            c1[i][2] = T( 1.0 / 6.0 ) * a + T( 1.0 / 24.0 ) * b + T( 1.0 / 12.0 ) * c;
            c1[i][0] = c0[i] - c1[i][1] - c1[i][2];
        }
    }
};

template < typename T >
struct StokesParams
{
    int           N, n1, nc1;
    const double* coords; // fine lateral coords (unit vectors: the outward normals)
    const T*      table;  // triangles of the fine mesh
    int           bc_cmb, bc_surf;
};

// a -= (n . a) n with the outward normal of lateral point c
template < typename T >
__device__ __forceinline__ void project_tangential( const double* __restrict__ c, T a[3] )
{
    const T n[3] = { T( c[0] ), T( c[1] ), T( c[2] ) }, d = dot3( n, a );
    a[0] -= d * n[0], a[1] -= d * n[1], a[2] -= d * n[2];
}

// radial sums of one fine cell: Ra[ib][nb] = h sum_zeta radc_ib r nr_nb, Rb[ib] = sum_zeta radc_ib r^2
template < typename T >
__device__ __forceinline__ void radial_sums( T h, T r1, int frad, T Ra[2][2], T Rb[2] )
{
    Ra[0][0] = Ra[0][1] = Ra[1][0] = Ra[1][1] = Rb[0] = Rb[1] = T( 0 );
#pragma unroll
    for ( int zq = 0; zq < 2; ++zq )
    {
        const T zeta = zq ? T( kFelippaZ ) : T( -kFelippaZ );
        const T rr   = r1 + h * ( T( 1 ) + zeta );
        const T nr[2] = { T( 0.5 ) * ( T( 1 ) - zeta ), T( 0.5 ) * ( T( 1 ) + zeta ) };
        const T rc[2] = { frad == 0 ? T( 0.25 ) * ( T( 3 ) - zeta ) : T( 0.25 ) * ( T( 1 ) - zeta ),
                          frad == 0 ? T( 0.25 ) * ( T( 1 ) + zeta ) : T( 0.25 ) * ( T( 3 ) + zeta ) };
#pragma unroll
        for ( int ib = 0; ib < 2; ++ib )
        {
            Rb[ib] += rc[ib] * rr * rr;
#pragma unroll
            for ( int nb = 0; nb < 2; ++nb )
                Ra[ib][nb] += rc[ib] * rr * h * nr[nb];
        }
    }
}

// p_coarse += B u
// Blocks per SM, level 6: FP64 at 3 / 4 / 6 blocks 126 / 109 / 111 us, FP32 at 4 / 5 / 6 86 / 80 / 76 us.
template < typename T >
__global__ void __launch_bounds__( 128, sizeof( T ) == 8 ? 4 : 6 ) divergence_kernel( StokesParams< T > P, Ptr3< const T > u, T* __restrict__ p )
{
    const int  N = P.N, n1 = P.n1, nc1 = P.nc1, lane = int( threadIdx.x ) & 31;
    int        d, x, y, r;
    const bool in = cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, N, d, x, y, r );
    unsigned node[4];
    T        uu[4][2][3];
    cell_nodes( n1, d, x, y, r, node );
#pragma unroll
    for ( int i = 0; i < 4; ++i )
#pragma unroll
        for ( int l = 0; l < 2; ++l )
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                uu[i][l][c] = u.p[c][node[i] + l];
    // velocity boundary conditions: Dirichlet nodes are dropped, free-slip ones projected
#pragma unroll
    for ( int l = 0; l < 2; ++l )
    {
        const int bc = l == 0 ? ( r == 0 ? P.bc_cmb : 0 ) : ( r == N - 1 ? P.bc_surf : 0 );
        if ( bc == TN_BC_DIRICHLET )
#pragma unroll
            for ( int i = 0; i < 4; ++i )
                uu[i][l][0] = uu[i][l][1] = uu[i][l][2] = T( 0 );
        else if ( bc == TN_BC_FREESLIP )
#pragma unroll
            for ( int i = 0; i < 4; ++i )
                project_tangential( P.coords + lat_index( n1, d, x + ( i & 1 ), y + ( i >> 1 ) ) * 3, uu[i][l] );
    }
    T Ra[2][2], Rb[2];
    radial_sums( layer_h( P.table, N, r ), layer_r( P.table, N, r ), r & 1, Ra, Rb );
    T acc[4][2]; // coarse columns as the fine ones
#pragma unroll
    for ( int i = 0; i < 4; ++i )
        acc[i][0] = acc[i][1] = T( 0 );
#pragma unroll
    for ( int w = 0; w < 2; ++w )
    {
        const Triangle< T >      G( P.table, N, d, x, y, w );
        const CoarseMoments< T > C( fine_lateral_wedge( x, y, w ) );
        const T                  sg = G.iD < T( 0 ) ? T( 1 ) : T( -1 );
        T                        S[2], wv[2][3];
#pragma unroll
        for ( int l = 0; l < 2; ++l )
        {
            const T *u0 = uu[w ? 3 : 0][l], *u1 = uu[w ? 2 : 1][l], *u2 = uu[w ? 1 : 2][l];
            const T  e1[3] = { u1[0] - u0[0], u1[1] - u0[1], u1[2] - u0[2] };
            const T  e2[3] = { u2[0] - u0[0], u2[1] - u0[1], u2[2] - u0[2] };
            wv[l][0] = dot3( G.v, u0 ), wv[l][1] = dot3( G.v, u1 ), wv[l][2] = dot3( G.v, u2 );
            S[l] = dot3( G.b1, e1 ) + dot3( G.b2, e2 ) + wv[l][0]; // sum_m beta_m . u_m
        }
#pragma unroll
        for ( int i = 0; i < 3; ++i )
        {
            const T qb = C.c1[i][0] * wv[0][0] + C.c1[i][1] * wv[0][1] + C.c1[i][2] * wv[0][2];
            const T qt = C.c1[i][0] * wv[1][0] + C.c1[i][1] * wv[1][1] + C.c1[i][2] * wv[1][2];
            const T fb = sg * ( C.c0[i] * S[0] - qb ), ft = sg * ( C.c0[i] * S[1] - qt ), fv = sg * T( 0.5 ) * ( qt - qb );
            const int col = i == 0 ? ( w ? 3 : 0 ) : ( w ? 3 - i : i );
            acc[col][0] += Ra[0][0] * fb + Ra[0][1] * ft + Rb[0] * fv;
            acc[col][1] += Ra[1][0] * fb + Ra[1][1] * ft + Rb[1] * fv;
        }
    }
    // the two fine cells r = 2 rc, 2 rc + 1 (lanes 2k, 2k + 1) add to the same coarse nodes; the upper ones go to
    // the next pair, which holds them as its lower ones
    unsigned coarse[4];
    cell_nodes( nc1, d, x >> 1, y >> 1, r >> 1, coarse );
    const bool from_below = lane > 1 && r > 1, own_top = lane >= 30 || r >= N - 2;
#pragma unroll
    for ( int i = 0; i < 4; ++i )
    {
        const T low   = acc[i][0] + __shfl_down_sync( 0xffffffffu, acc[i][0], 1 );
        const T high  = acc[i][1] + __shfl_down_sync( 0xffffffffu, acc[i][1], 1 );
        const T below = __shfl_up_sync( 0xffffffffu, high, 2 );
        if ( !in || ( lane & 1 ) )
            continue;
        T* o = p + coarse[i];
        atomicAdd( o, from_below ? low + below : low );
        if ( own_top )
            atomicAdd( o + 1, high );
    }
}

// u_fine += B^T p.  Boundary treatment acts on the lower nodes of r = 0 and the upper ones of r = N - 1, which only
// their own cell writes.
// Blocks per SM, level 6: FP64 at 3 / 4 / 6 blocks 144 / 127 / 131 us, FP32 at 4 / 5 / 6 97 / 97 / 91 us.
template < typename T >
__global__ void __launch_bounds__( 128, sizeof( T ) == 8 ? 4 : 6 ) gradient_kernel( StokesParams< T > P, const T* __restrict__ p, Ptr3< T > u )
{
    const int  N = P.N, n1 = P.n1, nc1 = P.nc1;
    int        d, x, y, r;
    const bool in = cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, N, d, x, y, r );
    T* const   dst[3] = { u.p[0], u.p[1], u.p[2] };
    T          Ra[2][2], Rb[2], pc[4][2];
    unsigned   node[4], coarse[4];
    cell_nodes( n1, d, x, y, r, node );
    cell_nodes( nc1, d, x >> 1, y >> 1, r >> 1, coarse );
    radial_sums( layer_h( P.table, N, r ), layer_r( P.table, N, r ), r & 1, Ra, Rb );
#pragma unroll
    for ( int i = 0; i < 4; ++i )
    {
        pc[i][0] = p[coarse[i]], pc[i][1] = p[coarse[i] + 1];
    }
    const int bc_low = r == 0 ? P.bc_cmb : 0, bc_high = r == N - 1 ? P.bc_surf : 0;
    const auto emit = [&]( int i, T( &low )[3], T( &high )[3] ) {
        const size_t lat = lat_index( n1, d, x + ( i & 1 ), y + ( i >> 1 ) );
        if ( bc_low == TN_BC_FREESLIP )
            project_tangential( P.coords + lat * 3, low );
        if ( bc_high == TN_BC_FREESLIP )
            project_tangential( P.coords + lat * 3, high );
        add_column< T, 3 >( dst, node[i], r, N, in, bc_low != TN_BC_DIRICHLET, bc_high != TN_BC_DIRICHLET, low, high );
    };
    T acc[2][2][3]; // columns 1 and 2 get both wedges
#pragma unroll
    for ( int w = 0; w < 2; ++w )
    {
        const Triangle< T >      G( P.table, N, d, x, y, w );
        const CoarseMoments< T > C( fine_lateral_wedge( x, y, w ) );
        const T                  sg = G.iD < T( 0 ) ? T( 1 ) : T( -1 );
        T                        A[2] = { T( 0 ), T( 0 ) }, B[2][3] = { { T( 0 ), T( 0 ), T( 0 ) }, { T( 0 ), T( 0 ), T( 0 ) } };
#pragma unroll
        for ( int i = 0; i < 3; ++i )
        {
            const int col = i == 0 ? ( w ? 3 : 0 ) : ( w ? 3 - i : i );
            const T   p0 = sg * pc[col][0], p1 = sg * pc[col][1];
            const T   prb = Ra[0][0] * p0 + Ra[1][0] * p1, prt = Ra[0][1] * p0 + Ra[1][1] * p1;
            const T   pl = T( 0.5 ) * ( Rb[0] * p0 + Rb[1] * p1 );
            A[0] += C.c0[i] * prb, A[1] += C.c0[i] * prt;
#pragma unroll
            for ( int m = 0; m < 3; ++m )
                B[0][m] -= C.c1[i][m] * ( prb + pl ), B[1][m] += C.c1[i][m] * ( pl - prt );
        }
#pragma unroll
        for ( int m = 0; m < 3; ++m )
        {
            T o[2][3];
#pragma unroll
            for ( int l = 0; l < 2; ++l )
#pragma unroll
                for ( int c = 0; c < 3; ++c )
                {
                    const T beta = m == 0 ? G.v[c] - G.b1[c] - G.b2[c] : ( m == 1 ? G.b1[c] : G.b2[c] );
                    o[l][c]      = A[l] * beta + B[l][m] * G.v[c];
                }
            if ( m == 0 )
                emit( w ? 3 : 0, o[0], o[1] );
            else if ( w == 0 )
            {
#pragma unroll
                for ( int c = 0; c < 3; ++c )
                    acc[m - 1][0][c] = o[0][c], acc[m - 1][1][c] = o[1][c];
            }
            else
            {
                const int a = 2 - m; // vertex m of wedge 1 is column 3 - m
#pragma unroll
                for ( int c = 0; c < 3; ++c )
                    o[0][c] += acc[a][0][c], o[1][c] += acc[a][1][c];
                emit( 3 - m, o[0], o[1] );
            }
        }
    }
}

int check_pair( const tn_mesh* f, const tn_mesh* c )
{
    TN_CHECK_ARG( f && c, "stokes block: null mesh" );
    TN_CHECK_ARG( c->level == f->level - 1 && c->r_min == f->r_min && c->r_max == f->r_max,
                  "stokes block: the pressure mesh must be the velocity mesh coarsened once" );
    // the B kernel pairs even and odd lanes: every warp must hold whole pairs of
    // radial cells (10 N^3 a multiple of 32 and N even, N >= 4)
    const long long N = f->N;
    TN_CHECK_ARG( N >= 4 && N % 2 == 0 && ( 10LL * N * N * N ) % 32 == 0,
                  "stokes block: the velocity mesh needs level >= 2 (whole radial columns per warp)" );
    return TN_OK;
}

}  // namespace

template < typename T >
int divergence_apply( const tn_mesh* f, const tn_mesh* c, int bc_cmb, int bc_surf, int apply_mode, int comm_mode,
                      const T* const* u, T* p, cudaStream_t st )
{
    int rc;
    if ( ( rc = check_pair( f, c ) ) )
        return rc;
    TN_CHECK_ARG( u && u[0] && u[1] && u[2] && p, "divergence: null vector" );
    if ( apply_mode == TN_APPLY_REPLACE )
        TN_CUDA_TRY( cudaMemsetAsync( p, 0, c->ns * sizeof( T ), st ) );
    StokesParams< T > P{ f->N, f->n1, c->n1, f->d_coords, triangle_table< T >( f ), bc_cmb, bc_surf };
    const long long cells = (long long) kDiamonds * f->N * f->N * f->N;
    divergence_kernel< T ><<< unsigned( ( cells + 127 ) / 128 ), 128, 0, st >>>( P, Ptr3< const T >{ { u[0], u[1], u[2] } }, p );
    TN_LAUNCH_CHECK();
    if ( comm_mode == TN_COMM_ADDITIVE )
    {
        T* fl[1] = { p };
        return halo_sum< T >( c, fl, 1, st );
    }
    return TN_OK;
}

template < typename T >
int gradient_apply( const tn_mesh* f, const tn_mesh* c, int bc_cmb, int bc_surf, int apply_mode, int comm_mode,
                    const T* p, T* const* u, cudaStream_t st )
{
    int rc;
    if ( ( rc = check_pair( f, c ) ) )
        return rc;
    TN_CHECK_ARG( u && u[0] && u[1] && u[2] && p, "gradient: null vector" );
    if ( apply_mode == TN_APPLY_REPLACE )
        TN_CUDA_TRY( zero_fields( u, 3, f->ns, st ) );
    StokesParams< T > P{ f->N, f->n1, c->n1, f->d_coords, triangle_table< T >( f ), bc_cmb, bc_surf };
    const long long cells = (long long) kDiamonds * f->N * f->N * f->N;
    gradient_kernel< T ><<< unsigned( ( cells + 127 ) / 128 ), 128, 0, st >>>( P, p, Ptr3< T >{ { u[0], u[1], u[2] } } );
    TN_LAUNCH_CHECK();
    if ( comm_mode == TN_COMM_ADDITIVE )
        return halo_sum< T >( f, u, 3, st );
    return TN_OK;
}

template int divergence_apply< double >( const tn_mesh*, const tn_mesh*, int, int, int, int, const double* const*,
                                         double*, cudaStream_t );
template int divergence_apply< float >( const tn_mesh*, const tn_mesh*, int, int, int, int, const float* const*,
                                        float*, cudaStream_t );
template int gradient_apply< double >( const tn_mesh*, const tn_mesh*, int, int, int, int, const double*,
                                       double* const*, cudaStream_t );
template int gradient_apply< float >( const tn_mesh*, const tn_mesh*, int, int, int, int, const float*, float* const*,
                                      cudaStream_t );

}  // namespace tn

using namespace tn;

extern "C" int tn_divergence_apply_f64( const tn_mesh* f, const tn_mesh* c, int bcc, int bcs, int am, int cm,
                                        const double* const* u, double* p, void* s )
{
    return divergence_apply< double >( f, c, bcc, bcs, am, cm, u, p, as_stream( s ) );
}
extern "C" int tn_divergence_apply_f32( const tn_mesh* f, const tn_mesh* c, int bcc, int bcs, int am, int cm,
                                        const float* const* u, float* p, void* s )
{
    return divergence_apply< float >( f, c, bcc, bcs, am, cm, u, p, as_stream( s ) );
}
extern "C" int tn_gradient_apply_f64( const tn_mesh* f, const tn_mesh* c, int bcc, int bcs, int am, int cm,
                                      const double* p, double* const* u, void* s )
{
    return gradient_apply< double >( f, c, bcc, bcs, am, cm, p, u, as_stream( s ) );
}
extern "C" int tn_gradient_apply_f32( const tn_mesh* f, const tn_mesh* c, int bcc, int bcs, int am, int cm,
                                      const float* p, float* const* u, void* s )
{
    return gradient_apply< float >( f, c, bcc, bcs, am, cm, p, u, as_stream( s ) );
}
