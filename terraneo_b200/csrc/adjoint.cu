// Viscosity derivative of the epsilon-div-div form (the backward kernel of
// the adjoint viscosity gradient; no reference counterpart).
//
// The one-point kerngen operator (fe/wedge/operators/shell/
// epsilon_divdiv_kerngen.hpp:1055-1940) is linear in the nodal coefficient:
// every wedge uses k_eval = (1/6) sum of its six nodal k, so
//     d(lambda^T A(k) u) / d k_n = sum over wedges w containing n of c_w / 6,
//     c_w = lambda_w^T A_w(k = 1) u_w,
// with A_w the wedge's 18x18 action including the boundary treatment:
// Dirichlet nodes leave the coupling and keep their diagonal
// |det J| (|g_n|^2 + g_{n,c}^2 / 3); free-slip nodes enter projected on the
// tangent plane on both sides and add |det J| (|g_n|^2 + (n.g_n)^2 / 3)
// (n.u)(n.lambda).  The rigid-rotation penalty does not depend on k and
// does not enter.  In the interior c_w = |det J| (2 E(u):E(lambda) -
// 2/3 div u div lambda) at the single quadrature point.
//
// One thread per cell (r fastest).  In the factored form of cell.cuh the scaled
// gradient matrix at the centroid is beta_1 (x) S_1 + beta_2 (x) S_2 + v (x) Z with
// edge differences S_i and Z = rho T - (S_1 + S_2) / 3, so a wedge needs no
// Jacobian: about 120 multiply-adds for both fields.  The cell's node sums go out
// by add_column.  Cells of a boundary layer with a condition are left to the first
// blocks of the launch (one thread per lateral cell, wedge and side), which add the boundary
// terms: with the lanes along r, every warp would otherwise carry that code for
// one lane.  Level-6 free-slip FP64: 612 -> 127 us, FP32 276 -> 87 us.
// Without communication the result is the derivative with respect to each
// stored copy of k (each diamond's wedges use their own copy); with the
// additive halo it is the derivative with respect to the unique node's value,
// stored on all of its copies.
#include "cell.cuh"
#include "common.cuh"
#include "wedge.cuh"

namespace tn {

template < typename T >
int halo_sum( const tn_mesh* m, T* const* fields, int nfields, cudaStream_t st );

namespace {

template < typename T >
struct KGradParams
{
    int             N, n1;
    const double*   coords; // lateral points (unit vectors: the outward normals)
    const T*        table;
    Ptr3< const T > u, lam;
    T*              out;
    int             bc_cmb, bc_surf;
    unsigned        edge_blocks; // blocks of boundary cells, before those of all cells
};

// scaled gradient matrix (times 3: the weights 1/3 of the centroid, whose rounding every wedge would share, are left to
// the one factor 1/54 at the end) of the node values s of a wedge at its centroid
template < typename T >
__device__ __forceinline__ void centroid_gradient( const Triangle< T >& G, T rho, const T ( &s )[6][3], T ( &M )[3][3] )
{
#pragma unroll
    for ( int c = 0; c < 3; ++c )
    {
        const T S1 = T( 0.5 ) * ( ( s[1][c] - s[0][c] ) + ( s[4][c] - s[3][c] ) );
        const T S2 = T( 0.5 ) * ( ( s[2][c] - s[0][c] ) + ( s[5][c] - s[3][c] ) );
        const T t  = ( s[3][c] - s[0][c] ) + ( s[4][c] - s[1][c] ) + ( s[5][c] - s[2][c] );
        const T Z = T( 0.5 ) * rho * t - S1 - S2, S13 = T( 3 ) * S1, S23 = T( 3 ) * S2;
#pragma unroll
        for ( int a = 0; a < 3; ++a )
            M[a][c] = G.b1[a] * S13 + G.b2[a] * S23 + G.v[a] * Z;
    }
}

// 2 E(u) : E(l) - 2/3 div u div l of two gradient matrices
template < typename T >
__device__ __forceinline__ T strain_product( const T ( &A )[3][3], const T ( &B )[3][3] )
{
    const T tr = ( A[0][0] + A[1][1] + A[2][2] ) * ( B[0][0] + B[1][1] + B[2][2] );
    return T( 2 ) * ( A[0][0] * B[0][0] + A[1][1] * B[1][1] + A[2][2] * B[2][2] ) +
           ( A[0][1] + A[1][0] ) * ( B[0][1] + B[1][0] ) + ( A[0][2] + A[2][0] ) * ( B[0][2] + B[2][0] ) +
           ( A[1][2] + A[2][1] ) * ( B[1][2] + B[2][1] ) - T( 2.0 / 3.0 ) * tr;
}

// the values of field f at the nodes of a wedge (id: wedge_columns)
template < typename T >
__device__ __forceinline__ void wedge_values( const Ptr3< const T >& f, const unsigned ( &id )[3], T ( &v )[6][3] )
{
#pragma unroll
    for ( int n = 0; n < 6; ++n )
#pragma unroll
        for ( int a = 0; a < 3; ++a )
            v[n][a] = f.p[a][id[n % 3] + n / 3];
}

// Takes the boundary condition bc out of the values v of a wedge's boundary side (top: nodes 3..5): Dirichlet values
// are zeroed, free-slip ones projected.  b[m][.]: what was taken out, all three components or (b[m][0]) the normal one.
template < typename T >
__device__ __forceinline__ void split_boundary( const T ( &nn )[3][3], int bc, bool top, T ( &v )[6][3], T ( &b )[3][3] )
{
#pragma unroll
    for ( int m = 0; m < 3; ++m )
    {
        T s[3], t[3];
#pragma unroll
        for ( int a = 0; a < 3; ++a )
            s[a] = top ? v[3 + m][a] : v[m][a];
        const T un = dot3( nn[m], s );
#pragma unroll
        for ( int a = 0; a < 3; ++a )
        {
            t[a]    = bc == TN_BC_DIRICHLET ? T( 0 ) : s[a] - un * nn[m][a];
            b[m][a] = bc == TN_BC_DIRICHLET ? s[a] : un;
            if ( top )
                v[3 + m][a] = t[a];
            else
                v[m][a] = t[a];
        }
    }
}

// Cells of the layers with a boundary condition (the first edge_blocks blocks): one thread per lateral cell, wedge and
// side.  A cell has a condition on one side (N > 1).
template < typename T >
__device__ __forceinline__ void kgrad_boundary( const KGradParams< T >& P )
{
    int  d, x, y, r, w;
    bool top;
    if ( !boundary_item( blockIdx.x * blockDim.x + threadIdx.x, P.N, d, x, y, r, w, top ) )
        return;
    const int bc = top ? P.bc_surf : P.bc_cmb;
    if ( bc == 0 )
        return;
    const Triangle< T > G( P.table, P.N, d, x, y, w );
    const T             h = layer_h( P.table, P.N, r ), rho = layer_q( P.table, P.N, r ) + T( 1 );
    unsigned            node[4], id[3];
    T                   nn[3][3], v[6][3], A[3][3], B[3][3], ub[3][3], lb[3][3], bnd = T( 0 );
    cell_nodes( P.n1, d, x, y, r, node );
    wedge_columns( node, w, id );
#pragma unroll
    for ( int m = 0; m < 3; ++m )
#pragma unroll
        for ( int a = 0; a < 3; ++a )
            nn[m][a] = T( P.coords[size_t( ( id[m] - unsigned( r ) ) / unsigned( P.n1 ) ) * 3 + a] );
    wedge_values( P.u, id, v );
    split_boundary( nn, bc, top, v, ub );
    centroid_gradient( G, rho, v, A );
    wedge_values( P.lam, id, v );
    split_boundary( nn, bc, top, v, lb );
    centroid_gradient( G, rho, v, B );
#pragma unroll
    for ( int m = 0; m < 3; ++m )
    {
        T g[3];
        scaled_gradient( G, m, top ? T( 1 ) : T( -1 ), T( 1.0 / 3.0 ), T( 1.0 / 3.0 ), T( 0 ), rho, g );
        const T gg = dot3( g, g );
        if ( bc == TN_BC_DIRICHLET )
        {
#pragma unroll
            for ( int a = 0; a < 3; ++a )
                bnd += lb[m][a] * ub[m][a] * ( gg + g[a] * g[a] * T( 1.0 / 3.0 ) );
        }
        else
        {
            const T ng = dot3( nn[m], g );
            bnd += ( gg + ng * ng * T( 1.0 / 3.0 ) ) * ub[m][0] * lb[m][0];
        }
    }
    const T cw = h * fabs( G.iD ) * ( strain_product( A, B ) + T( 9 ) * bnd ) * T( 1.0 / 54.0 );
#pragma unroll
    for ( int n = 0; n < 6; ++n )
        atomicAdd( P.out + id[n % 3] + n / 3, cw );
}

// Blocks per SM, level 6: FP64 at 3 / 4 / 5 blocks 128 / 134 / 155 us, FP32 at 4 / 6 89 / 86 us.
template < typename T >
__global__ void __launch_bounds__( 128, sizeof( T ) == 8 ? 3 : 6 ) kgrad_kernel( KGradParams< T > P )
{
    if ( blockIdx.x < P.edge_blocks )
    {
        kgrad_boundary( P );
        return;
    }
    const int  N = P.N, n1 = P.n1;
    int        d, x, y, r;
    const bool in = cell_of( ( blockIdx.x - P.edge_blocks ) * (long long) blockDim.x + threadIdx.x, N, d, x, y, r );
    const T    h = layer_h( P.table, N, r ), rho = layer_q( P.table, N, r ) + T( 1 );
    unsigned   node[4];
    T          cw[2];
    cell_nodes( n1, d, x, y, r, node );
#pragma unroll
    for ( int w = 0; w < 2; ++w )
    {
        const Triangle< T > G( P.table, N, d, x, y, w );
        T                   v[6][3], A[3][3], B[3][3];
        unsigned            id[3];
        wedge_columns( node, w, id );
        wedge_values( P.u, id, v );
        centroid_gradient( G, rho, v, A );
        wedge_values( P.lam, id, v );
        centroid_gradient( G, rho, v, B );
        cw[w] = h * fabs( G.iD ) * strain_product( A, B ) * T( 1.0 / 54.0 );
    }
    if ( ( r == 0 && P.bc_cmb ) || ( r == N - 1 && P.bc_surf ) ) // a boundary cell: kgrad_boundary's
        cw[0] = cw[1] = T( 0 );
    T* const out[1] = { P.out };
#pragma unroll
    for ( int i = 0; i < 4; ++i )
    {
        const T v[1] = { i == 0 ? cw[0] : ( i == 3 ? cw[1] : cw[0] + cw[1] ) };
        add_column< T, 1 >( out, node[i], r, N, in, true, true, v, v );
    }
}

}  // namespace

template < typename T >
int epsdivdiv_kgrad( const tn_mesh* m, int bc_cmb, int bc_surf, int comm_mode, const T* const* u, const T* const* lam,
                     T* out, cudaStream_t st )
{
    TN_CHECK_ARG( m && u && lam && out, "epsdivdiv_kgrad: null argument" );
    TN_CHECK_ARG( bc_cmb >= 0 && bc_cmb <= 2 && bc_surf >= 0 && bc_surf <= 2, "epsdivdiv_kgrad: bad boundary code" );
    KGradParams< T > P{};
    for ( int c = 0; c < 3; ++c )
    {
        TN_CHECK_ARG( u[c] && lam[c], "epsdivdiv_kgrad: null field pointer" );
        P.u.p[c]   = u[c];
        P.lam.p[c] = lam[c];
    }
    P.N = m->N, P.n1 = m->n1, P.coords = m->d_coords, P.out = out, P.bc_cmb = bc_cmb, P.bc_surf = bc_surf;
    P.table = triangle_table< T >( m );
    TN_CUDA_TRY( cudaMemsetAsync( out, 0, m->ns * sizeof( T ), st ) );
    const long long cells = (long long) kDiamonds * m->N * m->N * m->N;
    P.edge_blocks = bc_cmb || bc_surf ? ( boundary_items( m->N ) + 127u ) / 128u : 0u;
    kgrad_kernel< T ><<< P.edge_blocks + unsigned( ( cells + 127 ) / 128 ), 128, 0, st >>>( P );
    TN_LAUNCH_CHECK();
    if ( comm_mode != TN_COMM_ADDITIVE )
        return TN_OK;
    T* f[1] = { out };
    return halo_sum< T >( m, f, 1, st );
}

template int epsdivdiv_kgrad< double >( const tn_mesh*, int, int, int, const double* const*, const double* const*,
                                        double*, cudaStream_t );

}  // namespace tn

using namespace tn;

extern "C" int tn_epsdivdiv_kgrad_f64( const tn_mesh* m, int bc_cmb, int bc_surface, int comm_mode,
                                       const double* const* u, const double* const* lambda, double* grad_k, void* s )
{
    return epsdivdiv_kgrad< double >( m, bc_cmb, bc_surface, comm_mode, u, lambda, grad_k, as_stream( s ) );
}
extern "C" int tn_epsdivdiv_kgrad_f32( const tn_mesh* m, int bc_cmb, int bc_surface, int comm_mode,
                                       const float* const* u, const float* const* lambda, float* grad_k, void* s )
{
    return epsdivdiv_kgrad< float >( m, bc_cmb, bc_surface, comm_mode, u, lambda, grad_k, as_stream( s ) );
}
