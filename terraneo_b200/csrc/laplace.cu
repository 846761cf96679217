// The gradient-form operators: Laplace (fe/wedge/operators/shell/laplace.hpp),
// DivKGrad (div_k_grad.hpp) and VectorLaplace (vector_laplace.hpp).
//
// int k grad u . grad v with the 3x2 Felippa rule (or the 1-point rule for
// DivKGrad's single-quadpoint mode) and the curved radial map; k = 1 for
// Laplace and VectorLaplace, k interpolated by the wedge shape functions at
// each quadrature point for DivKGrad; three independent components for
// VectorLaplace.  Boundary layers decouple their boundary nodes and keep the
// diagonal, as selected per operator below.
#include <cmath>

#include "cell.cuh"
#include "common.cuh"
#include "lateral_cg.cuh"
#include "wedge.cuh"

namespace tn {

namespace {

template < typename T >
struct DivKGradParams
{
    int      N, n1;
    const T* table;
    const T* k; // nodal coefficient
    const T* src;
    T*       dst;
    int      treat, single;
    unsigned cell_blocks; // blocks of cells; those after them add diagonals
};

// One wedge of DivKGrad from the values s of its nodes and k there; out[n] = its
// row of node n.  In the factored form of cell.cuh the scaled gradient of u is
// beta_1 S_1 + beta_2 S_2 + v Z with edge differences S_i that depend on zeta only
// and Z = rho T - xi S_1 - eta S_2, so a point needs Z and its product with v,
// and the rows follow from the zeta's summed flux against beta_1, beta_2 and the
// moments of (flux . v) over the points, all through the six scalar products of
// beta_1, beta_2, v: about 150 multiply-adds per wedge (470 when the symmetric
// 6 x 6 matrix is formed from a table of 63 lateral factors per wedge).
// Apply with its halo, FP64: 330 -> 91 us at level 6, 2,562 -> 642 us at level 7;
// bound by instruction issue (56 % of the slots).
template < typename T, bool SINGLE >
__device__ __forceinline__ void divkgrad_wedge( const Triangle< T >& G, T h, T rho_m, const T ( &s )[6], const T ( &kn )[6],
                                                T ( &out )[6] )
{
    const T b11 = dot3( G.b1, G.b1 ), b12 = dot3( G.b1, G.b2 ), b22 = dot3( G.b2, G.b2 );
    const T a1 = dot3( G.b1, G.v ), a2 = dot3( G.b2, G.v ), vv = dot3( G.v, G.v );
    const T t[3] = { T( 0.5 ) * ( s[3] - s[0] ), T( 0.5 ) * ( s[4] - s[1] ), T( 0.5 ) * ( s[5] - s[2] ) };
    const T e1b = s[1] - s[0], e2b = s[2] - s[0], e1t = s[4] - s[3], e2t = s[5] - s[3];
    T       L[3] = { T( 0 ), T( 0 ), T( 0 ) };
#pragma unroll
    for ( int n = 0; n < 6; ++n )
        out[n] = T( 0 );
    if ( SINGLE )
    {
        // quad_felippa_1x1: (1/3, 1/3, 0), weight 1; k at the centroid is the mean of the six
        const T w  = ( kn[0] + kn[1] + kn[2] + kn[3] + kn[4] + kn[5] ) * T( 1.0 / 6.0 ) * h * fabs( G.iD );
        const T S1 = T( 0.5 ) * ( e1b + e1t ), S2 = T( 0.5 ) * ( e2b + e2t );
        const T Z  = ( rho_m * ( t[0] + t[1] + t[2] ) - S1 - S2 ) * T( 1.0 / 3.0 );
        const T x  = w * ( a1 * S1 + a2 * S2 + vv * Z ) * T( 1.0 / 3.0 );
        const T f1 = w * ( b11 * S1 + b12 * S2 + a1 * Z ) - x, f2 = w * ( b12 * S1 + b22 * S2 + a2 * Z ) - x;
        out[0] = out[3] = T( -0.5 ) * ( f1 + f2 ), out[1] = out[4] = T( 0.5 ) * f1, out[2] = out[5] = T( 0.5 ) * f2;
        L[0] = L[1] = L[2] = rho_m * x;
    }
    else
    {
        // omega = k h / (6 |D|) at the lateral points, bottom and top: k there is (the sum + 3 the near vertex) / 6, and both
        // sixths are one rounded factor
        const T scale = T( 1.0 / 36.0 ) * h * fabs( G.iD );
        const T sb = kn[0] + kn[1] + kn[2], st = kn[3] + kn[4] + kn[5];
        const T ts = ( t[0] + t[1] + t[2] ) * T( 1.0 / 6.0 );
#pragma unroll
        for ( int zq = 0; zq < 2; ++zq )
        {
            const T nb = T( zq ? 0.5 * ( 1.0 - kFelippaZ ) : 0.5 * ( 1.0 + kFelippaZ ) );
            const T nt = T( zq ? 0.5 * ( 1.0 + kFelippaZ ) : 0.5 * ( 1.0 - kFelippaZ ) );
            const T rho = rho_m + T( zq ? kFelippaZ : -kFelippaZ );
            const T S1 = nb * e1b + nt * e1t, S2 = nb * e2b + nt * e2t;
            const T Z0 = rho * ts - T( 1.0 / 6.0 ) * ( S1 + S2 ), pv = a1 * S1 + a2 * S2;
            T       om = T( 0 ), Zs = T( 0 ), ev[2];
#pragma unroll
            for ( int q = 0; q < 3; ++q )
            {
                const int m = ( q + 1 ) % 3; // point q lies next to vertex m
                const T   w = scale * ( nb * ( sb + T( 3 ) * kn[m] ) + nt * ( st + T( 3 ) * kn[3 + m] ) );
                const T   Z = Z0 + T( 0.5 ) * ( q == 0 ? rho * t[1] - S1 : ( q == 1 ? rho * t[2] - S2 : rho * t[0] ) );
                om += w;
                Zs += w * Z;
                if ( q < 2 )
                    ev[q] = w * ( pv + vv * Z );
            }
            // flux . v summed over the points and its moments with xi and eta
            const T V = om * pv + vv * Zs, X = T( 1.0 / 6.0 ) * V + T( 0.5 ) * ev[0], Y = T( 1.0 / 6.0 ) * V + T( 0.5 ) * ev[1];
            const T f1 = om * ( b11 * S1 + b12 * S2 ) + a1 * Zs - X, f2 = om * ( b12 * S1 + b22 * S2 ) + a2 * Zs - Y;
            const T f0 = -( f1 + f2 );
            out[0] += nb * f0, out[1] += nb * f1, out[2] += nb * f2;
            out[3] += nt * f0, out[4] += nt * f1, out[5] += nt * f2;
            L[0] += rho * ( V - X - Y ), L[1] += rho * X, L[2] += rho * Y;
        }
    }
#pragma unroll
    for ( int m = 0; m < 3; ++m )
        out[m] -= T( 0.5 ) * L[m], out[3 + m] += T( 0.5 ) * L[m];
}

// adds the diagonal entries of the three lower (top false) or upper nodes of a wedge times their values
template < typename T >
__device__ __forceinline__ void divkgrad_diagonal( const DivKGradParams< T >& P, int d, int x, int y, int r, int w, bool top )
{
    const T             h = layer_h( P.table, P.N, r ), rq = layer_q( P.table, P.N, r ), side = top ? T( 1 ) : T( -1 );
    const Triangle< T > G( P.table, P.N, d, x, y, w );
    unsigned            node[4], id[3];
    T                   kn[6], o[3] = { T( 0 ), T( 0 ), T( 0 ) };
    cell_nodes( P.n1, d, x, y, r, node );
    wedge_columns( node, w, id );
#pragma unroll
    for ( int n = 0; n < 6; ++n )
        kn[n] = P.k[id[n % 3] + n / 3];
    for ( int q = 0; q < ( P.single ? 1 : 6 ); ++q )
    {
        const T xi = P.single ? T( 1.0 / 3.0 ) : T( felippa_xi( q ) ), eta = P.single ? T( 1.0 / 3.0 ) : T( felippa_eta( q ) );
        const T zeta   = P.single ? T( 0 ) : T( q < 3 ? -kFelippaZ : kFelippaZ );
        const T lat[3] = { T( 1 ) - xi - eta, xi, eta };
        T       k      = T( 0 );
#pragma unroll
        for ( int n = 0; n < 6; ++n )
            k += lat[n % 3] * T( 0.5 ) * ( n < 3 ? T( 1 ) - zeta : T( 1 ) + zeta ) * kn[n];
        const T om = ( P.single ? T( 1 ) : T( kFelippaW ) ) * k * h * fabs( G.iD ), rho = rq + T( 1 ) + zeta;
#pragma unroll
        for ( int m = 0; m < 3; ++m )
        {
            T g[3];
            scaled_gradient( G, m, side, xi, eta, zeta, rho, g );
            o[m] += om * dot3( g, g );
        }
    }
#pragma unroll
    for ( int m = 0; m < 3; ++m )
        atomicAdd( P.dst + id[m] + top, o[m] * P.src[id[m] + top] );
}

// One thread per cell (r fastest), contributions added by add_column.  With the
// boundary treatment the CMB nodes of layer 0 (otherwise the SURFACE nodes of
// layer N - 1) enter with zero and keep their diagonal, which further blocks of the
// launch add (one thread per lateral cell, wedge and side).  Blocks per SM, FP64: at 4 / 5 / 6 95 / 91 / 97 us at
// level 6, 689 / 642 / 670 us at level 7; FP32 takes 70 registers whatever the bound (seven blocks).
template < typename T, bool SINGLE >
__global__ void __launch_bounds__( 128, 5 ) divkgrad_kernel( DivKGradParams< T > P )
{
    const int N = P.N, n1 = P.n1;
    int       d, x, y, r;
    if ( blockIdx.x >= P.cell_blocks )
    {
        int  w;
        bool top;
        if ( boundary_item( ( blockIdx.x - P.cell_blocks ) * blockDim.x + threadIdx.x, N, d, x, y, r, w, top ) )
            divkgrad_diagonal( P, d, x, y, r, w, top );
        return;
    }
    const bool in  = cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, N, d, x, y, r );
    const bool bot = P.treat && r == 0, top = P.treat && !bot && r == N - 1;
    const T    h = layer_h( P.table, N, r ), rho_m = layer_q( P.table, N, r ) + T( 1 );
    T* const   dst[1] = { P.dst };
    unsigned   node[4];
    T          s[4][2], k[4][2], acc[2][2];
    cell_nodes( n1, d, x, y, r, node );
#pragma unroll
    for ( int i = 0; i < 4; ++i )
    {
#pragma unroll
        for ( int l = 0; l < 2; ++l )
        {
            const T v = P.src[node[i] + l];
            s[i][l]   = ( l ? top : bot ) ? T( 0 ) : v;
            k[i][l]   = P.k[node[i] + l];
        }
    }
#pragma unroll
    for ( int w = 0; w < 2; ++w )
    {
        const Triangle< T > G( P.table, N, d, x, y, w );
        T                   sw[6], kw[6], out[6];
#pragma unroll
        for ( int n = 0; n < 6; ++n )
        {
            const int i = wedge_node( w, n, 0 ) + 2 * wedge_node( w, n, 1 );
            sw[n] = s[i][n / 3], kw[n] = k[i][n / 3];
        }
        divkgrad_wedge< T, SINGLE >( G, h, rho_m, sw, kw, out );
        const T low0[1] = { out[0] }, high0[1] = { out[3] };
        add_column< T, 1 >( dst, node[w ? 3 : 0], r, N, in, !bot, !top, low0, high0 );
#pragma unroll
        for ( int m = 1; m < 3; ++m )
        {
            const int a = w ? 2 - m : m - 1; // vertex m of wedge 0 is vertex 3 - m of wedge 1
            if ( w == 0 )
                acc[a][0] = out[m], acc[a][1] = out[3 + m];
            else
            {
                const T low[1] = { acc[a][0] + out[m] }, high[1] = { acc[a][1] + out[3 + m] };
                add_column< T, 1 >( dst, node[3 - m], r, N, in, !bot, !top, low, high );
            }
        }
    }
}

// the diagonal alone: one thread per cell, wedge and side (blockIdx.y)
template < typename T >
__global__ void __launch_bounds__( 128 ) divkgrad_diagonal_kernel( DivKGradParams< T > P )
{
    int d, x, y, r;
    if ( cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, P.N, d, x, y, r ) )
        divkgrad_diagonal( P, d, x, y, r, int( blockIdx.y & 1 ), blockIdx.y >= 2 );
}

// The lateral factors of a triangle at a lateral point with sig = 1 / |D|: u[3] and lat[3] (factored stiffness
// above); v = a x b.
struct LateralTriangle
{
    double a[3], b[3], v[3], p0[3], sig;
    __host__ __device__ LateralTriangle( const double* q0, const double* q1, const double* q2 )
    {
        for ( int k = 0; k < 3; ++k )
            p0[k] = q0[k], a[k] = q1[k] - q0[k], b[k] = q2[k] - q0[k];
        cross( a, b, v );
        sig = 1.0 / fabs( dot( v, p0 ) );
    }
    __host__ __device__ void at( double xi, double eta, double u[3][3], double lat[3] ) const
    {
        double c[3];
        for ( int k = 0; k < 3; ++k )
            c[k] = p0[k] + xi * a[k] + eta * b[k];
        cross( b, c, u[1] );
        cross( c, a, u[2] );
        for ( int k = 0; k < 3; ++k )
            u[0][k] = -( u[1][k] + u[2][k] );
        lat[0] = 1.0 - xi - eta, lat[1] = xi, lat[2] = eta;
    }
    static __host__ __device__ void cross( const double* x, const double* y, double* o )
    {
        o[0] = x[1] * y[2] - x[2] * y[1];
        o[1] = x[2] * y[0] - x[0] * y[2];
        o[2] = x[0] * y[1] - x[1] * y[0];
    }
    static __host__ __device__ double dot( const double* x, const double* y ) { return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]; }
};

// A layer's two rows of the Laplacian from the lateral sums of its levels with
// the stencils U, W^T (per level; rows sum to zero because sum_m u_m = 0) and
// Lam, W (on the difference of the levels), all summed over the 3x2 rule's
// lateral points with weight 1/6, and its radial factors R[0] = R[2], R[1],
// S2 / 4, P[0] / 2, P[1] / 2 (R = h sum nr nr, S2 = sum r^2 / h, P = sum r nr),
// both rows sharing the differences.
// Apply with its halo, FP64, before (one thread per cell, atomics) and now:
// Laplace 112 -> 33 us at level 6, 911 -> 226 us at level 7 (1.5 TB/s of its
// 16 bytes per node); VectorLaplace 228 -> 99 us at level 6; FP32 Laplace
// 84 -> 25 us at level 6.
template < typename T >
struct LaplaceOp
{
    static constexpr int           S = 2, D = 2, K = S + D, R = 5;
    static constexpr bool          kDiff = true;
    static constexpr bool          kExactDot = false; // <p, A p> summed as tn_pcg_pap sums it
    static __device__ __forceinline__ void layer( const T ( &f )[R], const T ( &b )[S], const T ( &t )[S], const T ( &d )[D + 1],
                                                  T& low, T& high )
    {
        const T x = f[2] * d[0], e = f[3] * b[1] + f[4] * t[1];
        low  = f[0] * b[0] + f[1] * t[0] - x + f[3] * d[1] - e;
        high = f[0] * t[0] + f[1] * b[0] + x + f[4] * d[1] + e;
    }
    static __device__ __forceinline__ T side_low( const T ( &f )[R], const T ( &s )[S], const T ( &v )[D + 1] )
    {
        return f[0] * s[0] + f[2] * v[0] - f[3] * ( v[1] + s[1] );
    }
    static __device__ __forceinline__ T side_high( const T ( &f )[R], const T ( &s )[S], const T ( &v )[D + 1] )
    {
        return f[0] * s[0] + f[2] * v[0] + f[4] * ( v[1] + s[1] );
    }
    static __device__ __forceinline__ T self_low( const T ( &f )[R], const T ( &v )[K] )
    {
        return f[0] * v[0] + f[2] * v[2] - f[3] * ( v[3] + v[1] );
    }
    static __device__ __forceinline__ T self_high( const T ( &f )[R], const T ( &v )[K] )
    {
        return f[0] * v[0] + f[2] * v[2] + f[4] * ( v[3] + v[1] );
    }
    using Sum = double;
    static __device__ double entry( double a, int ) { return a; }
    static __device__ void triangle( const double* p0, const double* p1, const double* p2, int i, const int ( &e )[3],
                                     double ( &A )[kStencil][K] )
    {
        const LateralTriangle tri( p0, p1, p2 );
        const double          vv = LateralTriangle::dot( tri.v, tri.v ), f = kFelippaW * tri.sig;
#pragma unroll
        for ( int q = 0; q < 3; ++q )
        {
            double u[3][3], l[3];
            tri.at( felippa_xi( q ), felippa_eta( q ), u, l );
#pragma unroll
            for ( int j = 0; j < 3; ++j )
            {
                double* a = A[e[j]];
                a[0] += f * LateralTriangle::dot( u[i], u[j] );
                a[1] += f * LateralTriangle::dot( u[j], tri.v ) * l[i];
                a[2] += f * l[i] * l[j] * vv;
                a[3] += f * LateralTriangle::dot( u[i], tri.v ) * l[j];
            }
        }
    }
    static __device__ void radial( double r1, double r2, double* f )
    {
        const double h = 0.5 * ( r2 - r1 );
        for ( int k = 0; k < R; ++k )
            f[k] = 0.0;
        for ( int zq = 0; zq < 2; ++zq )
        {
            const double zeta = zq ? kFelippaZ : -kFelippaZ, nb = 0.5 * ( 1.0 - zeta ), nt = 0.5 * ( 1.0 + zeta );
            const double rr   = r1 + h * ( 1.0 + zeta );
            f[0] += h * nb * nb, f[1] += h * nb * nt, f[2] += 0.25 * rr * rr / h;
            f[3] += 0.5 * rr * nb, f[4] += 0.5 * rr * nt;
        }
    }
};

}  // namespace

// Laplace / VectorLaplace driver (lateral.cuh).
template < typename T >
int constant_gradient_apply( const tn_mesh* m, int nc, const T* const* src, T* const* dst, int mode_first, int mode_inner,
                             int mode_last, int apply_mode, int comm_mode, cudaStream_t st, const char* what )
{
    TN_CHECK_ARG( m && src && dst, std::string( what ) + ": null argument" );
    TN_CHECK_ARG( apply_mode == TN_APPLY_REPLACE || apply_mode == TN_APPLY_ADD, std::string( what ) + ": bad apply mode" );
    LateralParams< T > P{};
    for ( int c = 0; c < nc; ++c )
    {
        TN_CHECK_ARG( src[c] && dst[c], std::string( what ) + ": null field pointer" );
        P.src.p[c] = src[c];
        P.dst.p[c] = dst[c];
    }
    if ( !lateral_tables< LaplaceOp< T > >( m, &tn_mesh::laplace_tables, P ) )
    {
        set_error( std::string( what ) + ": allocating the lateral stencils failed" );
        return TN_ERR_NOMEM;
    }
    P.mode_first = mode_first, P.mode_inner = mode_inner, P.mode_last = mode_last;
    return launch_lateral< LaplaceOp< T > >( m, P, nc, apply_mode, comm_mode, st );
}

// Laplace / DivKGrad coupling (laplace.hpp:140-168, div_k_grad.hpp:455-512):
// with treat_boundary the first layer decouples its CMB nodes, the last one
// (unless it is also the first) its SURFACE nodes; diagonal mode keeps only
// the diagonal everywhere.
static void scalar_modes( int N, int treat, int diag, int& first, int& inner, int& last )
{
    inner = diag ? kDiag : kNeu;
    first = diag ? kDiag : ( treat ? kBot : kNeu );
    last  = diag ? kDiag : ( treat ? ( N == 1 ? kBot : kTop ) : kNeu );
}

template < typename T >
int laplace_apply( const tn_mesh* m, int treat, int diag, int apply_mode, int comm_mode, const T* src, T* dst,
                   cudaStream_t st )
{
    TN_CHECK_ARG( m && src && dst, "laplace_apply: null argument" );
    int f, i, l;
    scalar_modes( m->N, treat, diag, f, i, l );
    const T* s[1] = { src };
    T*       d[1] = { dst };
    return constant_gradient_apply< T >( m, 1, s, d, f, i, l, apply_mode, comm_mode, st, "laplace_apply" );
}

// CG on Laplace(treat_boundary) from x's values (lateral_cg.cuh)
int laplace_cg( const tn_mesh* m, const double* b, double* x, int max_iterations, double rtol, double atol, int* iterations,
                double* relres, cudaStream_t st )
{
    LateralParams< double > P{};
    if ( !lateral_tables< LaplaceOp< double > >( m, &tn_mesh::laplace_tables, P ) )
    {
        set_error( "laplace_cg: allocating the lateral stencils failed" );
        return TN_ERR_NOMEM;
    }
    scalar_modes( m->N, 1, 0, P.mode_first, P.mode_inner, P.mode_last );
    const size_t    ns = m->ns;
    const WorkBlock w( m, 4 * ns + lateral_cg_scratch< LaplaceOp< double > >( m, max_iterations ) );
    if ( !w.get() )
    {
        set_error( "laplace_cg: allocating the work fields failed" );
        return TN_ERR_NOMEM;
    }
    double* const fields[4] = { w.get(), w.get() + ns, w.get() + 2 * ns, w.get() + 3 * ns };
    return lateral_cg< LaplaceOp< double > >( m, P, b, x, fields, w.get() + 4 * ns, max_iterations, rtol, atol, iterations, relres,
                                              st );
}

template < typename T >
int divkgrad_apply( const tn_mesh* m, const T* k, int treat, int diag, int single, int apply_mode, int comm_mode,
                    const T* src, T* dst, cudaStream_t st )
{
    TN_CHECK_ARG( m && k && src && dst, "divkgrad_apply: null argument" );
    TN_CHECK_ARG( apply_mode == TN_APPLY_REPLACE || apply_mode == TN_APPLY_ADD, "divkgrad_apply: bad apply mode" );
    DivKGradParams< T > P{};
    if ( apply_mode == TN_APPLY_REPLACE )
        TN_CUDA_TRY( cudaMemsetAsync( dst, 0, m->ns * sizeof( T ), st ) );
    P.N = m->N, P.n1 = m->n1, P.table = triangle_table< T >( m );
    P.k = k, P.src = src, P.dst = dst, P.single = single != 0, P.treat = treat != 0;
    const long long cells = (long long) kDiamonds * m->N * m->N * m->N;
    P.cell_blocks         = unsigned( ( cells + 127 ) / 128 );
    const unsigned edge   = P.treat ? ( boundary_items( m->N ) + 127u ) / 128u : 0u;
    if ( diag )
        divkgrad_diagonal_kernel< T ><<< dim3( P.cell_blocks, 4 ), 128, 0, st >>>( P );
    else if ( single )
        divkgrad_kernel< T, true ><<< P.cell_blocks + edge, 128, 0, st >>>( P );
    else
        divkgrad_kernel< T, false ><<< P.cell_blocks + edge, 128, 0, st >>>( P );
    TN_LAUNCH_CHECK();
    if ( comm_mode == TN_COMM_ADDITIVE )
        return halo_sum< T >( m, &dst, 1, st );
    return TN_OK;
}

// VectorLaplace coupling (vector_laplace.hpp:181-210): the branch follows the
// boundary flag of the cell's own (x, y, r) node, CMB for layer 0 and
// SURFACE for every other layer, so a Dirichlet surface decouples the
// SURFACE-side nodes of every cell above layer 0.  Neumann and Dirichlet
// only (the reference aborts on free-slip).
template < typename T >
int vector_laplace_apply( const tn_mesh* m, int bc_cmb, int bc_surface, int diag, int apply_mode, int comm_mode,
                          const T* const* src, T* const* dst, cudaStream_t st )
{
    TN_CHECK_ARG( m, "vector_laplace_apply: mesh is NULL" );
    TN_CHECK_ARG( ( bc_cmb == TN_BC_NEUMANN || bc_cmb == TN_BC_DIRICHLET ) &&
                      ( bc_surface == TN_BC_NEUMANN || bc_surface == TN_BC_DIRICHLET ),
                  "vector_laplace_apply: boundary conditions must be Neumann or Dirichlet" );
    const int first = diag ? kDiag : ( bc_cmb == TN_BC_DIRICHLET ? kBot : kNeu );
    const int inner = diag ? kDiag : ( bc_surface == TN_BC_DIRICHLET ? kTop : kNeu );
    return constant_gradient_apply< T >( m, 3, src, dst, first, inner, inner, apply_mode, comm_mode, st,
                                         "vector_laplace_apply" );
}

}  // namespace tn

using namespace tn;

extern "C" int tn_laplace_apply_f64( const tn_mesh* m, int treat, int diag, int am, int cm, const double* src,
                                     double* dst, void* s )
{
    return laplace_apply< double >( m, treat, diag, am, cm, src, dst, as_stream( s ) );
}
extern "C" int tn_laplace_apply_f32( const tn_mesh* m, int treat, int diag, int am, int cm, const float* src,
                                     float* dst, void* s )
{
    return laplace_apply< float >( m, treat, diag, am, cm, src, dst, as_stream( s ) );
}
extern "C" int tn_divkgrad_apply_f64( const tn_mesh* m, const double* k, int treat, int diag, int single, int am,
                                      int cm, const double* src, double* dst, void* s )
{
    return divkgrad_apply< double >( m, k, treat, diag, single, am, cm, src, dst, as_stream( s ) );
}
extern "C" int tn_divkgrad_apply_f32( const tn_mesh* m, const float* k, int treat, int diag, int single, int am,
                                      int cm, const float* src, float* dst, void* s )
{
    return divkgrad_apply< float >( m, k, treat, diag, single, am, cm, src, dst, as_stream( s ) );
}
extern "C" int tn_vector_laplace_apply_f64( const tn_mesh* m, int bcc, int bcs, int diag, int am, int cm,
                                            const double* const* src, double* const* dst, void* s )
{
    return vector_laplace_apply< double >( m, bcc, bcs, diag, am, cm, src, dst, as_stream( s ) );
}
extern "C" int tn_vector_laplace_apply_f32( const tn_mesh* m, int bcc, int bcs, int diag, int am, int cm,
                                            const float* const* src, float* const* dst, void* s )
{
    return vector_laplace_apply< float >( m, bcc, bcs, diag, am, cm, src, dst, as_stream( s ) );
}
