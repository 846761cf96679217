// SUPG-stabilised unsteady advection-diffusion operator (B200 design of
// UnsteadyAdvectionDiffusionSUPG, fe/wedge/operators/shell/
// unsteady_advection_diffusion_supg.hpp): the left-hand side
// mass_scaling M + dt (K + C + G) of an implicit BDF step for the temperature,
//   M_ij = int phi_i phi_j,  K_ij = int kappa grad phi_i . grad phi_j,
//   C_ij = int phi_i (u . grad phi_j),
//   G_ij = sum_E tau_E int_E (u . grad phi_i) (u . grad phi_j),
// on the 3x2 Felippa rule with the velocity interpolated at the quadrature
// points and tau_E the weight-averaged pointwise supg_tau of the wedge
// (h = r2 - r1; :16-50, :286-312).
//
// Matrix-free: instead of forming the 6 x 6 wedge matrices (:314-341) each
// quadrature point forms the source value s_q, its gradient and u . gs once, and
// every node's row follows as
//   ms phi_i s_q + dt (kappa grad phi_i . gs + phi_i u . gs + tau (u . grad phi_i)(u . gs)).
// In the factored form of cell.cuh the scaled gradient D r gs = beta_1 S_1 +
// beta_2 S_2 + v Z has edge differences S_i that depend on zeta only, so a point
// needs Z, the three products of u with beta_1, beta_2, v and nothing per node:
// the rows are formed once per zeta from the points' sums and their moments
// with the lateral shape functions.  tau multiplies one of those sums, so a single
// pass accumulates it beside them.  The matrix modifications of the reference
// are expressed on that form: the lumped mass is ms phi_i per point times the
// node's own value; the boundary mask (off-diagonal entries of the rows and
// columns of CMB / surface nodes zeroed, :350-386) is the action on the source
// with those nodes zeroed for the other rows and the diagonal entry times the
// node's value for the boundary rows (further blocks of the launch, one thread
// per lateral cell, wedge and side); the diagonal mode (:388-394) is the diagonal
// entries alone.
//
// One thread per cell, lanes along r, contributions added by add_column, then
// the additive halo sum.  Level-6 apply: FP64 1,480 -> 457 us, FP32 620 -> 208 us
// (half of what is left is tau: a root, an exponential and a division at each of
// twelve points per cell).
#include <cmath>

#include "cell.cuh"
#include "common.cuh"
#include "wedge.cuh"

namespace tn {

template < typename T >
int halo_sum( const tn_mesh* m, T* const* fields, int nfields, cudaStream_t st );

namespace {

template < typename T >
struct SupgParams
{
    int             N, n1;
    const T*        table;
    Ptr3< const T > vel;
    const T*        src;
    T*              dst;
    T               kappa, dt, ms;
    int             lumped, treat;
    unsigned        cell_blocks; // blocks of cells; those after them add diagonals
};

// supg_tau (:16-50) = (r2 - r1) / (2 |u|) (coth(pe) - 1 / pe), pe = |u| (r2 - r1) / (2 kappa'), kappa' = max(kappa,
// 1e-8), zero for a vanishing |u| or pe; the reference's cap 10 (r2 - r1) / |u| is never reached (coth(x) - 1 / x < 1).
// uu = |u|^2, kv = kappa', hk = (r2 - r1) / (2 kappa').  With e = exp(-2 pe), coth = (1 + e) / (1 - e): one exponential
// and one division; below pe = 1/2, where that difference cancels, coth(x) - 1/x = x sum_n 2^2n B_2n / (2n)! x^(2n-2)
// (B_2n the Bernoulli numbers), whose terms fall by (x / pi)^2 < 1/39: ten of them (five in FP32), and no root.
template < typename T >
__device__ __forceinline__ T supg_tau( T uu, T kv, T hk )
{
    const T pe2 = uu * hk * hk;
    if ( uu <= T( 1e-24 ) || pe2 <= T( 1e-16 ) )
        return T( 0 );
    if ( pe2 < T( 0.25 ) )
    {
        constexpr double c[10] = { 1.0 / 3.0,
                                   -1.0 / 45.0,
                                   2.0 / 945.0,
                                   -1.0 / 4725.0,
                                   2.0 / 93555.0,
                                   -1382.0 / 638512875.0,
                                   4.0 / 18243225.0,
                                   -3617.0 / 162820783125.0,
                                   87734.0 / 38979295480125.0,
                                   -349222.0 / 1531329465290625.0 };
        constexpr int    terms = sizeof( T ) == 8 ? 10 : 5;
        T                s     = T( c[terms - 1] );
#pragma unroll
        for ( int n = terms - 2; n >= 0; --n )
            s = s * pe2 + T( c[n] );
        return kv * hk * hk * s;
    }
    const T pe = sqrt( uu ) * hk, e = exp( T( -2 ) * pe ), d = T( 1 ) - e;
    return kv * ( pe * ( T( 1 ) + e ) - d ) / ( uu * d );
}

template < typename T >
__device__ __forceinline__ void supg_wedge( const SupgParams< T >& P, const Triangle< T >& G, T h, T rho_b, T rho_t,
                                            const T ( &s )[6], const T ( &vn )[6][3], T ( &out )[6] )
{
    const T kv = fmax( P.kappa, T( 1e-8 ) ), hk = h / kv; // (r2 - r1) / (2 kappa') = h / kappa'
    const T b11 = dot3( G.b1, G.b1 ), b12 = dot3( G.b1, G.b2 ), b22 = dot3( G.b2, G.b2 );
    const T a1 = dot3( G.b1, G.v ), a2 = dot3( G.b2, G.v ), vv = dot3( G.v, G.v ), aD = fabs( G.iD );
    const T t[3] = { T( 0.5 ) * ( s[3] - s[0] ), T( 0.5 ) * ( s[4] - s[1] ), T( 0.5 ) * ( s[5] - s[2] ) };
    const T ts = ( t[0] + t[1] + t[2] ) * T( 1.0 / 6.0 );
    const T wD = T( kFelippaW ) * h / aD;              // w h |D|: |det J| w = r^2 wD
    const T wi = T( kFelippaW ) * h * aD * P.dt;       // dt w h / |D|
    T       tau = T( 0 ), L[3], B[6], M[3];            // radial parts; rows times tau and their radial parts
#pragma unroll
    for ( int n = 0; n < 6; ++n )
        out[n] = B[n] = T( 0 );
    L[0] = L[1] = L[2] = M[0] = M[1] = M[2] = T( 0 );
#pragma unroll
    for ( int zq = 0; zq < 2; ++zq )
    {
        const T nb = T( zq ? 0.5 * ( 1.0 - kFelippaZ ) : 0.5 * ( 1.0 + kFelippaZ ) );
        const T nt = T( zq ? 0.5 * ( 1.0 + kFelippaZ ) : 0.5 * ( 1.0 - kFelippaZ ) );
        const T rho = zq ? rho_t : rho_b, r = rho * h;
        T       sz[3], uz[3][3], us[3];
#pragma unroll
        for ( int m = 0; m < 3; ++m )
        {
            sz[m] = nb * s[m] + nt * s[3 + m];
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                uz[m][c] = nb * vn[m][c] + nt * vn[3 + m][c];
        }
#pragma unroll
        for ( int c = 0; c < 3; ++c )
            us[c] = ( uz[0][c] + uz[1][c] + uz[2][c] ) * T( 1.0 / 6.0 );
        const T ss = ( sz[0] + sz[1] + sz[2] ) * T( 1.0 / 6.0 );
        const T S1 = nb * ( s[1] - s[0] ) + nt * ( s[4] - s[3] ), S2 = nb * ( s[2] - s[0] ) + nt * ( s[5] - s[3] );
        const T Z0 = rho * ts - T( 1.0 / 6.0 ) * ( S1 + S2 );
        const T al = r * r * wD, adv = P.dt * G.iD / r; // w |det J|; dt / (D r)
        T       R[3], q1 = T( 0 ), q2 = T( 0 ), qv[3], Z[3];
#pragma unroll
        for ( int q = 0; q < 3; ++q )
        {
            const int m = ( q + 1 ) % 3; // point q lies next to vertex m
            const T   u[3] = { us[0] + T( 0.5 ) * uz[m][0], us[1] + T( 0.5 ) * uz[m][1], us[2] + T( 0.5 ) * uz[m][2] };
            const T   c1 = dot3( G.b1, u ), c2 = dot3( G.b2, u ), cv = dot3( G.v, u );
            Z[q] = Z0 + T( 0.5 ) * ( m == 1 ? rho * t[1] - S1 : ( m == 2 ? rho * t[2] - S2 : rho * t[0] ) );
            const T ug = c1 * S1 + c2 * S2 + cv * Z[q]; // D r u . gs
            R[q] = al * ( ( P.lumped ? T( 0 ) : P.ms * ( ss + T( 0.5 ) * sz[m] ) ) + adv * ug );
            q1 += c1 * ug, q2 += c2 * ug;
            qv[q] = cv * ug;
            tau += supg_tau( dot3( u, u ), kv, hk );
        }
        // sums and moments over the points: those of xi, eta, lat_0 are the sum / 6 plus half of point 0, 1, 2
        const T Rs = ( R[0] + R[1] + R[2] ) * T( 1.0 / 6.0 ), qs = ( qv[0] + qv[1] + qv[2] ) * T( 1.0 / 6.0 );
        const T Zs = Z[0] + Z[1] + Z[2], k3 = wi * P.kappa;
        const T p1 = k3 * ( T( 3 ) * ( S1 * b11 + S2 * b12 ) + a1 * Zs ), p2 = k3 * ( T( 3 ) * ( S1 * b12 + S2 * b22 ) + a2 * Zs );
        const T pv = a1 * S1 + a2 * S2;
        const T ps = k3 * ( T( 0.5 ) * pv + vv * Zs * T( 1.0 / 6.0 ) );
        const T lump = P.lumped ? al * P.ms : T( 0 );
        T       X[3], Q[3];
#pragma unroll
        for ( int m = 0; m < 3; ++m )
        {
            const int q = ( m + 2 ) % 3; // the point next to vertex m
            X[m] = ps + T( 0.5 ) * k3 * ( pv + vv * Z[q] );
            Q[m] = wi * ( qs + T( 0.5 ) * qv[q] );
        }
        const T f1 = p1 - X[1], f2 = p2 - X[2], g1 = wi * q1 - Q[1], g2 = wi * q2 - Q[2];
#pragma unroll
        for ( int m = 0; m < 3; ++m )
        {
            const int q   = ( m + 2 ) % 3;
            const T   f   = m == 0 ? -( f1 + f2 ) : ( m == 1 ? f1 : f2 ), g = m == 0 ? -( g1 + g2 ) : ( m == 1 ? g1 : g2 );
            const T   row = f + Rs + T( 0.5 ) * R[q];
            out[m] += nb * ( row + lump * s[m] ), out[3 + m] += nt * ( row + lump * s[3 + m] );
            B[m] += nb * g, B[3 + m] += nt * g;
            L[m] += rho * X[m], M[m] += rho * Q[m];
        }
    }
    tau *= T( 1.0 / 6.0 );
#pragma unroll
    for ( int m = 0; m < 3; ++m )
    {
        const T l = T( 0.5 ) * ( L[m] + tau * M[m] );
        out[m] += tau * B[m] - l, out[3 + m] += tau * B[3 + m] + l;
    }
}

// adds the diagonal entries of the three lower (top false) or upper nodes of a wedge times their values
template < typename T >
__device__ __forceinline__ void supg_diagonal( const SupgParams< T >& P, int d, int x, int y, int r, int w, bool top )
{
    const T             h = layer_h( P.table, P.N, r ), rh = layer_q( P.table, P.N, r ), side = top ? T( 1 ) : T( -1 );
    const T             kv = fmax( P.kappa, T( 1e-8 ) ), hk = h / kv;
    const Triangle< T > G( P.table, P.N, d, x, y, w );
    unsigned            node[4], id[3];
    T                   vn[6][3], o[3] = { T( 0 ), T( 0 ), T( 0 ) }, b[3] = { T( 0 ), T( 0 ), T( 0 ) }, tau = T( 0 );
    cell_nodes( P.n1, d, x, y, r, node );
    wedge_columns( node, w, id );
#pragma unroll
    for ( int n = 0; n < 6; ++n )
#pragma unroll
        for ( int c = 0; c < 3; ++c )
            vn[n][c] = P.vel.p[c][id[n % 3] + n / 3];
    for ( int q = 0; q < 6; ++q )
    {
        const T xi = T( felippa_xi( q ) ), eta = T( felippa_eta( q ) ), zeta = T( q < 3 ? -kFelippaZ : kFelippaZ );
        const T lat[3] = { T( 1 ) - xi - eta, xi, eta };
        T       u[3] = { T( 0 ), T( 0 ), T( 0 ) };
#pragma unroll
        for ( int n = 0; n < 6; ++n )
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                u[c] += lat[n % 3] * T( 0.5 ) * ( n < 3 ? T( 1 ) - zeta : T( 1 ) + zeta ) * vn[n][c];
        const T rho = rh + T( 1 ) + zeta, rq = h * rho, ad = T( kFelippaW ) * rq * rq * h / fabs( G.iD ), iDr = G.iD / rq;
        tau += supg_tau( dot3( u, u ), kv, hk ) * T( 1.0 / 6.0 );
#pragma unroll
        for ( int m = 0; m < 3; ++m )
        {
            T g[3];
            scaled_gradient( G, m, side, xi, eta, zeta, rho, g );
            const T phi = lat[m] * T( 0.5 ) * ( T( 1 ) + side * zeta ), ug = iDr * dot3( u, g ), gg = iDr * iDr * dot3( g, g );
            o[m] += ad * ( P.ms * phi * ( P.lumped ? T( 1 ) : phi ) + P.dt * ( P.kappa * gg + phi * ug ) );
            b[m] += ad * P.dt * ug * ug;
        }
    }
#pragma unroll
    for ( int m = 0; m < 3; ++m )
        atomicAdd( P.dst + id[m] + top, ( o[m] + tau * b[m] ) * P.src[id[m] + top] );
}

// Blocks per SM, level 6: FP64 at 3 / 4 / 5 blocks 459 / 456 / 604 us (level 5: 71 / 74 / 88), FP32 at 3 / 4 / 6 237 /
// 207 / 230 us.
template < typename T >
__global__ void __launch_bounds__( 128, sizeof( T ) == 8 ? 3 : 4 ) supg_kernel( SupgParams< T > P )
{
    const int N = P.N, n1 = P.n1;
    int       d, x, y, r;
    if ( blockIdx.x >= P.cell_blocks )
    {
        // the kept diagonal of the CMB nodes (layer 0) and of the SURFACE nodes (layer N - 1)
        int  w;
        bool top;
        if ( boundary_item( ( blockIdx.x - P.cell_blocks ) * blockDim.x + threadIdx.x, N, d, x, y, r, w, top ) )
            supg_diagonal( P, d, x, y, r, w, top );
        return;
    }
    const bool in  = cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, N, d, x, y, r );
    const bool cmb = P.treat && r == 0, surf = P.treat && r == N - 1;
    const T    h = layer_h( P.table, N, r ), rh = layer_q( P.table, N, r );
    const T    rho_b = rh + T( 1.0 - kFelippaZ ), rho_t = rh + T( 1.0 + kFelippaZ );
    unsigned   node[4];
    cell_nodes( n1, d, x, y, r, node );
    T* const   dst[1] = { P.dst };
    T          acc[2][2]; // columns (x + 1, y) and (x, y + 1) get both wedges
#pragma unroll
    for ( int w = 0; w < 2; ++w )
    {
        const Triangle< T > G( P.table, N, d, x, y, w );
        T                   s[6], vn[6][3], out[6];
        const unsigned      id[3] = { node[w ? 3 : 0], node[w ? 2 : 1], node[w ? 1 : 2] };
#pragma unroll
        for ( int n = 0; n < 6; ++n )
        {
            const unsigned i = id[n % 3] + n / 3;
            const T        v = P.src[i];
            s[n]             = ( n < 3 ? cmb : surf ) ? T( 0 ) : v;
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                vn[n][c] = P.vel.p[c][i];
        }
        supg_wedge( P, G, h, rho_b, rho_t, s, vn, out );
        const T low0[1] = { out[0] }, high0[1] = { out[3] };
        add_column< T, 1 >( dst, id[0], r, N, in, !cmb, !surf, low0, high0 );
#pragma unroll
        for ( int m = 1; m < 3; ++m )
        {
            const int a = w ? 2 - m : m - 1; // vertex m of wedge 0 is vertex 3 - m of wedge 1
            if ( w == 0 )
                acc[a][0] = out[m], acc[a][1] = out[3 + m];
            else
            {
                const T low[1] = { acc[a][0] + out[m] }, high[1] = { acc[a][1] + out[3 + m] };
                add_column< T, 1 >( dst, id[m], r, N, in, !cmb, !surf, low, high );
            }
        }
    }
}

// the diagonal alone: one thread per cell, wedge and side (blockIdx.y)
template < typename T >
__global__ void __launch_bounds__( 128 ) supg_diagonal_kernel( SupgParams< T > P )
{
    int d, x, y, r;
    if ( cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, P.N, d, x, y, r ) )
        supg_diagonal( P, d, x, y, r, int( blockIdx.y & 1 ), blockIdx.y >= 2 );
}

template < typename T >
int supg_apply( const tn_mesh* m, const T* const* vel, double kappa, double dt, double mass_scaling, int lumped,
                int treat_boundary, int diagonal, int apply_mode, int comm_mode, const T* src, T* dst, void* s )
{
    TN_CHECK_ARG( m && vel && vel[0] && vel[1] && vel[2] && src && dst, "supg apply: null argument" );
    TN_CHECK_ARG( apply_mode == TN_APPLY_REPLACE || apply_mode == TN_APPLY_ADD, "supg apply: bad apply mode" );
    TN_CHECK_ARG( comm_mode == TN_COMM_SKIP || comm_mode == TN_COMM_ADDITIVE, "supg apply: bad communication mode" );
    cudaStream_t st = as_stream( s );
    if ( apply_mode == TN_APPLY_REPLACE )
        TN_CUDA_TRY( cudaMemsetAsync( dst, 0, m->ns * sizeof( T ), st ) );
    SupgParams< T > P;
    P.N = m->N, P.n1 = m->n1, P.table = triangle_table< T >( m );
    P.vel   = Ptr3< const T >{ { vel[0], vel[1], vel[2] } };
    P.src = src, P.dst = dst;
    P.kappa = T( kappa ), P.dt = T( dt ), P.ms = T( mass_scaling );
    P.lumped = lumped != 0, P.treat = treat_boundary != 0;
    const long long cells = 10LL * m->N * m->N * m->N;
    P.cell_blocks         = unsigned( ( cells + 127 ) / 128 );
    const unsigned edge   = P.treat ? ( boundary_items( m->N ) + 127u ) / 128u : 0u;
    if ( diagonal )
        supg_diagonal_kernel< T ><<< dim3( P.cell_blocks, 4 ), 128, 0, st >>>( P );
    else
        supg_kernel< T ><<< P.cell_blocks + edge, 128, 0, st >>>( P );
    TN_LAUNCH_CHECK();
    if ( comm_mode == TN_COMM_ADDITIVE )
        return halo_sum< T >( m, &dst, 1, st );
    return TN_OK;
}

}  // namespace
}  // namespace tn

using namespace tn;

extern "C" int tn_supg_apply_f64( const tn_mesh* m, const double* const* vel, double kappa, double dt,
                                  double mass_scaling, int lumped_mass, int treat_boundary, int diagonal, int apply_mode,
                                  int comm_mode, const double* src, double* dst, void* stream )
{
    return supg_apply< double >( m, vel, kappa, dt, mass_scaling, lumped_mass, treat_boundary, diagonal, apply_mode,
                                 comm_mode, src, dst, stream );
}

extern "C" int tn_supg_apply_f32( const tn_mesh* m, const float* const* vel, double kappa, double dt, double mass_scaling,
                                  int lumped_mass, int treat_boundary, int diagonal, int apply_mode, int comm_mode,
                                  const float* src, float* dst, void* stream )
{
    return supg_apply< float >( m, vel, kappa, dt, mass_scaling, lumped_mass, treat_boundary, diagonal, apply_mode,
                                comm_mode, src, dst, stream );
}

#include "../cpp/tn/operators.hpp"
#include "../cpp/tn/solvers.hpp"

extern "C" int tn_supg_solve_f64( const tn_mesh* m, const double* const* vel, double kappa, double dt,
                                  double mass_scaling, int lumped_mass, int treat_boundary, const double* rhs, double* x,
                                  int l, int max_iterations, double relative_tolerance, double absolute_tolerance,
                                  double* work, int* iterations, double* relative_residual, void* s )
{
    TN_CHECK_ARG( m && vel && vel[0] && vel[1] && vel[2] && rhs && x && work, "tn_supg_solve_f64: null argument" );
    TN_CHECK_ARG( l >= 1 && l <= 8 && max_iterations >= 1, "tn_supg_solve_f64: bad solver parameters" );
    cudaStream_t st = as_stream( s );
    const size_t ns = m->ns;
    try
    {
        struct StreamScope // the C++ layer issues on tn::stream(): this call's stream for its duration
        {
            cudaStream_t prev;
            explicit StreamScope( cudaStream_t s ) : prev( stream_ref() ) { stream_ref() = s; }
            ~StreamScope() { stream_ref() = prev; }
        } scope( st );
        Mesh                     mesh = Mesh::wrap( m );
        VectorQ1Scalar< double > b( mesh, const_cast< double* >( rhs ) ), xx( mesh, x );
        // the velocity as a non-owning view of its three contiguous components
        TN_CHECK_ARG( vel[1] == vel[0] + ns && vel[2] == vel[0] + 2 * ns,
                      "tn_supg_solve_f64: the velocity components must be one contiguous [3][nodes] array" );
        VectorQ1Vec< double > u( mesh, const_cast< double* >( vel[0] ) );
        std::vector< VectorQ1Scalar< double > > tmps;
        for ( int i = 0; i < 2 * ( l + 1 ) + 2; ++i )
            tmps.emplace_back( mesh, work + size_t( i ) * ns );
        UnsteadyAdvectionDiffusionSUPG< double > A( mesh, u, kappa, dt, treat_boundary != 0, false, mass_scaling,
                                                    lumped_mass != 0 );
        PBiCGStab< UnsteadyAdvectionDiffusionSUPG< double > > solver(
            l, IterativeSolverParameters{ max_iterations, relative_tolerance, absolute_tolerance }, tmps );
        solve( solver, A, xx, b );
        if ( iterations )
            *iterations = solver.stats.iterations;
        if ( relative_residual )
            *relative_residual = solver.stats.relative_residuals.empty() ? 0.0 : solver.stats.relative_residuals.back();
    }
    catch ( const std::exception& e )
    {
        set_error( std::string( "tn_supg_solve_f64: " ) + e.what() );
        return TN_ERR_CUDA;
    }
    return TN_OK;
}
