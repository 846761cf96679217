// KMass apply (fe/wedge/operators/shell/kmass.hpp): int k u v with the 3x2
// Felippa rule, k interpolated at the quadrature points; consistent,
// diagonal or lumped-diagonal action.  With k = 1 it is the plain Mass
// (mass.hpp); applied per component it is the VectorMass used for right-hand
// sides (vector_mass.hpp).
//
// The plain mass matrix (k = 1, consistent or diagonal), which the FV -> FE
// projection applies in every CG iteration, separates into one lateral stencil
// and a radial factor (MassOp, lateral.cuh).  With a nodal k, and lumped: one
// thread per cell, atomic accumulation, then the additive halo (setup work).
#include "common.cuh"
#include "lateral_cg.cuh"
#include "wedge.cuh"

namespace tn {

namespace {

__device__ __constant__ const double kMQP[6][3] = { { 0.6666666666666666, 0.1666666666666667, -0.5773502691896257 },
                                                    { 0.1666666666666667, 0.6666666666666666, -0.5773502691896257 },
                                                    { 0.1666666666666667, 0.1666666666666667, -0.5773502691896257 },
                                                    { 0.6666666666666666, 0.1666666666666667, 0.5773502691896257 },
                                                    { 0.1666666666666667, 0.6666666666666666, 0.5773502691896257 },
                                                    { 0.1666666666666667, 0.1666666666666667, 0.5773502691896257 } };

template < typename T >
__global__ void __launch_bounds__( 128 ) kmass_kernel( int N, int n1, const double* __restrict__ coords,
                                                      const T* __restrict__ radii, const T* __restrict__ k,
                                                      const T* __restrict__ src, T* __restrict__ dst, int mode )
{
    const long long t = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    if ( t >= (long long) kDiamonds * N * N * N )
        return;
    const int r = int( t % N ), y = int( ( t / N ) % N ), x = int( ( t / ( (long long) N * N ) ) % N );
    const int d = int( t / ( (long long) N * N * N ) );
    const T   r1 = radii[d * n1 + r], r2 = radii[d * n1 + r + 1];
    for ( int w = 0; w < 2; ++w )
    {
        T      p[3][3], kn[6], s[6], o[6] = { 0, 0, 0, 0, 0, 0 };
        size_t idx[6];
        for ( int n = 0; n < 6; ++n )
        {
            const size_t lat = lat_index( n1, d, x + kWedgeNode[w][n][0], y + kWedgeNode[w][n][1] );
            if ( n < 3 )
            {
                const double* c = coords + lat * 3;
                p[n][0] = T( c[0] ), p[n][1] = T( c[1] ), p[n][2] = T( c[2] );
            }
            idx[n] = lat * n1 + r + kWedgeNode[w][n][2];
            kn[n]  = k ? k[idx[n]] : T( 1 );
            s[n]   = src[idx[n]];
        }
        for ( int q = 0; q < 6; ++q )
        {
            const T xi = T( kMQP[q][0] ), eta = T( kMQP[q][1] ), zeta = T( kMQP[q][2] );
            T       M[3][3];
            for ( int a = 0; a < 3; ++a )
            {
                M[a][0] = p[1][a] - p[0][a];
                M[a][1] = p[2][a] - p[0][a];
                M[a][2] = ( T( 1 ) - xi - eta ) * p[0][a] + xi * p[1][a] + eta * p[2][a];
            }
            const T det = M[0][0] * ( M[1][1] * M[2][2] - M[1][2] * M[2][1] ) -
                          M[0][1] * ( M[1][0] * M[2][2] - M[1][2] * M[2][0] ) +
                          M[0][2] * ( M[1][0] * M[2][1] - M[1][1] * M[2][0] );
            const T rq = r1 + T( 0.5 ) * ( r2 - r1 ) * ( T( 1 ) + zeta ), gr = T( 0.5 ) * ( r2 - r1 );
            const T lat[3] = { T( 1 ) - xi - eta, xi, eta };
            T       Nn[6], kq = 0, us = 0;
            for ( int n = 0; n < 6; ++n )
            {
                Nn[n] = lat[n % 3] * ( n < 3 ? T( 0.5 ) * ( T( 1 ) - zeta ) : T( 0.5 ) * ( T( 1 ) + zeta ) );
                kq += Nn[n] * kn[n];
                us += Nn[n] * s[n];
            }
            const T f = T( 0.1666666666666667 ) * kq * rq * rq * gr * fabs( det );
            for ( int i = 0; i < 6; ++i )
            {
                if ( mode == 0 )
                    o[i] += f * Nn[i] * us; // consistent: sum_j N_i N_j s_j
                else if ( mode == 1 )
                    o[i] += f * Nn[i] * Nn[i] * s[i];
                else
                    o[i] += f * Nn[i] * s[i]; // lumped: sum_j N_i N_j = N_i
            }
        }
        for ( int n = 0; n < 6; ++n )
            atomicAdd( dst + idx[n], o[n] );
    }
}

// A layer's two rows of the mass matrix from the lateral sums of its levels (stencil sum_q |D| lat_i lat_j / 6)
// and its radial factors B[li + lj] = h sum_zeta r^2 n_li n_lj.
// FP64 apply with its halo: 177 -> 23 us at level 6, 1,344 -> 171 us at level 7
// (one thread per cell and quadrature point by point before).
template < typename T >
struct MassOp
{
    static constexpr int           S = 1, D = 0, K = 1, R = 3;
    static constexpr bool          kDiff = false;
    static constexpr bool          kExactDot = true; // <p, A p> of the projection's CG: 20 steps at level 6 take 1 % longer
    static __device__ __forceinline__ void layer( const T ( &f )[R], const T ( &b )[S], const T ( &t )[S], const T ( & )[D + 1],
                                                  T& low, T& high )
    {
        low  = f[0] * b[0] + f[1] * t[0];
        high = f[1] * b[0] + f[2] * t[0];
    }
    static __device__ __forceinline__ T side_low( const T ( &f )[R], const T ( &s )[S], const T ( & )[D + 1] ) { return f[0] * s[0]; }
    static __device__ __forceinline__ T side_high( const T ( &f )[R], const T ( &s )[S], const T ( & )[D + 1] ) { return f[2] * s[0]; }
    static __device__ __forceinline__ T self_low( const T ( &f )[R], const T ( &v )[K] ) { return f[0] * v[0]; }
    static __device__ __forceinline__ T self_high( const T ( &f )[R], const T ( &v )[K] ) { return f[2] * v[0]; }
    // The tables are formed to their last bit: every layer of a column uses the same stencil and every column the same
    // radial factors, so their rounding does not average out (20 CG steps at levels 2 to 4 against extended precision: 7.0e-16 with plain
    // sums over the points, 6.5e-16 now; 6.6e-16 when every wedge was integrated by itself).
    // |D| of a triangle; the rule's sums of lat_i lat_j / 6 are 1/12 for i = j and else 1/24
    using Sum = Pair;
    static __device__ double entry( const Pair& a, int e ) { return quotient( a, e == 0 ? 12.0 : 24.0 ); }
    static __device__ void   triangle( const double* p0, const double* p1, const double* p2, int, const int ( &e )[3],
                                       Pair ( &A )[kStencil][K] )
    {
        Pair a[3], b[3], D;
#pragma unroll
        for ( int k = 0; k < 3; ++k )
            a[k] = pair_sum( p1[k], -p0[k] ), b[k] = pair_sum( p2[k], -p0[k] );
#pragma unroll
        for ( int k = 0; k < 3; ++k )
        {
            const int i = ( k + 1 ) % 3, j = ( k + 2 ) % 3;
            D           = D + ( a[i] * b[j] + -( a[j] * b[i] ) ) * Pair{ p0[k] };
        }
        if ( D.v < 0.0 )
            D = -D;
#pragma unroll
        for ( int j = 0; j < 3; ++j )
            A[e[j]][0] = A[e[j]][0] + D;
    }
    // h sum over zeta = -+1/sqrt(3) of r^2 n_li n_lj in closed form, m = r1 + h:
    // h (6 r1 m + 2 h^2) / 9, h (3 m^2 + h^2) / 9, h (6 r2 m + 2 h^2) / 9
    static __device__ void radial( double r1, double r2, double* f )
    {
        const Pair d = pair_sum( r2, -r1 ), s = pair_sum( r1, r2 ), h{ 0.5 * d.v, 0.5 * d.e }, m{ 0.5 * s.v, 0.5 * s.e };
        const Pair hh = h * h;
        f[0] = quotient( h * ( m * Pair{ r1 } * Pair{ 6.0 } + hh + hh ), 9.0 );
        f[1] = quotient( h * ( m * m * Pair{ 3.0 } + hh ), 9.0 );
        f[2] = quotient( h * ( m * Pair{ r2 } * Pair{ 6.0 } + hh + hh ), 9.0 );
    }
};

}  // namespace

template < typename T >
int kmass_apply( const tn_mesh* m, const T* k, int mode, int apply_mode, int comm_mode, const T* src, T* dst,
                 cudaStream_t st )
{
    TN_CHECK_ARG( m && src && dst, "kmass: null argument" );
    TN_CHECK_ARG( mode >= 0 && mode <= 2, "kmass: mode must be 0 (full), 1 (diagonal) or 2 (lumped)" );
    if ( !k && mode != 2 )
    {
        LateralParams< T > P{};
        P.src.p[0] = src, P.dst.p[0] = dst, P.mode_first = P.mode_inner = P.mode_last = mode == 1 ? kDiag : kNeu;
        if ( !lateral_tables< MassOp< T > >( m, &tn_mesh::mass_tables, P ) )
        {
            set_error( "kmass: allocating the lateral stencil failed" );
            return TN_ERR_NOMEM;
        }
        return launch_lateral< MassOp< T > >( m, P, 1, apply_mode, comm_mode, st );
    }
    if ( apply_mode == TN_APPLY_REPLACE )
        TN_CUDA_TRY( cudaMemsetAsync( dst, 0, m->ns * sizeof( T ), st ) );
    const T* radii = sizeof( T ) == 8 ? reinterpret_cast< const T* >( m->d_radii )
                                      : reinterpret_cast< const T* >( m->d_radii32 );
    const long long cells = (long long) kDiamonds * m->N * m->N * m->N;
    kmass_kernel< T ><<< unsigned( ( cells + 127 ) / 128 ), 128, 0, st >>>( m->N, m->n1, m->d_coords, radii, k, src, dst,
                                                                          mode );
    TN_LAUNCH_CHECK();
    if ( comm_mode == TN_COMM_ADDITIVE )
    {
        T* f[1] = { dst };
        return halo_sum< T >( m, f, 1, st );
    }
    return TN_OK;
}

// The stencils of the plain mass matrix are formed with the mesh, in both precisions: its apply had no table before it
// was separated, so a first one may not allocate or wait (it may be inside a stream capture).
size_t mass_table_words( const tn_mesh* m, bool radial ) { return lateral_table_words< MassOp< double > >( m, radial ); }
bool   fill_mass_tables( const tn_mesh* m )
{
    const tn_lateral_tables& t = m->mass_tables;
    return lateral_fill< MassOp< double > >( m, LateralTables{ t.lat, t.rad, t.lat32, t.rad32 }, nullptr );
}

// CG on the plain mass matrix from x's values (lateral_cg.cuh); fields: 4 stored-node fields
int mass_cg( const tn_mesh* m, const double* b, double* x, double* fields, int max_iterations, double rtol, double atol,
             int* iterations, cudaStream_t st )
{
    LateralParams< double > P{};
    if ( !lateral_tables< MassOp< double > >( m, &tn_mesh::mass_tables, P ) )
    {
        set_error( "mass_cg: allocating the lateral stencil failed" );
        return TN_ERR_NOMEM;
    }
    const size_t    ns = m->ns;
    const WorkBlock w( m, lateral_cg_scratch< MassOp< double > >( m, max_iterations ) );
    if ( !w.get() )
    {
        set_error( "mass_cg: allocating the scratch failed" );
        return TN_ERR_NOMEM;
    }
    double* const f[4] = { fields, fields + ns, fields + 2 * ns, fields + 3 * ns };
    return lateral_cg< MassOp< double > >( m, P, b, x, f, w.get(), max_iterations, rtol, atol, iterations, nullptr, st );
}

template int kmass_apply< double >( const tn_mesh*, const double*, int, int, int, const double*, double*, cudaStream_t );
template int kmass_apply< float >( const tn_mesh*, const float*, int, int, int, const float*, float*, cudaStream_t );

}  // namespace tn

using namespace tn;

extern "C" int tn_kmass_apply_f64( const tn_mesh* m, const double* k, int mode, int am, int cm, const double* src,
                                   double* dst, void* s )
{
    return kmass_apply< double >( m, k, mode, am, cm, src, dst, as_stream( s ) );
}
extern "C" int tn_kmass_apply_f32( const tn_mesh* m, const float* k, int mode, int am, int cm, const float* src,
                                   float* dst, void* s )
{
    return kmass_apply< float >( m, k, mode, am, cm, src, dst, as_stream( s ) );
}
