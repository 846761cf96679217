// Finite-volume FCT advection-diffusion on the hex cells of the shell
// (fv/hex/operators/fct_advection_diffusion.hpp, geometry_helper.hpp,
// fv/hex/helpers.hpp, communication/shell/fv_communication.hpp).
//
// FV fields are [10][N+2][N+2][N+2] with one ghost layer (r fastest); cell
// (x, y, r), 1 <= x, y, r <= N, is the FE cell (x-1, y-1, r-1).  Lateral
// ghosts are copies of the real cells across each diamond face (the mesh's
// FV ghost map); radial ghosts hold what the boundary treatment writes.
//
// The kernels of a step take the cells in runs along x, one per thread, r fastest (March).  The cell
// geometry (face fluxes beta, face vectors S, volume M) is formed from the
// mesh's triangle vectors (cell.cuh) and the Q1 velocity in FP64 in the dt and
// predictor kernels, with the reference's face and volume quadrature sums
// evaluated in closed form (FvWalk).
//
// The antidiffusive flux of cell i towards neighbour j is F_ij = dt / M_i
// |beta_ij| / 2 (T_i - T_j): apart from M_i it is the same for both sides of a
// face with opposite signs, so one value per face is stored,
//     g = |beta| / 2 (T_i - T_j) of cell i's face towards its lower neighbour j,
// three planes instead of six (48 bytes per cell less over the step's one write
// and two reads; those and T_L, R+ and R- are what bounds the step).  A cell takes
// its upper faces from its upper neighbours' entries; the last cell in a direction
// stores its own upper face in the ghost cell there.  Level 7 (20,971,520 cells):
// step 2.09 -> 1.20 ms, stable dt 0.81 -> 0.46 ms.
#include <algorithm>

#include "cell.cuh"
#include "common.cuh"
#include "wedge.cuh"

namespace tn {

namespace {

constexpr int kFvThreads = 128;

__device__ __constant__ const int kFvOff[6][3] = { { -1, 0, 0 }, { 1, 0, 0 }, { 0, -1, 0 },
                                                   { 0, 1, 0 },  { 0, 0, -1 }, { 0, 0, 1 } };

__device__ __forceinline__ size_t fv_index( int n2, int d, int x, int y, int r )
{
    return ( ( size_t( d ) * n2 + x ) * n2 + y ) * n2 + r;
}

struct FvGeom
{
    int                  N;
    const double*        table; // triangles (cell.cuh)
    const double*        radii;
    Ptr3< const double > cen; // FV cell centres with ghosts
    Ptr3< const double > vel; // Q1 velocity (stored nodes)
    const uint8_t*       orient; // face orientation bits per cell
};

// GeometryHelper::compute_geometry (geometry_helper.hpp:180-363) in closed form (the sums are FvWalk's, below).
//
// The reference integrates each face of the two wedges of the cell with a
// quadrature rule over the wedge map x = r(zeta) (p0 + xi a + eta b),
// a = p1 - p0, b = p2 - p0, r(zeta) = r1 + h (1 + zeta), h = (r2 - r1) / 2, and
// the Q1 velocity u(q) = sum_i N_i(q) u_i: beta = sum_q w_q u(q) . n(q),
// S = sum_q w_q n(q), and M = sum over the 3x2 volume rule of |det J| / 6.  On
// this map every such sum has a closed form:
//   * the radial triangles zeta = -+1 (neighbours 4, 5; 3-point rule, 1/6
//     weights): n = r^2 (a x b) is constant, each lateral shape function sums
//     to 1 over the points, so beta = r^2 / 6 (a x b) . (u_0 + u_1 + u_2) of
//     the face's nodes and S = r^2 / 2 (a x b);
//   * the quad xi = 0 (2x2 Gauss, weights 1/2 on [0,1] x [-1,1]): n = r(zeta)
//     h (b x p0), so beta = h (b x p0) . (R_b (u_0 + u_2) + R_t (u_3 + u_5)),
//     S = (r(-g) + r(g)) h (b x p0), with g = 1/sqrt(3),
//     R_b = (r(-g) (1 + g) + r(g) (1 - g)) / 4 and R_t = (r(-g) (1 - g) +
//     r(g) (1 + g)) / 4 the Gauss sums of r(zeta) times the bottom / top
//     radial shape functions; the quad eta = 0 alike with a in place of b and
//     nodes 1, 4 in place of 2, 5;
//   * det J = r(zeta)^2 h (a x b) . p0, so M = sum_w h |(a x b) . p0|
//     (r(-g)^2 + r(g)^2) / 2: a lateral factor times a radial one, whose inverses
//     are tabulated (iM = 1 / M, fv_inverse_volume).
// These are the same sums (exact algebra, different rounding: ~1e-16
// relative), about 120 FP64 operations per cell instead of ~3,000, with b x p0,
// a x p0 = -(p0 x a), a x b and 1 / ((a x b) . p0) from the triangle table (FvWalk).  Every
// face is oriented from its cell towards the neighbour's centre: that test, here, is
// made once per mesh and kept as one bit per face (set: the normal points inwards).
__device__ __forceinline__ unsigned inward_faces( const FvGeom& G, int d, int x, int y, int r )
{
    const int    N = G.N, n1 = N + 1, n2 = N + 2;
    const double r1 = G.radii[d * n1 + r - 1], r2 = G.radii[d * n1 + r];
    const double g = 0.5773502691896258, h = 0.5 * ( r2 - r1 ); // g = 1 / sqrt(3)
    const double rs = ( r1 + h * ( 1.0 - g ) ) + ( r1 + h * ( 1.0 + g ) );
    const Triangle< double > t0( G.table, N, d, x - 1, y - 1, 0 ), t1( G.table, N, d, x - 1, y - 1, 1 );
    const size_t ci   = fv_index( n2, d, x, y, r );
    unsigned     bits = 0;
    double       dc[6] = { 0.0, 0.0, 0.0, 0.0, 0.0, 0.0 };
#pragma unroll
    for ( int c = 0; c < 3; ++c )
    {
        const double S[6] = { rs * h * t0.b1[c],
                              rs * h * t1.b1[c],
                              -rs * h * t0.b2[c],
                              -rs * h * t1.b2[c],
                              0.5 * r1 * r1 * ( t0.v[c] + t1.v[c] ),
                              0.5 * r2 * r2 * ( t0.v[c] + t1.v[c] ) };
#pragma unroll
        for ( int n = 0; n < 6; ++n )
        {
            const size_t cj = fv_index( n2, d, x + kFvOff[n][0], y + kFvOff[n][1], r + kFvOff[n][2] );
            dc[n] += S[n] * ( G.cen.p[c][cj] - G.cen.p[c][ci] );
        }
    }
#pragma unroll
    for ( int n = 0; n < 6; ++n )
        if ( dc[n] < 0 )
            bits |= 1u << n;
    return bits;
}

__device__ __forceinline__ bool cell_of_thread( int N, int& d, int& x, int& y, int& r )
{
    const bool in = cell_of( blockIdx.x * (long long) blockDim.x + threadIdx.x, N, d, x, y, r );
    ++x, ++y, ++r;
    return in;
}

// compute_cell_centers (fv/hex/helpers.hpp:101-150)
__global__ void __launch_bounds__( kFvThreads ) cell_centers_kernel( int N, const double* __restrict__ coords,
                                                                     const double* __restrict__ radii, Ptr3< double > c )
{
    int d, x, y, r;
    if ( !cell_of_thread( N, d, x, y, r ) )
        return;
    const int    n1 = N + 1, n2 = N + 2;
    const double r1 = radii[d * n1 + r - 1], r2 = radii[d * n1 + r];
    double       vol = 0.0, acc[3] = { 0, 0, 0 };
    for ( int w = 0; w < 2; ++w )
    {
        double p[3][3];
        for ( int i = 0; i < 3; ++i )
        {
            const size_t lat = lat_index( n1, d, x - 1 + kWedgeNode[w][i][0], y - 1 + kWedgeNode[w][i][1] );
            for ( int a = 0; a < 3; ++a )
                p[i][a] = coords[lat * 3 + a];
        }
        for ( int q = 0; q < 6; ++q )
        {
            const double xi = q % 3 == 0 ? 0.6666666666666666 : 0.1666666666666667;
            const double et = q % 3 == 1 ? 0.6666666666666666 : 0.1666666666666667;
            const double ze = q < 3 ? -0.5773502691896257 : 0.5773502691896257;
            double       IT[3][3];
            const double Jw = fabs( wedge_jacobian_it( p[0], p[1], p[2], r1, r2, xi, et, ze, IT ) ) * 0.1666666666666667;
            const double rq = r1 + 0.5 * ( r2 - r1 ) * ( 1.0 + ze );
            vol += Jw;
            for ( int a = 0; a < 3; ++a )
                acc[a] += ( ( 1.0 - xi - et ) * p[0][a] + xi * p[1][a] + et * p[2][a] ) * rq * Jw;
        }
    }
    const size_t i = fv_index( n2, d, x, y, r );
    for ( int a = 0; a < 3; ++a )
        c.p[a][i] = acc[a] / vol;
}

// lateral ghost layer: thread per (ghost cell, r)
__global__ void fv_ghost_kernel( int N, const int* __restrict__ map, Ptr3< double > fields )
{
    double* f = fields.at( blockIdx.y );
    const long long t     = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    const long long total = (long long) kDiamonds * 4 * N * N;
    if ( t >= total )
        return;
    const int  r     = int( t % N ) + 1;
    const long long e = t / N; // (d * 4 + side) * N + i
    const int  i     = int( e % N );
    const int  side  = int( ( e / N ) % 4 );
    const int  d     = int( e / ( 4LL * N ) );
    const int* m     = map + e * 3;
    const int  n2    = N + 2;
    const int  gx    = side == 0 ? 0 : ( side == 1 ? N + 1 : i + 1 );
    const int  gy    = side == 2 ? 0 : ( side == 3 ? N + 1 : i + 1 );
    f[fv_index( n2, d, gx, gy, r )] = f[fv_index( n2, m[0], m[1], m[2], r )];
}

// compute_dt_stable (fct_advection_diffusion.hpp:193-254): min over cells of
// M / (inflow + diffusion); positive doubles order like their bit patterns
// the face orientation bits of every interior cell (the centre test of inward_faces)
__global__ void __launch_bounds__( kFvThreads ) orient_kernel( FvGeom G, uint8_t* bits )
{
    int d, x, y, r;
    if ( !cell_of_thread( G.N, d, x, y, r ) )
        return;
    bits[fv_index( G.N + 2, d, x, y, r )] = uint8_t( inward_faces( G, d, x, y, r ) );
}

// The geometry and face fluxes of a run of cells in x (the sums above): the velocity at the four nodes of the
// upper x face and the face's flux and vector stay for the next cell, whose lower x face it is, so a cell after the
// first loads 12 node values instead of 24 and forms 7 of the 8 wedge faces.
template < bool DIFFUSION >
struct FvWalk
{
    double h, hb, ht, b6, t6, rs, b2, t2; // h; h R_b, h R_t, r1^2 / 6, r2^2 / 6; h (r(-g) + r(g)), r1^2 / 2, r2^2 / 2
    double u[2][2][3];                    // lower x nodes: [y][bottom, top][component]
    double face, S[3];                    // upper x face of the cell before, seen from there

    __device__ __forceinline__ void plane( const FvGeom& G, int d, int x, int y, int r, double ( &v )[2][2][3] ) const
    {
        const int      n1 = G.N + 1;
        const unsigned id = unsigned( ( ( d * n1 + x ) * n1 + y ) ) * n1 + r;
#pragma unroll
        for ( int c = 0; c < 3; ++c )
        {
            const double* const p = G.vel.p[c] + id;
            v[0][0][c] = p[0], v[0][1][c] = p[1], v[1][0][c] = p[n1], v[1][1][c] = p[n1 + 1];
        }
    }
    // flux and vector of the quad over the nodes a, b with the lateral vector n
    __device__ __forceinline__ double quad( const double* n, const double ( &a )[2][3], const double ( &b )[2][3], double* s ) const
    {
        double f = 0.0;
#pragma unroll
        for ( int c = 0; c < 3; ++c )
        {
            f += n[c] * ( hb * ( a[0][c] + b[0][c] ) + ht * ( a[1][c] + b[1][c] ) );
            if ( DIFFUSION )
                s[c] = rs * n[c];
        }
        return f;
    }
    // cell (x, y, r), x the first of the run
    __device__ __forceinline__ void begin( const FvGeom& G, int d, int x, int y, int r )
    {
        const double r1 = G.radii[d * ( G.N + 1 ) + r - 1], r2 = G.radii[d * ( G.N + 1 ) + r], g = 0.5773502691896258;
        h = 0.5 * ( r2 - r1 );
        const double rm = r1 + h * ( 1.0 - g ), rp = r1 + h * ( 1.0 + g );
        hb = h * ( 0.25 * ( rm * ( 1.0 + g ) + rp * ( 1.0 - g ) ) ), ht = h * ( 0.25 * ( rm * ( 1.0 - g ) + rp * ( 1.0 + g ) ) );
        rs = h * ( rm + rp ), b6 = r1 * r1 / 6.0, t6 = r2 * r2 / 6.0, b2 = 0.5 * r1 * r1, t2 = 0.5 * r2 * r2;
        plane( G, d, x - 1, y - 1, r - 1, u );
        const Triangle< double > t( G.table, G.N, d, x - 1, y - 1, 0 );
        face = quad( t.b1, u[0], u[1], S );
        if ( G.orient[fv_index( G.N + 2, d, x, y, r )] & 1u )
            turn( face, S );
        turn( face, S ); // as the cell before would see it
    }
    __device__ __forceinline__ static void turn( double& f, double* s )
    {
        f = -f;
        if ( DIFFUSION )
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                s[c] = -s[c];
    }
    __device__ __forceinline__ void cell( const FvGeom& G, int d, int x, int y, int r, double ( &beta )[6], double& iM,
                                          double ( &Sf )[6][3] )
    {
        const unsigned bits = G.orient[fv_index( G.N + 2, d, x, y, r )];
        double         v[2][2][3];
        plane( G, d, x, y - 1, r - 1, v );
        const Triangle< double > t0( G.table, G.N, d, x - 1, y - 1, 0 ), t1( G.table, G.N, d, x - 1, y - 1, 1 );
        const double             n0[3] = { -t0.b2[0], -t0.b2[1], -t0.b2[2] }, n1[3] = { -t1.b2[0], -t1.b2[1], -t1.b2[2] };
        beta[0] = face;
        if ( DIFFUSION )
#pragma unroll
            for ( int c = 0; c < 3; ++c )
                Sf[0][c] = S[c];
        turn( beta[0], Sf[0] );
        beta[1] = quad( t1.b1, v[1], v[0], Sf[1] );
        beta[2] = quad( n0, u[0], v[0], Sf[2] );
        beta[3] = quad( n1, v[1], u[1], Sf[3] );
        double f[2][2] = { { 0.0, 0.0 }, { 0.0, 0.0 } };
#pragma unroll
        for ( int c = 0; c < 3; ++c )
        {
#pragma unroll
            for ( int k = 0; k < 2; ++k )
            {
                const double m = u[1][k][c] + v[0][k][c]; // the edge both wedges share
                f[k][0] += t0.v[c] * ( u[0][k][c] + m );
                f[k][1] += t1.v[c] * ( v[1][k][c] + m );
            }
            if ( DIFFUSION )
                Sf[4][c] = b2 * ( t0.v[c] + t1.v[c] ), Sf[5][c] = t2 * ( t0.v[c] + t1.v[c] );
        }
        beta[4] = b6 * ( f[0][0] + f[0][1] ), beta[5] = t6 * ( f[1][0] + f[1][1] );
        iM = fv_inverse_volume( G.table, G.N, d, x - 1, y - 1, r - 1 );
#pragma unroll
        for ( int n = 1; n < 6; ++n )
            if ( bits >> n & 1u )
                turn( beta[n], Sf[n] );
        face = beta[1];
#pragma unroll
        for ( int c = 0; c < 3; ++c )
        {
            if ( DIFFUSION )
                S[c] = Sf[1][c];
#pragma unroll
            for ( int k = 0; k < 2; ++k )
                u[0][k][c] = v[0][k][c], u[1][k][c] = v[1][k][c];
        }
    }
};

// The kernels of a step march: a thread owns a (y, r) and takes `run` cells in x, so what it reads of the x
// neighbours (and in FvWalk forms of the shared face) comes from the cell before, and a block holds several y of 32
// cells in r, so most of the y neighbours come from L1.  With one cell per thread the limiter and the correction
// read each plane about twice from L2 and were bound by that, and the other two loaded every node and formed every
// x face twice.  Level 7: limiter 306 -> 255 us, correction 351 -> 270 us, predictor 625 -> 540 us, dt 511 -> 440 us.
// The run leaves at least 1,024 threads per SM (step at level 5, runs of 1 / 2: 56.4 / 52.2 us; level 6, 2 / 4 / 8:
// 210 / 198 / 200 us) and gains nothing above 8 cells (level 7, 4 / 8 / 16 in the limiter and the correction: 1,289 /
// 1,269 / 1,267 us the step).
struct March
{
    int run, lanes, rows; // cells in x per thread; r lanes and y rows of a block
    unsigned blocks;
};

March march_shape( const tn_mesh* m )
{
    March           s;
    const long long cells = (long long) kDiamonds * m->N * m->N * m->N;
    s.run   = int( std::clamp( cells / ( 148LL * 1024 ), 1LL, 8LL ) );
    s.lanes = std::min( m->N, 32 );
    s.rows  = kFvThreads / s.lanes;
    s.blocks = unsigned( kDiamonds * ( ( m->N + s.run - 1 ) / s.run ) ) * unsigned( ( m->N + s.rows - 1 ) / s.rows ) *
               unsigned( m->N / s.lanes );
    return s;
}

// y and r of this thread in block b, its diamond and first x; false: no cell
__device__ __forceinline__ bool march_of_thread( int N, const March& s, unsigned b, int& d, int& x, int& y, int& r )
{
    const unsigned rb = unsigned( N / s.lanes ), yb = unsigned( ( N + s.rows - 1 ) / s.rows ), xb = unsigned( ( N + s.run - 1 ) / s.run );
    r = int( b % rb ) * s.lanes + int( threadIdx.x ) % s.lanes + 1, b /= rb;
    y = int( b % yb ) * s.rows + int( threadIdx.x ) / s.lanes + 1, b /= yb;
    x = int( b % xb ) * s.run + 1, d = int( b / xb );
    return y <= N;
}

// Blocks take the runs in turn and one atomic per block closes the minimum: one per warp on the single result cost
// as much as the geometry (level 7: 655,360 of them).
template < bool DIFFUSION >
__global__ void __launch_bounds__( kFvThreads, 4 ) dt_kernel( FvGeom G, March s, double kappa, unsigned long long* out )
{
    __shared__ double sh[kFvThreads / 32];
    const int         n2  = G.N + 2;
    double            dtc = 1e300;
    for ( unsigned b = blockIdx.x; b < s.blocks; b += gridDim.x )
    {
        int d, x, y, r;
        if ( !march_of_thread( G.N, s, b, d, x, y, r ) )
            continue;
        FvWalk< DIFFUSION > walk;
        walk.begin( G, d, x, y, r );
        for ( const int end = min( x + s.run, G.N + 1 ); x < end; ++x )
        {
            double beta[6], iM, S[6][3], lambda = 0.0;
            walk.cell( G, d, x, y, r, beta, iM, S );
            const size_t ci = fv_index( n2, d, x, y, r );
#pragma unroll
            for ( int n = 0; n < 6; ++n )
            {
                if ( beta[n] < 0 )
                    lambda -= beta[n];
                if ( DIFFUSION && kappa > 0 )
                {
                    const size_t cj  = fv_index( n2, d, x + kFvOff[n][0], y + kFvOff[n][1], r + kFvOff[n][2] );
                    double       den = 0.0, ss = 0.0;
                    for ( int a = 0; a < 3; ++a )
                    {
                        den += ( G.cen.p[a][cj] - G.cen.p[a][ci] ) * S[n][a];
                        ss += S[n][a] * S[n][a];
                    }
                    if ( den > 0 )
                        lambda += kappa * ss / den;
                }
            }
            dtc = fmin( dtc, lambda > 0 ? 1.0 / ( iM * lambda ) : 1e30 );
        }
    }
    for ( int off = 16; off > 0; off >>= 1 )
        dtc = fmin( dtc, __shfl_down_sync( 0xffffffffu, dtc, off ) );
    if ( ( threadIdx.x & 31 ) == 0 )
        sh[threadIdx.x >> 5] = dtc;
    __syncthreads();
    if ( threadIdx.x == 0 )
    {
        for ( int w = 1; w < kFvThreads / 32; ++w )
            dtc = fmin( dtc, sh[w] );
        atomicMin( out, (unsigned long long) __double_as_longlong( dtc ) );
    }
}

// FCTPredictorKernel (fct_advection_diffusion.hpp:262-376); DIFFUSION: kappa != 0 (with 4 blocks per SM its spills cost
// more than the occupancy gives: level 7 step 1,765 -> 1,809 us; 5 blocks without it: 1,196 -> 1,241 us)
template < bool DIFFUSION >
__global__ void __launch_bounds__( kFvThreads, DIFFUSION ? 3 : 4 )
    predictor_kernel( FvGeom G, March s, const double* __restrict__ T, double* __restrict__ TL, double* __restrict__ g,
                      double dt, double kappa, const double* __restrict__ src, int subtract_divergence )
{
    int d, x, y, r;
    if ( !march_of_thread( G.N, s, blockIdx.x, d, x, y, r ) )
        return;
    const int           n2 = G.N + 2, sx = n2 * n2, end = min( x + s.run, G.N + 1 );
    const size_t        nf = size_t( kDiamonds ) * n2 * sx; // g holds 3 planes of nf (SoA)
    size_t              i  = fv_index( n2, d, x, y, r );
    double              below = T[i - sx], Ti = T[i];
    FvWalk< DIFFUSION > walk;
    walk.begin( G, d, x, y, r );
    for ( ; x < end; ++x, i += sx )
    {
        const double above = T[i + sx], Tn[6] = { below, above, T[i - n2], T[i + n2], T[i - 1], T[i + 1] };
        double       beta[6], iM, S[6][3], lo_diag = 0.0, lo_update = 0.0, bsum = 0.0;
        walk.cell( G, d, x, y, r, beta, iM, S );
#pragma unroll
        for ( int n = 0; n < 6; ++n )
        {
            const size_t j  = n / 2 == 0 ? ( n % 2 ? i + sx : i - sx ) : ( n / 2 == 1 ? ( n % 2 ? i + n2 : i - n2 ) : ( n % 2 ? i + 1 : i - 1 ) );
            const double Tj = Tn[n];
            if ( beta[n] >= 0 )
                lo_diag += beta[n];
            else
                lo_update += beta[n] * Tj;
            bsum += beta[n];
            if ( DIFFUSION ) // the diffusion term; zero without diffusivity (no centre loads)
            {
                double den = 0.0, ss = 0.0;
                for ( int a = 0; a < 3; ++a )
                {
                    den += ( G.cen.p[a][j] - G.cen.p[a][i] ) * S[n][a];
                    ss += S[n][a] * S[n][a];
                }
                const double dc = kappa * ( ss / den );
                lo_diag += dc;
                lo_update -= dc * Tj;
            }
            // face 2a towards the lower neighbour in direction a; the last cell's upper face goes to the ghost cell
            if ( n % 2 == 0 )
                g[( n / 2 ) * nf + i] = fabs( beta[n] ) * 0.5 * ( Ti - Tj );
            else if ( ( n == 1 ? x : ( n == 3 ? y : r ) ) == G.N )
                g[( n / 2 ) * nf + j] = fabs( beta[n] ) * 0.5 * ( Tj - Ti );
        }
        if ( subtract_divergence )
            lo_diag -= bsum;
        double tl = Ti - ( dt * iM ) * ( lo_diag * Ti + lo_update );
        if ( src )
            tl += dt * src[i];
        TL[i] = tl;
        below = Ti, Ti = above;
    }
}

// apply_dirichlet_bcs (fv/hex/helpers.hpp:26-64): thread per lateral column
__global__ void dirichlet_kernel( int N, double* __restrict__ T, double t_cmb, double t_surf, int cmb, int surf )
{
    const long long t = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    if ( t >= (long long) kDiamonds * N * N )
        return;
    const int y = int( t % N ) + 1, x = int( ( t / N ) % N ) + 1, d = int( t / ( (long long) N * N ) );
    const int n2 = N + 2;
    if ( cmb )
        T[fv_index( n2, d, x, y, 1 )] = T[fv_index( n2, d, x, y, 0 )] = t_cmb;
    if ( surf )
        T[fv_index( n2, d, x, y, N )] = T[fv_index( n2, d, x, y, N + 1 )] = t_surf;
}

// FCTLimiterKernel (fct_advection_diffusion.hpp:486-531); the six antidiffusive fluxes of a cell are dt / M times its
// faces' g
__global__ void __launch_bounds__( kFvThreads )
    limiter_kernel( FvGeom G, March s, const double* __restrict__ TL, const double* __restrict__ g, double dt,
                    double* __restrict__ Rp, double* __restrict__ Rm )
{
    int d, x, y, r;
    if ( !march_of_thread( G.N, s, blockIdx.x, d, x, y, r ) )
        return;
    const int    n2 = G.N + 2, sx = n2 * n2, end = min( x + s.run, G.N + 1 );
    const size_t nf = size_t( kDiamonds ) * n2 * sx;
    size_t       i  = fv_index( n2, d, x, y, r );
    double       below = TL[i - sx], ti = TL[i], gx = g[i];
    for ( ; x < end; ++x, i += sx )
    {
        const double* const gy = g + nf + i;
        const double* const gr = gy + nf;
        const double        above = TL[i + sx], gu = g[i + sx];
        const double        tn[4] = { TL[i - n2], TL[i + n2], TL[i - 1], TL[i + 1] };
        const double        scale = dt * fv_inverse_volume( G.table, G.N, d, x - 1, y - 1, r - 1 );
        const double        f[6] = { scale * gx, -scale * gu, scale * gy[0], -scale * gy[n2], scale * gr[0], -scale * gr[1] };
        double              Pp = 0.0, Pm = 0.0;
#pragma unroll
        for ( int n = 0; n < 6; ++n )
            if ( f[n] > 0 )
                Pp += f[n];
            else
                Pm += f[n];
        const double tmax = fmax( fmax( fmax( fmax( fmax( fmax( ti, below ), above ), tn[0] ), tn[1] ), tn[2] ), tn[3] );
        const double tmin = fmin( fmin( fmin( fmin( fmin( fmin( ti, below ), above ), tn[0] ), tn[1] ), tn[2] ), tn[3] );
        Rp[i] = Pp > 0 ? fmin( 1.0, ( tmax - ti ) / Pp ) : 1.0;
        Rm[i] = Pm < 0 ? fmin( 1.0, ( tmin - ti ) / Pm ) : 1.0;
        below = ti, ti = above, gx = gu;
    }
}

// FCTCorrectionKernel (fct_advection_diffusion.hpp:605-650)
__global__ void __launch_bounds__( kFvThreads )
    correction_kernel( FvGeom G, March s, const double* __restrict__ TL, const double* __restrict__ g, double dt,
                       const double* __restrict__ Rp, const double* __restrict__ Rm, double* __restrict__ T )
{
    int d, x, y, r;
    if ( !march_of_thread( G.N, s, blockIdx.x, d, x, y, r ) )
        return;
    const int    n2 = G.N + 2, sx = n2 * n2, end = min( x + s.run, G.N + 1 );
    const size_t nf = size_t( kDiamonds ) * n2 * sx;
    size_t       i  = fv_index( n2, d, x, y, r );
    double       gx = g[i], pb = Rp[i - sx], mb = Rm[i - sx], rp = Rp[i], rm = Rm[i];
    for ( ; x < end; ++x, i += sx )
    {
        const double* const gy = g + nf + i;
        const double* const gr = gy + nf;
        const double        gu = g[i + sx], pa = Rp[i + sx], ma = Rm[i + sx];
        const double        scale = dt * fv_inverse_volume( G.table, G.N, d, x - 1, y - 1, r - 1 );
        const double        f[6] = { scale * gx, -scale * gu, scale * gy[0], -scale * gy[n2], scale * gr[0], -scale * gr[1] };
        const size_t        j[4] = { i - n2, i + n2, i - 1, i + 1 };
        double              corr = ( f[0] > 0 ? fmin( rp, mb ) : fmin( rm, pb ) ) * f[0];
        corr += ( f[1] > 0 ? fmin( rp, ma ) : fmin( rm, pa ) ) * f[1];
#pragma unroll
        for ( int n = 0; n < 4; ++n )
            corr += ( f[2 + n] > 0 ? fmin( rp, Rm[j[n]] ) : fmin( rm, Rp[j[n]] ) ) * f[2 + n];
        T[i] = TL[i] + corr;
        pb = rp, mb = rm, rp = pa, rm = ma, gx = gu;
    }
}

// Zeroes the ghost cells (all those outside 1..N in some direction) of nf fields: the first and last cell of every
// column, one thread per column, and whole ghost columns, one thread per cell of them (blocks after the first
// col_blocks).
__global__ void __launch_bounds__( 256 ) fv_zero_ghost_kernel( int N, Ptr3< double > f, int nf, unsigned col_blocks )
{
    const unsigned n2 = unsigned( N ) + 2, cols = unsigned( kDiamonds ) * n2 * n2, ring = 4 * ( n2 - 1 );
    if ( blockIdx.x < col_blocks )
    {
        const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
        if ( c < cols )
            for ( int k = 0; k < nf; ++k )
                f.at( k )[size_t( c ) * n2] = f.at( k )[size_t( c ) * n2 + n2 - 1] = 0.0;
        return;
    }
    const unsigned t = ( blockIdx.x - col_blocks ) * blockDim.x + threadIdx.x, e = t / n2, r = t % n2;
    if ( e >= unsigned( kDiamonds ) * ring )
        return;
    // column e % ring around the diamond: sides x = 0, y = n2 - 1, x = n2 - 1, y = 0 of n2 - 1 columns each
    const unsigned d = e / ring, s = e % ring / ( n2 - 1 ), i = e % ( n2 - 1 );
    const unsigned x = s == 0 ? 0u : ( s == 1 ? i : ( s == 2 ? n2 - 1 : n2 - 1 - i ) );
    const unsigned y = s == 0 ? i : ( s == 1 ? n2 - 1 : ( s == 2 ? n2 - 1 - i : 0u ) );
    for ( int k = 0; k < nf; ++k )
        f.at( k )[( ( size_t( d ) * n2 + x ) * n2 + y ) * n2 + r] = 0.0;
}

size_t fv_size( const tn_mesh* m )
{
    const size_t n2 = size_t( m->N ) + 2;
    return size_t( kDiamonds ) * n2 * n2 * n2;
}

unsigned cell_blocks( const tn_mesh* m )
{
    return unsigned( ( (long long) kDiamonds * m->N * m->N * m->N + kFvThreads - 1 ) / kFvThreads );
}

// lateral ghosts of one field, or of two in one launch
int ghost_update( const tn_mesh* m, double* f, cudaStream_t st, double* f2 = nullptr )
{
    const long long n = (long long) kDiamonds * 4 * m->N * m->N;
    fv_ghost_kernel<<< dim3( unsigned( ( n + 255 ) / 256 ), f2 ? 2 : 1 ), 256, 0, st >>>( m->N, m->d_fv_ghost,
                                                                                         Ptr3< double >{ { f, f2, nullptr } } );
    TN_LAUNCH_CHECK();
    return TN_OK;
}

// The face orientation bits of the mesh, from its own cell centres (compute_cell_centers, the centres
// tn_fv_cell_centers_f64 gives), built on the first FCT call of the mesh: the orientation is geometry, so the
// per-step kernels read one byte per cell instead of the six neighbours' centres.
const uint8_t* fv_orientation( const tn_mesh* m, const double* table, cudaStream_t st )
{
    tn_mesh*                      mm = const_cast< tn_mesh* >( m );
    std::lock_guard< std::mutex > lock( mm->geom_mutex );
    if ( !mm->d_fv_orient )
    {
        const size_t nf = fv_size( m );
        double*      c  = nullptr;
        uint8_t*     b  = nullptr;
        if ( cudaMalloc( &c, 3 * nf * sizeof( double ) ) != cudaSuccess )
            return nullptr;
        if ( cudaMalloc( &b, nf ) != cudaSuccess )
        {
            cudaFree( c );
            return nullptr;
        }
        bool ok = cudaMemsetAsync( c, 0, 3 * nf * sizeof( double ), st ) == cudaSuccess &&
                  cudaMemsetAsync( b, 0, nf, st ) == cudaSuccess;
        Ptr3< double > cp{ { c, c + nf, c + 2 * nf } };
        if ( ok )
        {
            cell_centers_kernel<<< cell_blocks( m ), kFvThreads, 0, st >>>( m->N, m->d_coords, m->d_radii, cp );
            ok = cudaGetLastError() == cudaSuccess;
        }
        for ( int a = 0; a < 3 && ok; ++a )
            ok = ghost_update( m, c + a * nf, st ) == TN_OK;
        if ( ok )
        {
            FvGeom G{};
            G.N = m->N, G.table = table, G.radii = m->d_radii;
            G.cen    = Ptr3< const double >{ { c, c + nf, c + 2 * nf } };
            G.orient = nullptr;
            orient_kernel<<< cell_blocks( m ), kFvThreads, 0, st >>>( G, b );
            ok = cudaGetLastError() == cudaSuccess && cudaStreamSynchronize( st ) == cudaSuccess;
        }
        cudaFree( c );
        if ( !ok )
        {
            cudaFree( b );
            return nullptr;
        }
        mm->d_fv_orient = b;
    }
    return mm->d_fv_orient;
}

int make_geom( const tn_mesh* m, const double* const* vel, const double* const* cen, FvGeom& G, cudaStream_t st )
{
    TN_CHECK_ARG( vel && cen, "fct: null field list" );
    for ( int a = 0; a < 3; ++a )
    {
        TN_CHECK_ARG( vel[a] && cen[a], "fct: null field pointer" );
        G.vel.p[a] = vel[a];
        G.cen.p[a] = cen[a];
    }
    G.N = m->N, G.table = triangle_table< double >( m ), G.radii = m->d_radii;
    G.orient = fv_orientation( m, G.table, st );
    if ( !G.orient )
    {
        set_error( "fct: building the face orientation of the mesh failed" );
        return TN_ERR_CUDA;
    }
    return TN_OK;
}

}  // namespace

}  // namespace tn

using namespace tn;

extern "C" int tn_fv_field_size( const tn_mesh* m, size_t* n )
{
    TN_CHECK_ARG( m && n, "tn_fv_field_size: null argument" );
    *n = fv_size( m );
    return TN_OK;
}

extern "C" int tn_fct_workspace_size( const tn_mesh* m, size_t* n )
{
    TN_CHECK_ARG( m && n, "tn_fct_workspace_size: null argument" );
    *n = 9 * fv_size( m );
    return TN_OK;
}

extern "C" int tn_fv_ghost_update_f64( const tn_mesh* m, double* field, void* s )
{
    TN_CHECK_ARG( m && field, "tn_fv_ghost_update_f64: null argument" );
    return ghost_update( m, field, as_stream( s ) );
}

extern "C" int tn_fv_cell_centers_f64( const tn_mesh* m, double* const* centers, void* s )
{
    TN_CHECK_ARG( m && centers && centers[0] && centers[1] && centers[2], "tn_fv_cell_centers_f64: null argument" );
    cudaStream_t st = as_stream( s );
    Ptr3< double > c{ { centers[0], centers[1], centers[2] } };
    for ( int a = 0; a < 3; ++a )
        TN_CUDA_TRY( cudaMemsetAsync( centers[a], 0, sizeof( double ) * fv_size( m ), st ) );
    cell_centers_kernel<<< cell_blocks( m ), kFvThreads, 0, st >>>( m->N, m->d_coords, m->d_radii, c );
    TN_LAUNCH_CHECK();
    for ( int a = 0; a < 3; ++a )
    {
        int rc = ghost_update( m, centers[a], st );
        if ( rc )
            return rc;
    }
    return TN_OK;
}

extern "C" int tn_fct_dt_stable_f64( const tn_mesh* m, const double* const* vel, const double* const* centers,
                                     double diffusivity, double* dt_stable, void* s )
{
    TN_CHECK_ARG( m && dt_stable, "tn_fct_dt_stable_f64: null argument" );
    FvGeom G{};
    int    rc;
    cudaStream_t st = as_stream( s );
    if ( ( rc = make_geom( m, vel, centers, G, st ) ) )
        return rc;
    unsigned long long* slot = reinterpret_cast< unsigned long long* >( m->d_red_result + 12 );
    // bytes 0x7f: 1.4e306, above every candidate
    TN_CUDA_TRY( cudaMemsetAsync( slot, 0x7f, sizeof( double ), st ) );
    const March    march  = march_shape( m );
    const unsigned blocks = std::min( march.blocks, 148u * 16u );
    if ( diffusivity != 0.0 )
        dt_kernel< true ><<< blocks, kFvThreads, 0, st >>>( G, march, diffusivity, slot );
    else
        dt_kernel< false ><<< blocks, kFvThreads, 0, st >>>( G, march, diffusivity, slot );
    TN_LAUNCH_CHECK();
    TN_CUDA_TRY( cudaMemcpyAsync( dt_stable, slot, sizeof( double ), cudaMemcpyDeviceToHost, st ) );
    TN_CUDA_TRY( cudaStreamSynchronize( st ) );
    return TN_OK;
}

extern "C" int tn_fct_apply_dirichlet_f64( const tn_mesh* m, double* T, const tn_fct_dirichlet* bcs, void* s )
{
    TN_CHECK_ARG( m && T && bcs, "tn_fct_apply_dirichlet_f64: null argument" );
    const long long n = (long long) kDiamonds * m->N * m->N;
    dirichlet_kernel<<< unsigned( ( n + 255 ) / 256 ), 256, 0, as_stream( s ) >>>(
        m->N, T, bcs->T_cmb, bcs->T_surface, bcs->apply_cmb, bcs->apply_surface );
    TN_LAUNCH_CHECK();
    return TN_OK;
}

extern "C" int tn_fct_step_f64( const tn_mesh* m, double* T, const double* const* vel, const double* const* centers,
                                double dt, double diffusivity, const double* source, int subtract_divergence,
                                const tn_fct_dirichlet* bcs, double* workspace, void* s )
{
    TN_CHECK_ARG( m && T && workspace, "tn_fct_step_f64: null argument" );
    FvGeom G{};
    int    rc;
    cudaStream_t st = as_stream( s );
    if ( ( rc = make_geom( m, vel, centers, G, st ) ) )
        return rc;
    const size_t nf = fv_size( m );
    double *     TL = workspace, *g = workspace + nf, *Rp = workspace + 7 * nf, *Rm = workspace + 8 * nf;
    // the radial ghosts enter as zeros where no boundary treatment sets them; every interior cell is written below
    const unsigned n2 = unsigned( m->N ) + 2, col_blocks = ( unsigned( kDiamonds ) * n2 * n2 + 255u ) / 256u;
    const unsigned ring_blocks = ( unsigned( kDiamonds ) * 4u * ( n2 - 1 ) * n2 + 255u ) / 256u;
    fv_zero_ghost_kernel<<< col_blocks + ring_blocks, 256, 0, st >>>( m->N, Ptr3< double >{ { TL, Rp, Rm } }, 3, col_blocks );
    TN_LAUNCH_CHECK();
    // predictor (fct_advection_diffusion.hpp:384-433) on T with fresh lateral ghosts
    if ( ( rc = ghost_update( m, T, st ) ) )
        return rc;
    const March march = march_shape( m );
    if ( diffusivity != 0.0 )
        predictor_kernel< true ><<< march.blocks, kFvThreads, 0, st >>>( G, march, T, TL, g, dt, diffusivity, source,
                                                                         subtract_divergence );
    else
        predictor_kernel< false ><<< march.blocks, kFvThreads, 0, st >>>( G, march, T, TL, g, dt, diffusivity, source,
                                                                          subtract_divergence );
    TN_LAUNCH_CHECK();
    if ( bcs && ( rc = tn_fct_apply_dirichlet_f64( m, TL, bcs, s ) ) )
        return rc;
    // limiter (:539-566) and correction (:658-680)
    if ( ( rc = ghost_update( m, TL, st ) ) )
        return rc;
    limiter_kernel<<< march.blocks, kFvThreads, 0, st >>>( G, march, TL, g, dt, Rp, Rm );
    TN_LAUNCH_CHECK();
    if ( ( rc = ghost_update( m, Rp, st, Rm ) ) )
        return rc;
    correction_kernel<<< march.blocks, kFvThreads, 0, st >>>( G, march, TL, g, dt, Rp, Rm, T );
    TN_LAUNCH_CHECK();
    return TN_OK;
}
