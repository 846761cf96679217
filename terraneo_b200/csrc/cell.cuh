// Factored wedge geometry and the scatter of cell contributions, shared by the
// kernels that run one thread per cell (r fastest: the lanes of a warp are
// consecutive radial cells of one column from N = 32 on).
//
// For the wedge map x = r(zeta) (p0 + xi a + eta b), a = p1 - p0, b = p2 - p0,
// with h = (r2 - r1) / 2, rho = r(zeta) / h and
//     beta_1 = b x p0, beta_2 = p0 x a, v = a x b, D = v . p0,
//     beta_0 = v - beta_1 - beta_2,
// the physical gradient of the shape function of node n (lateral vertex m, side
// sign s_n = -+1/2, radial factor nr_n(zeta) = (1 -+ zeta)/2) is
//     g_n = ( nr_n u_m + s_n lat_m rho v ) / (D r),  u_m = beta_m - lat_m v,
// and |det J| = r^2 h |D|.  A quadrature point's k |det J| g_i (x) g_j therefore
// needs no Jacobian and no inverse: k h / |D| times products of u_m, v and rho.
// beta_1, beta_2, v and 1 / D depend on the triangle only and are tabulated once
// per mesh (10 values per wedge; 80 bytes, read by all lanes of a warp at once),
// with h, r1 / h and r1 of every layer behind them.  These kernels are bound by
// instruction issue, so what all of them share counts: N is a power of two, so a
// thread's cell comes from shifts, nodes are 32-bit indices, and the divisions by
// h and D are in the table.
#pragma once

#include "common.cuh"
#include "wedge.cuh"

namespace tn {

constexpr int kTriangle = 10; // beta_1, beta_2, v, 1 / D

// The mesh's table in the precision of T (formed with the mesh, mesh.cu: on a first apply its allocation took 0.3 to
// 2 ms, more than the apply).  [diamond][x][y][wedge][kTriangle], then h, r1 / h and r1 of the N layers, then the
// inverse volumes of the FV cells as a lateral factor per (diamond, x, y) times a radial one per layer.
template < typename T >
const T* triangle_table( const tn_mesh* m )
{
    if constexpr ( sizeof( T ) == 8 )
        return m->d_triangles;
    else
        return m->d_triangles32;
}

template < typename T >
struct Triangle
{
    T b1[3], b2[3], v[3], iD;
    __device__ __forceinline__ Triangle( const T* __restrict__ table, int N, int d, int x, int y, int w )
    {
        const T* p = table + ( ( ( size_t( d ) * N + x ) * N + y ) * 2 + w ) * kTriangle;
        T        q[kTriangle];
#pragma unroll
        for ( int i = 0; i < kTriangle / 2; ++i )
        {
            if constexpr ( sizeof( T ) == 8 )
            {
                const double2 e = reinterpret_cast< const double2* >( p )[i];
                q[2 * i] = e.x, q[2 * i + 1] = e.y;
            }
            else
            {
                const float2 e = reinterpret_cast< const float2* >( p )[i];
                q[2 * i] = e.x, q[2 * i + 1] = e.y;
            }
        }
#pragma unroll
        for ( int a = 0; a < 3; ++a )
            b1[a] = q[a], b2[a] = q[3 + a], v[a] = q[6 + a];
        iD = q[9];
    }
};

// h = (r2 - r1) / 2, r1 / h and r1 of layer r; the inverse volume of FV cell (d, x, y, r) of the cells' numbering
template < typename T >
__device__ __forceinline__ T layer_h( const T* __restrict__ table, int N, int r )
{
    return table[size_t( 2 * kDiamonds * kTriangle ) * N * N + r];
}
template < typename T >
__device__ __forceinline__ T layer_q( const T* __restrict__ table, int N, int r )
{
    return table[size_t( 2 * kDiamonds * kTriangle ) * N * N + N + r];
}
template < typename T >
__device__ __forceinline__ T layer_r( const T* __restrict__ table, int N, int r )
{
    return table[size_t( 2 * kDiamonds * kTriangle ) * N * N + 2 * N + r];
}
__device__ __forceinline__ double fv_inverse_volume( const double* __restrict__ table, int N, int d, int x, int y, int r )
{
    const double* p = table + size_t( 2 * kDiamonds * kTriangle ) * N * N + 3 * N;
    return p[( size_t( d ) * N + x ) * N + y] * p[size_t( kDiamonds ) * N * N + r];
}

template < typename T >
__device__ __forceinline__ T dot3( const T a[3], const T b[3] )
{
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// gradient of the node at lateral vertex m on side s = -1 (bottom) or 1 (top) at a point, times D r:
// nr u_m + s / 2 lat rho v
template < typename T >
__device__ __forceinline__ void scaled_gradient( const Triangle< T >& G, int m, T s, T xi, T eta, T zeta, T rho, T g[3] )
{
    const T lat = m == 0 ? T( 1 ) - xi - eta : ( m == 1 ? xi : eta );
    const T nr  = T( 0.5 ) * ( T( 1 ) + s * zeta );
#pragma unroll
    for ( int a = 0; a < 3; ++a )
    {
        const T beta = m == 0 ? G.v[a] - G.b1[a] - G.b2[a] : ( m == 1 ? G.b1[a] : G.b2[a] );
        g[a]         = nr * ( beta - lat * G.v[a] ) + T( 0.5 ) * s * lat * rho * G.v[a];
    }
}

// 3x2 Felippa rule: lateral points (2/3, 1/6), (1/6, 2/3), (1/6, 1/6), zeta = -+1/sqrt(3), weight 1/6 each
constexpr double kFelippaZ = 0.5773502691896257;
__host__ __device__ constexpr double felippa_xi( int q ) { return q % 3 == 0 ? 0.6666666666666666 : 0.1666666666666667; }
__host__ __device__ constexpr double felippa_eta( int q ) { return q % 3 == 1 ? 0.6666666666666666 : 0.1666666666666667; }
constexpr double kFelippaW = 1.0 / 6.0;

// The cell of thread t, r fastest; false past the last cell (the coordinates are then those of the last one, so that
// such a thread can take part in its warp's shuffles).
__device__ __forceinline__ bool cell_of( long long t, int N, int& d, int& x, int& y, int& r )
{
    const int       L     = 31 - __clz( N ); // N = 2^L
    const long long cells = (long long) kDiamonds << ( 3 * L );
    const bool      in    = t < cells;
    const unsigned  c     = unsigned( in ? t : cells - 1 ), m = unsigned( N ) - 1u; // at most 10 * 512^3 cells
    r = int( c & m ), y = int( c >> L & m ), x = int( c >> ( 2 * L ) & m ), d = int( c >> ( 3 * L ) );
    return in;
}
// the lateral cell c of [0, 10 N^2)
__device__ __forceinline__ void lateral_cell_of( unsigned c, int N, int& d, int& x, int& y )
{
    const int      L = 31 - __clz( N );
    const unsigned m = unsigned( N ) - 1u;
    y = int( c & m ), x = int( c >> L & m ), d = int( c >> ( 2 * L ) );
}

// lower nodes (level r) of a cell's columns 0 = (x, y), 1 = (x + 1, y), 2 = (x, y + 1), 3 = (x + 1, y + 1); there are
// fewer than 2^32 nodes
__device__ __forceinline__ void cell_nodes( int n1, int d, int x, int y, int r, unsigned ( &node )[4] )
{
    const unsigned n = unsigned( n1 );
    node[0] = ( ( unsigned( d ) * n + unsigned( x ) ) * n + unsigned( y ) ) * n + unsigned( r );
    node[1] = node[0] + n * n, node[2] = node[0] + n, node[3] = node[1] + n;
}

// the columns (of cell_nodes) under the three vertices of wedge w; w need not be a compile-time value
__device__ __forceinline__ void wedge_columns( const unsigned ( &node )[4], int w, unsigned ( &v )[3] )
{
    v[0] = w ? node[3] : node[0], v[1] = w ? node[2] : node[1], v[2] = w ? node[1] : node[2];
}

// Work on one side (lower or upper nodes) of one wedge of the cells of a layer, the form of the boundary rows: item t of
// 4 x 10 N^2 is (side, wedge, lateral cell), so that each thread's serial work is short (at coarse levels the longest
// thread is the kernel's time).  A layer-0 cell has its boundary nodes below (top false), a layer N - 1 cell above.
constexpr unsigned boundary_items( int N ) { return 4u * kDiamonds * unsigned( N ) * unsigned( N ); }
__device__ __forceinline__ bool boundary_item( unsigned t, int N, int& d, int& x, int& y, int& r, int& w, bool& top )
{
    const unsigned cols = unsigned( kDiamonds ) * N * N;
    if ( t >= 4u * cols )
        return false;
    top = t >= 2u * cols, w = t >= 2u * cols ? t >= 3u * cols : t >= cols;
    r = top ? N - 1 : 0;
    lateral_cell_of( t % cols, N, d, x, y );
    return true;
}

// dst[c] = 0 for nc fields of n values, in one memset where the fields follow one another
template < typename T >
inline cudaError_t zero_fields( T* const* dst, int nc, size_t n, cudaStream_t st )
{
    for ( int c = 0, e; c < nc; c = e )
    {
        for ( e = c + 1; e < nc && dst[e] == dst[e - 1] + n; ++e )
            ;
        const cudaError_t rc = cudaMemsetAsync( dst[c], 0, size_t( e - c ) * n * sizeof( T ), st );
        if ( rc != cudaSuccess )
            return rc;
    }
    return cudaSuccess;
}

// Adds a cell's contributions to the lower (node r) and upper (node r + 1) end of one of its columns, NC components.
// The upper ones go to the lane above by shuffle where that lane holds the next cell of the column, so about half
// the atomics remain.  Called by all lanes of a warp; write_low / write_high false: that node's row is not written
// (by the cell itself; what the lane below hands over follows that lane's write_high).
template < typename T, int NC >
__device__ __forceinline__ void add_column( T* const* dst, unsigned node, int r, int N, bool in, bool write_low, bool write_high,
                                            const T ( &low )[NC], const T ( &high )[NC] )
{
    const int  lane       = int( threadIdx.x ) & 31;
    const bool from_below = lane > 0 && r > 0, own_top = lane == 31 || r == N - 1;
#pragma unroll
    for ( int c = 0; c < NC; ++c )
    {
        const T below = __shfl_up_sync( 0xffffffffu, high[c], 1 );
        const T v     = ( write_low ? low[c] : T( 0 ) ) + ( from_below ? below : T( 0 ) );
        if ( in && ( write_low || from_below ) )
            atomicAdd( dst[c] + node, v );
        if ( in && own_top && write_high )
            atomicAdd( dst[c] + node + 1, high[c] );
    }
}

}  // namespace tn
