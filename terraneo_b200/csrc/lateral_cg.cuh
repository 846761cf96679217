// Conjugate gradients on the separated operators of lateral.cuh (the Dirichlet
// Laplacian and the mass matrix, FP64), two kernels per iteration:
//   lateral_cg_kernel: p = r + beta p, ap = A p and <p, ap> in one pass: the tile
//     blocks form the new direction while they stage its operands (so it is never
//     read back), write it to the other of two direction fields and sum the
//     product while they write ap out (every term compensated where OP::kExactDot,
//     else plainly per thread); the halo is part of the apply;
//   tn_pcg_update: x, r, |r|, the stopping rule and beta (krylov.cu).
// The steps are those of tn_pcg_* (pcg.hpp:78-102 with z = r): every kernel returns
// at once when the stopping rule has fired, so the host runs ahead of the device
// and looks at the flag some steps later.  A step issued after the rule has fired costs
// its two launches, 9 us at level 6 (45 us when it read its operands and left out the
// writes only); a step of a solve takes 0.5 % longer for waiting on the flag first at
// level 6, no longer at level 5.
// Per iteration: the Laplacian at level 5 38 us of kernels (apply, halo, product,
// update, direction; 61 us with the gaps) -> 24 us, the mass matrix at level 6 350 us
// with two host reads -> 83 us.
#pragma once

#include "lateral.cuh"

namespace tn {

template < typename OP >
__global__ void __launch_bounds__( kLateralThreads, 4 ) lateral_cg_kernel( LateralParams< double > P, LateralCG cg )
{
    extern __shared__ double lateral_smem[];
    if ( cg.state[4] != 0.0 ) // done
        return;
    const double beta = cg.state[3];
    Neumaier     dot;
    if ( blockIdx.x < P.edge_blocks )
        lateral_edge< OP, true >( P, cg, beta, blockIdx.x, dot );
    else
        lateral_tile< OP, true >( P, cg, beta, blockIdx.x - P.edge_blocks, lateral_smem, dot );
    block_sum_finish< 1 >( &dot, cg.partials, cg.counter, cg.state + 1 ); // pap
}

// steps after which the residual history of tn_pcg_* (which nothing reads here) is written over from its start
constexpr int kLateralHistory = 4096;

// doubles of the work array of lateral_cg besides its four fields r, p, p', ap
template < typename OP >
size_t lateral_cg_scratch( const tn_mesh* m, int max_iterations )
{
    LateralParams< double > P{};
    return 2 * size_t( lateral_shape( m, true, P ) ) + 2 + 8 + size_t( std::clamp( max_iterations, 0, kLateralHistory ) ) + 1;
}

// Solves A x = b from x's values; P: the operator's tables and layer modes.  fields: r, p, p', ap (stored nodes each);
// scratch: lateral_cg_scratch doubles.  Returns after the solve: iterations and relative residual as tn_pcg_* count them.
template < typename OP >
int lateral_cg( const tn_mesh* m, LateralParams< double > P, const double* b, double* x, double* const fields[4], double* scratch,
                int max_iterations, double rtol, double atol, int* iterations, double* relres, cudaStream_t st )
{
    // the scratch goes back to its owner on every way out, so nothing may still be running on it
    struct StreamEnd
    {
        cudaStream_t s;
        ~StreamEnd() { cudaStreamSynchronize( s ); }
    } const end{ st };
    double *       r = fields[0], *p[2] = { fields[1], fields[2] }, *ap = fields[3];
    const unsigned blocks = lateral_shape( m, true, P );
    LateralCG      cg{};
    cg.r = r, cg.partials = scratch, cg.counter = reinterpret_cast< unsigned int* >( scratch + 2 * size_t( blocks ) );
    cg.state = scratch + 2 * size_t( blocks ) + 2;
    P.add    = 0;
    static std::atomic< bool > opted_in[kMaxDevices];
    int                        rc;
    if ( ( rc = lateral_opt_in< OP, double >( opted_in, lateral_cg_kernel< OP > ) ) )
        return rc;
    constexpr size_t smem = sizeof( double ) * lateral_words< OP >();
    // r = b - A x, p = r
    P.src.p[0] = x, P.dst.p[0] = r;
    if ( ( rc = launch_lateral< OP >( m, P, 1, TN_APPLY_REPLACE, TN_COMM_ADDITIVE, st ) ) )
        return rc;
    double* const       rr[1] = { r };
    double*             pp[1] = { p[0] };
    const double* const bx[9] = { b, nullptr, nullptr, r };
    const double        c[3]  = { 1.0, -1.0, 0.0 };
    double* const       xx[1] = { x };
    const double* const aa[1] = { ap };
    const tn_mesh* const mm[1] = { m };
    TN_CUDA_TRY( cudaMemsetAsync( cg.counter, 0, sizeof( double ), st ) );
    if ( ( rc = tn_vec_lincomb_f64( m, 1, rr, 0.0, 2, c, bx, st ) ) ||
         ( rc = tn_pcg_begin_f64( 1, mm, rr, pp, cg.state, atol, st ) ) )
        return rc;
    // the stopping flag travels to a pinned slot before steps 2, 8, 16, ... and is looked at before the next of these (the
    // slot, like the partial sums of tn_pcg_*, is the mesh's: one reduction or solve on a mesh at a time)
    constexpr int kEvery = 8;
    cudaEvent_t   ev     = nullptr;
    TN_CUDA_TRY( cudaEventCreateWithFlags( &ev, cudaEventDisableTiming ) );
    double* const flag    = m->h_red_result + 15;
    bool          pending = false;
    int           it      = 0;
    for ( ; it < max_iterations && rc == TN_OK; ++it )
    {
        if ( it == 2 || ( it > 0 && it % kEvery == 0 ) )
        {
            if ( pending && cudaEventSynchronize( ev ) == cudaSuccess && *static_cast< volatile double* >( flag ) != 0.0 )
                break;
            pending = cudaMemcpyAsync( flag, cg.state + 4, sizeof( double ), cudaMemcpyDeviceToHost, st ) == cudaSuccess &&
                      cudaEventRecord( ev, st ) == cudaSuccess;
        }
        P.src.p[0] = cg.p_old = p[it & 1];
        P.dst.p[0] = ap, cg.p_new = pp[0] = p[( it & 1 ) ^ 1];
        lateral_cg_kernel< OP ><<< blocks, kLateralThreads, smem, st >>>( P, cg );
        if ( cudaGetLastError() != cudaSuccess )
        {
            set_error( "lateral_cg: launch failed" );
            rc = TN_ERR_CUDA;
            break;
        }
        rc = tn_pcg_update_f64( 1, mm, xx, rr, pp, aa, cg.state, it % kLateralHistory + 1, rtol, atol, st );
    }
    cudaEventDestroy( ev );
    if ( rc )
        return rc;
    double out[2];
    TN_CUDA_TRY( cudaMemcpyAsync( out, cg.state + 5, sizeof( out ), cudaMemcpyDeviceToHost, st ) );
    TN_CUDA_TRY( cudaStreamSynchronize( st ) );
    // out[0] counts modulo kLateralHistory, and at most 16 of the `it` steps issued come after the last one taken
    if ( iterations )
        *iterations = out[0] == 0.0 ? 0 : it - ( it - int( out[0] ) ) % kLateralHistory;
    if ( relres )
        *relres = out[1];
    return TN_OK;
}

}  // namespace tn
