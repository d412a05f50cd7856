// FP64 Newton closure of tiny systems (n = nS nT <= TINY_N duals, at most 64
// nodes), a warp per cell.
//
// A step of a small mesh lasts as long as its slowest cell's Newton, so what
// counts is the dependent chain of an iteration, not throughput. Lane k takes
// node k (and k + 32): nodal duals, U and DU with one exponential and one
// reciprocal. The sums over the nodes are not butterflies (27 values through
// five levels of shuffles, some 400 instructions) but columns: lane e owns one
// entry of the lower triangle of the Hessian or of the gradient and runs over
// the nodes with its column of a constant table, Q(k, e) = phi_ki phi_kj wt_k or
// phi_ki wt_k, in four partial sums; the 27 results go through shared memory to
// every lane, and every lane eliminates the system for itself (L D L^T, one
// reciprocal per pivot, the gradient as an extra row). Gradient and Hessian come
// from the same pass, so a trial that is accepted has its next direction's
// matrix at hand. The iteration, tests and line search are newton_cell's
// (closure.cpp:133-193).
//
// Bound by that chain (the cells of a step fill a fraction of the SMs' issue
// slots). Burgers, 5 duals, 20 nodes: closure phase of a step on 500 cells 35 ->
// 20 us (with its launches and events), on 20k cells 65 -> 31; the whole solve of
// 500 cells 42 -> 23 us a step. Two CTAs of four warps per SM: the system, its
// matrix and the duals stay in 240 registers (at 168 they spill).
#pragma once
#include "ipm_kernels.cuh"

namespace uqc {

constexpr int TINY_N = 6, TINY_H = TINY_N * ( TINY_N + 1 ) / 2, TINY_MAX_NODES = 64;

// Duals in basis-major order a = i nS + s, so that a level's duals are a prefix
// whatever its moment count. Table entry (k, e): e < TINY_H the pair a >= b with
// e = a (a + 1) / 2 + b, then the gradient rows; phi and wt as in KParams.
inline double tiny_entry( int nS, int nT, const double* phiRow, double wt, int e ) {
    if( e < TINY_H ) {
        int a = 0;
        while( ( a + 1 ) * ( a + 2 ) / 2 <= e ) ++a;
        const int i = a / nS, j = ( e - a * ( a + 1 ) / 2 ) / nS;
        return i < nT ? phiRow[i] * phiRow[j] * wt : 0.0;
    }
    const int i = ( e - TINY_H ) / nS;
    return e < TINY_H + TINY_N && i < nT ? phiRow[i] * wt : 0.0;
}

// doubles of a warp's shared memory: DU blocks and U at the nodes, the 32 sums,
// moments, moment sums, reduction scratch
__host__ __device__ inline int tiny_warp_doubles( int nS, int NP, int nQ ) { return ( NP + nS ) * nQ + 32 + 2 * 8 + 32; }

template <int CL> __global__ void __launch_bounds__( 128, 2 ) k_newton_tiny( KParams P, int mode ) {
    constexpr int NS = Closure<CL>::NS, NP = Closure<CL>::NP, TN = TINY_N, TT = ( TN + NS - 1 ) / NS;
    extern __shared__ __align__( 16 ) double smem[];
    if( mode == 1 && !P.ctl->active ) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nWarps = blockDim.x >> 5;
    for( int i = threadIdx.x; i < 32 * P.nQ; i += blockDim.x ) smem[i] = P.tinyTab[i];
    const double* Q = smem + lane;    // the lane's column, row stride 32
    double* nod     = smem + 32 * P.nQ + warp * tiny_warp_doubles( NS, NP, P.nQ );    // DU (b nQ + k), then U (s nQ + k)
    double* uk      = nod + NP * P.nQ;
    double* sums    = uk + NS * P.nQ;
    double *uhS = sums + 32, *msS = uhS + 8, *red = msS + 8;
    // the lane's nodes
    double ph[2][TT];
#pragma unroll
    for( int q = 0; q < 2; ++q )
#pragma unroll
        for( int i = 0; i < TT; ++i ) {
            const int k = lane + 32 * q;
            ph[q][i]    = k < P.nQ && i < P.nT ? P.phi[size_t( k ) * P.ld + i] : 0.0;
        }
    // the lane's sum: Hessian entry (a, b) of the blocks (s, t), or gradient row a
    const double* src = uk;
    int msAt          = -1;    // place of its moment sum in msS (state-major)
    {
        if( lane < TINY_H ) {
            int a = 0;
            while( ( a + 1 ) * ( a + 2 ) / 2 <= lane ) ++a;
            src = nod + pair_index<NS>( a % NS, ( lane - a * ( a + 1 ) / 2 ) % NS ) * P.nQ;
        }
        else if( lane < TINY_H + TN ) {
            const int a = lane - TINY_H;
            src         = uk + ( a % NS ) * P.nQ;
            if( a / NS < P.nT ) msAt = ( a % NS ) * P.nT + a / NS;
        }
    }
    __syncthreads();
    const Grp<32> grp{lane, 0};
    const int ldc    = NS * P.nT;
    const double eps = P.eps;
    const bool guard = P.newtonMode != 0;
    int* alist;
    unsigned* acount;
    step_list( P, 0, alist, acount );
    const int nWork = alist ? int( *acount ) : P.nWork;
    unsigned long long itSum = 0, lsSum = 0;
    int failSum = 0, activeSum = 0;
    double dtMin = 1e300;
    // the first cells go to the CTAs in turn, so that a short list spreads over the SMs
    for( int item = warp * int( gridDim.x ) + int( blockIdx.x ); item < nWork; ) {
        const int cell = alist ? alist[item] : item;
        const int lev = P.level ? int( P.level[cell] ) : P.nLevels - 1;
        const int nTj = P.nTotalCell ? int( P.nTotalCell[cell] ) : P.nTLevel[lev], n = NS * nTj;
        double lam[TN], lamN[TN], uh[TN], d[TN], h[TINY_H], g[TN];
        bool bad = false;
        if( lane < ldc ) {
            const double a = P.lam[size_t( cell ) * ldc + lane], b = P.u[size_t( cell ) * ldc + lane];
            uhS[lane]      = b;
            bad            = !isfinite( a ) || !isfinite( b );
        }
        bad = __any_sync( 0xffffffffu, bad );
#pragma unroll
        for( int a = 0; a < TN; ++a ) {
            const int s = a % NS, i = a / NS;
            lam[a] = a < n ? P.lam[size_t( cell ) * ldc + s * P.nT + i] : 0.0;
            uh[a]  = a < n ? P.u[size_t( cell ) * ldc + s * P.nT + i] : 0.0;
        }
        // U and DU at the duals x, Hessian h and gradient g there; ||g||
        auto evaluate = [&]( const double( &x )[TN] ) {
            __syncwarp();    // the previous sums are read
#pragma unroll
            for( int q = 0; q < 2; ++q ) {
                const int k = lane + 32 * q;
                if( 32 * q < P.nQ && k < P.nQ ) {
                    double L[NS], u[NS], y[NP];
#pragma unroll
                    for( int s = 0; s < NS; ++s ) L[s] = 0.0;
#pragma unroll
                    for( int a = 0; a < TN; ++a ) L[a % NS] = fma( x[a], ph[q][a / NS], L[a % NS] );
                    closure_udu<CL>( L, u, y, P.phys );
#pragma unroll
                    for( int b = 0; b < NP; ++b ) nod[b * P.nQ + k] = y[b];
#pragma unroll
                    for( int s = 0; s < NS; ++s ) uk[s * P.nQ + k] = u[s];
                }
            }
            __syncwarp();
            double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
            int k = 0;
            for( ; k + 3 < P.nQ; k += 4 ) {
                a0 = fma( src[k], Q[32 * k], a0 );
                a1 = fma( src[k + 1], Q[32 * k + 32], a1 );
                a2 = fma( src[k + 2], Q[32 * k + 64], a2 );
                a3 = fma( src[k + 3], Q[32 * k + 96], a3 );
            }
            for( ; k < P.nQ; ++k ) a0 = fma( src[k], Q[32 * k], a0 );
            const double sum = ( a0 + a1 ) + ( a2 + a3 );
            sums[lane]       = sum;
            if( msAt >= 0 ) msS[msAt] = sum;
            __syncwarp();
#pragma unroll
            for( int e = 0; e < TINY_H; ++e ) h[e] = sums[e];
            double s0 = 0.0, s1 = 0.0;
#pragma unroll
            for( int a = 0; a < TN; ++a ) {
                g[a] = a < n ? sums[TINY_H + a] - uh[a] : 0.0;
                ( a & 1 ? s1 : s0 ) = fma( g[a], g[a], a & 1 ? s1 : s0 );
            }
            return sqrt( s0 + s1 );
        };
        // d = H^-1 g by L D L^T; false: not positive definite
        auto direction = [&]() {
            bool pd = true;
            double r[TN];
#pragma unroll
            for( int j = 0; j < TN; ++j ) {
                if( j >= n ) break;
                const double dj = h[j * ( j + 1 ) / 2 + j];
                pd              = pd && dj > 0.0;
                r[j]            = reciprocal( dj );
#pragma unroll
                for( int i = j + 1; i < TN; ++i ) {
                    const double l = h[i * ( i + 1 ) / 2 + j] * r[j];
#pragma unroll
                    for( int c = j + 1; c <= i; ++c ) h[i * ( i + 1 ) / 2 + c] = fma( -l, h[c * ( c + 1 ) / 2 + j], h[i * ( i + 1 ) / 2 + c] );
                    g[i] = fma( -l, g[j], g[i] );
                }
            }
#pragma unroll
            for( int j = TN - 1; j >= 0; --j ) {
                d[j] = 0.0;
                if( j < n ) {
                    double v = g[j];
#pragma unroll
                    for( int i = j + 1; i < TN; ++i ) v = fma( -h[i * ( i + 1 ) / 2 + j], d[i], v );
                    d[j] = v * r[j];
                }
            }
            return pd;
        };
        auto trial = [&]( double step ) {
#pragma unroll
            for( int a = 0; a < TN; ++a ) lamN[a] = fma( -step, d[a], lam[a] );
            return evaluate( lamN );
        };
        int iters = 0, ls = 0, rc = -1;
        if( bad )
            rc = UQC_CELL_NONFINITE;
        else {
            double gn = evaluate( lam );
            if( gn < eps ) rc = UQC_CELL_CONVERGED;
            while( rc < 0 ) {
                if( iters >= P.maxIter ) {
                    rc = UQC_CELL_MAX_ITER;
                    break;
                }
                if( !direction() ) {
                    rc = UQC_CELL_NOT_PD;
                    break;
                }
                ++iters;
                double step = 1.0, gnN = trial( 1.0 );
                if( P.maxIter == 1 )
                    rc = UQC_CELL_CONVERGED;    // One-Shot IPM: lam -= H^-1 g, no line search (closure.cpp:151-154)
                else {
                    int refine = 0;
                    while( gn < gnN || ( guard && !isfinite( gnN ) ) ) {
                        step *= 0.5;
                        ++ls;
                        gnN = trial( step );
                        if( gnN < eps ) break;
                        if( ++refine > 1000 ) {
                            rc = UQC_CELL_LINE_SEARCH;
                            break;
                        }
                    }
                    if( rc == UQC_CELL_LINE_SEARCH ) break;
                    if( gnN < eps ) rc = UQC_CELL_CONVERGED;
                }
#pragma unroll
                for( int a = 0; a < TN; ++a ) lam[a] = lamN[a];
                gn = gnN;
            }
        }
#pragma unroll
        for( int a = 0; a < TN; ++a )
            if( lane == a && a < n && !bad ) P.lam[size_t( cell ) * ldc + ( a % NS ) * P.nT + a / NS] = lam[a];
        if( lane == 0 ) {
            P.status[cell] = rc;
            P.iters[cell]  = iters;
            itSum += iters;
            lsSum += ls;
            failSum += rc != 0;
            activeSum += iters > 0;
        }
        if( mode == 1 ) {
            if( rc != UQC_CELL_CONVERGED ) evaluate( lam );    // U at the duals it keeps
            __syncwarp();
            const double dloc = cell_epilogue<CL, 32>( grp, P, P.phiWf, uhS, uk, cell, lev, nTj, red, msS );
            dtMin             = dloc < dtMin ? dloc : dtMin;
        }
        __syncwarp();
        unsigned next = 0;
        if( lane == 0 ) next = atomicAdd( P.workCounter, 1u );
        item = nWarps * int( gridDim.x ) + int( __shfl_sync( 0xffffffffu, next, 0 ) );
    }
    if( lane == 0 ) {
        if( itSum ) atomicAdd( &P.ctl->newtonIters, itSum );
        if( lsSum ) atomicAdd( &P.ctl->lineSearchTrials, lsSum );
        if( failSum ) atomicAdd( &P.ctl->failedCells, failSum );
        if( activeSum ) atomicAdd( &P.ctl->activeCells, activeSum );
        if( mode == 1 && dtMin < 1e300 ) atomic_min_pos_double( &P.ctl->dtBits, dtMin );
    }
}

}    // namespace uqc
