// FP64 Newton closure of tiny systems (n = nS nT <= 6 or 10 duals, at most 64
// nodes), a warp per cell.
//
// A step of a small mesh lasts as long as its slowest cell's Newton, so what
// counts is the dependent chain of an iteration, not throughput. Lane k takes
// node k (and k + 32): nodal duals, U and DU with one exponential and one
// reciprocal. The sums over the nodes are not butterflies (27 values through
// five levels of shuffles, some 400 instructions) but columns: lane e owns one
// entry of the lower triangle of the Hessian or of the gradient (two with ten
// duals) and runs over the nodes with its column of a constant table, Q(k, e) =
// phi_ki phi_kj wt_k or phi_ki wt_k, in four partial sums; the results go through
// shared memory to every lane, and every lane eliminates the system for itself (L D L^T, one
// reciprocal per pivot, the gradient as an extra row). Gradient and Hessian come
// from the same pass, so a trial that is accepted has its next direction's
// matrix at hand. The iteration, tests and line search are newton_cell's
// (closure.cpp:133-193).
//
// Bound by that chain (the cells of a step fill a fraction of the SMs' issue
// slots). Burgers, 5 duals, 20 nodes: closure phase of a step on 500 cells 35 ->
// 20 us (with its launches and events), on 20k cells 65 -> 31; the whole solve of
// 500 cells 42 -> 23 us a step. Two CTAs of four warps per SM: the system, its
// matrix and the duals of 6 stay in 240 registers (at 168 they spill); the instance
// of 10 spills 276 B, mostly the basis values of the lane's nodes, and still shortens
// the chain: Burgers, 10 duals, 40 nodes, a step on 500 cells 46 -> 33, on 20k 63 -> 56.
#pragma once
#include "ipm_kernels.cuh"

namespace uqc {

// Instances: systems of up to TINY_N or SMALL_N duals.
constexpr int TINY_N = 6, SMALL_N = 10, TINY_MAX_NODES = 64, SMALL_CELLS = 32768;
__host__ __device__ constexpr int tiny_h( int TN ) { return TN * ( TN + 1 ) / 2; }           // Hessian entries
__host__ __device__ constexpr int tiny_sums( int TN ) { return tiny_h( TN ) + TN; }
__host__ __device__ constexpr int tiny_cols( int TN ) { return ( tiny_sums( TN ) + 31 ) & ~31; }    // table columns

// Duals in basis-major order a = i nS + s, so that a level's duals are a prefix
// whatever its moment count. Table entry (k, e): e < tiny_h the pair a >= b with
// e = a (a + 1) / 2 + b, then the gradient rows; phi and wt as in KParams.
inline double tiny_entry( int TN, int nS, int nT, const double* phiRow, double wt, int e ) {
    if( e < tiny_h( TN ) ) {
        int a = 0;
        while( ( a + 1 ) * ( a + 2 ) / 2 <= e ) ++a;
        const int i = a / nS, j = ( e - a * ( a + 1 ) / 2 ) / nS;
        return i < nT ? phiRow[i] * phiRow[j] * wt : 0.0;
    }
    const int i = ( e - tiny_h( TN ) ) / nS;
    return e < tiny_sums( TN ) && i < nT ? phiRow[i] * wt : 0.0;
}

// doubles of a warp's shared memory: DU blocks and U at the nodes, the sums,
// moments, moment sums, reduction scratch
__host__ __device__ inline int tiny_warp_doubles( int TN, int nS, int NP, int nQ ) { return ( ( NP + nS ) * nQ + tiny_cols( TN ) + 2 * 12 + 32 + 1 ) & ~1; }

template <int CL, int TN> __global__ void __launch_bounds__( 128, 2 ) k_newton_tiny( KParams P, int mode ) {
    constexpr int NS = Closure<CL>::NS, NP = Closure<CL>::NP, TT = ( TN + NS - 1 ) / NS;
    constexpr int TH = tiny_h( TN ), SUMS = tiny_sums( TN ), COLS = tiny_cols( TN );
    // whole rounds of 32 sums, a lane each; up to two left over are spread over the lanes
    constexpr int REST = SUMS % 32 <= 2 ? SUMS % 32 : 0, ROUNDS = ( SUMS - REST + 31 ) / 32;
    extern __shared__ __align__( 16 ) double smem[];
    if( mode == 1 && !P.ctl->active ) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nWarps = blockDim.x >> 5;
    for( int i = threadIdx.x; i < COLS * P.nQ; i += blockDim.x ) smem[i] = P.tinyTab[i];
    const double* Q = smem + lane;    // the lane's columns, row stride COLS
    double* nod     = smem + COLS * P.nQ + warp * tiny_warp_doubles( TN, NS, NP, P.nQ );    // DU (b nQ + k), then U (s nQ + k)
    double* uk      = nod + NP * P.nQ;
    double* sums    = uk + NS * P.nQ;
    double *uhS = sums + COLS, *msS = uhS + 12, *red = msS + 12;
    // the lane's nodes
    double ph[2][TT];
#pragma unroll
    for( int q = 0; q < 2; ++q )
#pragma unroll
        for( int i = 0; i < TT; ++i ) {
            const int k = lane + 32 * q;
            ph[q][i]    = k < P.nQ && i < P.nT ? P.phi[size_t( k ) * P.ld + i] : 0.0;
        }
    // a sum's source: Hessian entry (a, b) of the blocks (s, t), or gradient row a;
    // and the place of a gradient row's moment sum in msS (state-major)
    auto source = [&]( int e, int& msAt ) {
        msAt = -1;
        if( e < TH ) {
            int a = 0;
            while( ( a + 1 ) * ( a + 2 ) / 2 <= e ) ++a;
            return (const double*)( nod + pair_index<NS>( a % NS, ( e - a * ( a + 1 ) / 2 ) % NS ) * P.nQ );
        }
        const int a = min( e - TH, TN - 1 );
        if( e < SUMS && a / NS < P.nT ) msAt = ( a % NS ) * P.nT + a / NS;
        return (const double*)( uk + ( a % NS ) * P.nQ );
    };
    const double* src[ROUNDS];
    int msAt[ROUNDS];
#pragma unroll
    for( int q = 0; q < ROUNDS; ++q ) src[q] = source( lane + 32 * q, msAt[q] );
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
        double lam[TN], lamN[TN], d[TN], h[TH], g[TN];
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
#pragma unroll
            for( int q = 0; q < ROUNDS; ++q ) {
                double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
                const double *x = src[q], *w = Q + 32 * q;
                int k = 0;
                for( ; k + 3 < P.nQ; k += 4, x += 4, w += 4 * COLS ) {
                    a0 = fma( x[0], w[0], a0 );
                    a1 = fma( x[1], w[COLS], a1 );
                    a2 = fma( x[2], w[2 * COLS], a2 );
                    a3 = fma( x[3], w[3 * COLS], a3 );
                }
                for( ; k < P.nQ; ++k, ++x, w += COLS ) a0 = fma( x[0], w[0], a0 );
                const double sum    = ( a0 + a1 ) + ( a2 + a3 );
                sums[lane + 32 * q] = sum;
                if( msAt[q] >= 0 ) msS[msAt[q]] = sum;
            }
#pragma unroll
            for( int e = SUMS - REST; e < SUMS; ++e ) {
                int at;
                const double* x = source( e, at );
                double v        = 0.0;
                for( int k = lane; k < P.nQ; k += 32 ) v = fma( x[k], smem[k * COLS + e], v );
                for( int o = 16; o > 0; o >>= 1 ) v += __shfl_xor_sync( 0xffffffffu, v, o );
                if( lane == 0 ) {
                    sums[e] = v;
                    if( at >= 0 ) msS[at] = v;
                }
            }
            __syncwarp();
#pragma unroll
            for( int e = 0; e < TH; ++e ) h[e] = sums[e];
            double s0 = 0.0, s1 = 0.0;
#pragma unroll
            for( int a = 0; a < TN; ++a ) {
                g[a] = a < n ? sums[TH + a] - uhS[( a % NS ) * P.nT + a / NS] : 0.0;
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
                    // (L D L^T x = b after the forward pass: x_j = y_j / D_j - sum_i l_ij x_i,
                    // with h holding l_ij D_j)
                    double v = g[j], z = 0.0;
#pragma unroll
                    for( int i = j + 1; i < TN; ++i ) ( i & 1 ? z : v ) = fma( -h[i * ( i + 1 ) / 2 + j], d[i], i & 1 ? z : v );
                    d[j] = ( v + z ) * r[j];
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
