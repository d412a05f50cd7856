// Check and update kernels for cells of few moments (at most NTM of them):
// LPC lanes per cell, several cells per warp.
//
// A warp per cell (k_check, k_update) spends most of its instructions on what a
// small cell does not have: one lane per basis function in the projections,
// lists and tests on one lane, idle lanes beyond the nodes. Here lane `sub` of
// a cell's takes the nodes k = sub (mod LPC) for everything, the nodal duals,
// the ansatz or the fluxes, and its share of every moment's sum in registers;
// the sums are then exchanged so that lane `sub` keeps the moments i = sub (mod
// LPC) (LPC - 1 exchanges per LPC moments, a fixed order).
//
// Bound by the latency of a cell's loads and then by issue (0.39 instructions per
// cycle and scheduler at 16 warps an SM, registers for the sums allow no more; 44 %
// of the stalls on global loads, FP64 pipe 20-30 %, DRAM 2.2 TB/s): so two nodes at a
// time, and on large meshes the next cell's state on its way. Four lanes per cell: two
// made the large meshes another 5-15 % faster and the small ones slower, eight the
// other way round. Adaptive shallow water, 1M cells: check 1240 us with a warp per
// cell, 472 with four lanes, 431 with nodes in pairs, 388 with the prefetch; update
// 1390, 410, 351, 308.
#pragma once
#include "ipm_kernels.cuh"

namespace uqc {

constexpr int LPC = 4;    // lanes per cell

// Moments a kernel instance holds in registers; the launcher takes the
// smallest that fits.
constexpr int SMALL_NT[3] = {6, 10, 16};

// x[0..LPC-1] of each of the cell's lanes -> the sum over the lanes of x[sub] in lane sub.
__device__ __forceinline__ double exchange_sum( double ( &x )[LPC], int sub ) {
#pragma unroll
    for( int h = LPC / 2; h > 0; h >>= 1 ) {
        const bool upper = sub & h;
#pragma unroll
        for( int j = 0; j < h; ++j ) {
            const double keep = upper ? x[j + h] : x[j], send = upper ? x[j] : x[j + h];
            x[j]              = keep + __shfl_xor_sync( 0xffffffffu, send, h );
        }
    }
    return x[0];
}

// Moment sums of all states: out[s][b] = the sum of acc[s][LPC b + sub] over the
// cell's lanes; blocks beyond nMax (warp-uniform) are left zero.
template <int NS, int NTM>
__device__ __forceinline__ void exchange_moments( const double ( &acc )[NS][NTM], int nMax, int sub, double ( &out )[NS][( NTM + LPC - 1 ) / LPC] ) {
#pragma unroll
    for( int b = 0; b < ( NTM + LPC - 1 ) / LPC; ++b )
#pragma unroll
        for( int s = 0; s < NS; ++s ) {
            out[s][b] = 0.0;
            if( LPC * b < nMax ) {
                double x[LPC];
#pragma unroll
                for( int j = 0; j < LPC; ++j ) x[j] = LPC * b + j < NTM ? acc[s][LPC * b + j < NTM ? LPC * b + j : 0] : 0.0;
                out[s][b] = exchange_sum( x, sub );
            }
        }
}

// Sum over the cell's lanes, in every one of them.
__device__ __forceinline__ double cell_sum( double v ) {
    for( int o = LPC / 2; o > 0; o >>= 1 ) v += __shfl_xor_sync( 0xffffffffu, v, o );
    return v;
}
__device__ __forceinline__ double cell_min( double v ) {
    for( int o = LPC / 2; o > 0; o >>= 1 ) v = fmin( v, __shfl_xor_sync( 0xffffffffu, v, o ) );
    return v;
}

// The next cell's state on its way into L2 while this one's is worked on: a line, or
// the n doubles at x by the cell's lanes in turn. On meshes of FAR rounds or more, whose
// state does not stay in L2 (adaptive shallow water, check / update us: 1M cells 431 / 351
// -> 388 / 308, 200k cells 199 / 120 -> 182 / 108; 50k cells 57 / 27 and without the rule 57 / 29).
constexpr int FAR = 8;
__device__ __forceinline__ void prefetch_line( const void* x ) { asm volatile( "prefetch.global.L2 [%0];" ::"l"( x ) ); }
__device__ __forceinline__ void prefetch_cell( const double* x, int n, int sub ) {
    for( int i = 16 * sub; i < n; i += 16 * LPC ) prefetch_line( x + i );
}

// Appends `cell` of the lanes where `on` holds to a device list: one atomic per warp.
__device__ __forceinline__ void warp_append( bool on, int cell, int* list, unsigned* count, int lane ) {
    const unsigned m = __ballot_sync( 0xffffffffu, on );
    if( m == 0 ) return;
    unsigned base    = 0;
    const int leader = __ffs( m ) - 1;
    if( lane == leader ) base = atomicAdd( count, unsigned( __popc( m ) ) );
    base = __shfl_sync( 0xffffffffu, base, leader );
    if( on ) list[base + __popc( m & ( ( 1u << lane ) - 1u ) )] = cell;
}

// The tables in shared memory: phi (or null), then phiWf.
__device__ __forceinline__ void stage_tables( const KParams& P, bool both, double* smem, const double*& phi, const double*& phiWf ) {
    const int tn = P.nQ * P.ld;
    for( int i = threadIdx.x; i < tn; i += blockDim.x ) {
        smem[i] = P.phiWf[i];
        if( both ) smem[tn + i] = P.phi[i];
    }
    phiWf = smem;
    phi   = both ? smem + tn : nullptr;
    __syncthreads();
}

// k_check for few moments: the same test, epilogue and lists.
template <int CL, int NTM> __global__ void __launch_bounds__( 256, 2 ) k_check_small( KParams P ) {
    constexpr int NS = Closure<CL>::NS, NB = ( NTM + LPC - 1 ) / LPC;
    extern __shared__ __align__( 16 ) double smem[];
    if( !P.ctl->active ) return;
    const bool listMode = P.ctl->listReady != 0;
    const int par       = P.ctl->steps & 1;
    const int nItems    = listMode ? int( P.checkCount[par] ) : P.nWork;
    if( nItems == 0 ) return;
    int* alist;
    unsigned* acount;
    step_list( P, 0, alist, acount );
    const double *phi, *phiWf;
    stage_tables( P, true, smem, phi, phiWf );
    const int lane = threadIdx.x & 31, sub = lane & ( LPC - 1 );
    const unsigned own = ( ( 1u << LPC ) - 1u ) << ( lane & ~( LPC - 1 ) );    // the cell's lanes
    const int ldc      = NS * P.nT;
    double dtMin       = 1e300;
    const int stride   = gridDim.x * ( blockDim.x / LPC );
    const bool far     = !listMode && nItems > FAR * stride;
    // whole warps go round together (the exchanges are warp-wide)
    for( int item0 = ( blockIdx.x * blockDim.x + ( threadIdx.x & ~31 ) ) / LPC; item0 < nItems; item0 += stride ) {
        const int item   = item0 + lane / LPC;
        const bool valid = item < nItems;
        const int cell   = listMode ? P.checkList[size_t( par ) * P.nCells + ( valid ? item : item0 )] : P.cellBase + ( valid ? item : item0 );
        const double* lam = P.lam + size_t( cell ) * ldc;
        const double* uh  = P.u + size_t( cell ) * ldc;
        if( !listMode && P.finFlag && valid && sub == 0 ) P.finFlag[cell] = 0;
        if( far && item + stride < nItems ) {
            const size_t next = size_t( cell ) + stride;
            prefetch_cell( P.lam + next * ldc, ldc, sub );
            prefetch_cell( P.u + next * ldc, ldc, sub );
            prefetch_line( sub & 1 ? (const void*)( P.level + next ) : P.dx + next );
        }
        const int lev = int( P.level[cell] ), nTj = P.nTLevel[lev];
        bool bad = false;
        for( int idx = sub; idx < ldc; idx += LPC ) bad = bad || !isfinite( lam[idx] ) || !isfinite( uh[idx] );
        bad = ( __ballot_sync( 0xffffffffu, bad ) & own ) != 0;
        int newLev = lev;
        if( P.nLevels > 1 ) newLev = level_rule( P, level_indicator( P, [&]( int i ) { return uh[i]; }, lev, nTj ), lev );
        const int nTn = P.nTLevel[newLev];
        // loop bound of the warp's cells
        const int nMax = __reduce_max_sync( 0xffffffffu, max( nTj, nTn ) );
        double l[NS][NTM], acc[NS][NTM];
#pragma unroll
        for( int i = 0; i < NTM; ++i )
#pragma unroll
            for( int s = 0; s < NS; ++s ) {
                acc[s][i] = 0.0;
                l[s][i]   = i < nTj ? lam[s * P.nT + i] : 0.0;
            }
        double* uq  = P.uQ + size_t( cell ) * NS * P.nQ;
        double dloc = 1e300;
        const double dx = P.dx[cell];
        // two nodes at a time: the chains of U and dt overlap, the loops' bounds are tested once for both
        for( int k = sub; k < P.nQ; k += 2 * LPC ) {
            const bool two = k + LPC < P.nQ;
            const int k1   = two ? k + LPC : k;    // no second node: the first again, left out of the sums
            double L[2][NS], y[2][NS];
#pragma unroll
            for( int s = 0; s < NS; ++s ) L[0][s] = L[1][s] = 0.0;
            const double *row0 = phi + k * P.ld, *row1 = phi + k1 * P.ld;
#pragma unroll
            for( int i = 0; i < NTM; ++i ) {
                if( i >= nMax ) break;
                const double r0 = row0[i], r1 = row1[i];
#pragma unroll
                for( int s = 0; s < NS; ++s ) {
                    L[0][s] = fma( l[s][i], r0, L[0][s] );
                    L[1][s] = fma( l[s][i], r1, L[1][s] );
                }
            }
            Closure<CL>::U( L[0], y[0], true, P.phys );
            Closure<CL>::U( L[1], y[1], true, P.phys );
            if( valid && !bad ) {
                // a cell that fails the test gets its nodal states from its Newton
#pragma unroll
                for( int s = 0; s < NS; ++s ) {
                    uq[s * P.nQ + k]  = y[0][s];
                    uq[s * P.nQ + k1] = y[1][s];
                }
            }
            const double d0 = Problem<CL>::dt( y[0], dx, P.phys ), d1 = Problem<CL>::dt( y[1], dx, P.phys );
            dloc             = d0 < dloc ? d0 : dloc;
            dloc             = d1 < dloc ? d1 : dloc;
            if( !two ) {
#pragma unroll
                for( int s = 0; s < NS; ++s ) y[1][s] = 0.0;
            }
            const double *w0 = phiWf + k * P.ld, *w1 = phiWf + k1 * P.ld;
#pragma unroll
            for( int i = 0; i < NTM; ++i ) {
                if( i >= nMax ) break;
                const double x0 = w0[i], x1 = w1[i];
#pragma unroll
                for( int s = 0; s < NS; ++s ) acc[s][i] = fma( y[1][s], x1, fma( y[0][s], x0, acc[s][i] ) );
            }
        }
        double m[NS][NB];
        exchange_moments<NS, NTM>( acc, nMax, sub, m );
        double sq = 0.0;
#pragma unroll
        for( int b = 0; b < NB; ++b ) {
            const int i = LPC * b + sub;
            if( i < nTj ) {
#pragma unroll
                for( int s = 0; s < NS; ++s ) {
                    const double d = m[s][b] - uh[s * P.nT + i];
                    sq             = fma( d, d, sq );
                }
            }
        }
        sq                   = cell_sum( sq );
        dloc                 = cell_min( dloc );
        const bool converged = valid && !bad && sqrt( sq ) < P.eps;
        const double u00     = uh[0];
        __syncwarp();    // uh is read: uRe may be u itself
        if( converged ) {
#pragma unroll
            for( int b = 0; b < NB; ++b ) {
                const int i = LPC * b + sub;
                if( i < P.nT ) {
#pragma unroll
                    for( int s = 0; s < NS; ++s ) {
                        const size_t at = size_t( cell ) * ldc + s * P.nT + i;
                        P.uRe[at]       = i < nTn ? m[s][b] : 0.0;
                        if( i >= nTn ) P.u[at] = 0.0;    // the update writes u below the level only
                    }
                }
            }
            if( sub == 0 ) {
                P.status[cell] = UQC_CELL_CONVERGED;
                P.iters[cell]  = 0;
                P.uOld0[cell]  = u00;
                P.level[cell]  = unsigned( newLev );
                if( P.cellDt ) P.cellDt[cell] = dloc;
                dtMin = dloc < dtMin ? dloc : dtMin;
            }
        }
        warp_append( valid && !converged && sub == 0, cell, alist, acount, lane );
    }
    for( int o = 16; o > 0; o >>= 1 ) dtMin = fmin( dtMin, __shfl_xor_sync( 0xffffffffu, dtMin, o ) );
    if( lane == 0 && dtMin < 1e300 ) atomic_min_pos_double( &P.ctl->dtBits, dtMin );
}

// k_update for few moments (no wall cells): the same fluxes, update, next-step
// test and lists.
template <int CL, bool FIN, int NTM> __global__ void __launch_bounds__( 256, Closure<CL>::NS == 4 ? 1 : 2 ) k_update_small( KParams P ) {
    constexpr int NS = Closure<CL>::NS, NB = ( NTM + LPC - 1 ) / LPC, NF = NS == 4 ? 3 : 2;
    // nodes at a time, as in the check: two for the cheap fluxes; with three and four
    // states the registers are short (1-D Euler, 100k cells: 51 us with one, 55 with two)
    constexpr int KN = NS <= 2 ? 2 : 1;
    const bool finish = FIN && P.finishInUpdate;
    extern __shared__ __align__( 16 ) double smem[];
    if( !P.ctl->active ) return;
    const double *phi, *phiWf;
    stage_tables( P, false, smem, phi, phiWf );
    const int lane = threadIdx.x & 31, sub = lane & ( LPC - 1 );
    const int ldc   = NS * P.nT;
    const double dt = __longlong_as_double( (long long)P.ctl->dtBits );
    double res = 0.0, dtNext = 1e300;
    int *nlist = nullptr, *clist = nullptr;
    unsigned *ncount = nullptr, *ccount = nullptr;
    if( finish ) {
        step_list( P, 1, nlist, ncount );
        clist  = P.checkList + size_t( ( P.ctl->steps + 1 ) & 1 ) * P.nCells;
        ccount = P.checkCount + ( ( P.ctl->steps + 1 ) & 1 );
    }
    const int stride = gridDim.x * ( blockDim.x / LPC );
    const bool far   = P.nWork > FAR * stride;
    for( int item0 = ( blockIdx.x * blockDim.x + ( threadIdx.x & ~31 ) ) / LPC; item0 < P.nWork; item0 += stride ) {
        const int item   = item0 + lane / LPC;
        const bool valid = item < P.nWork;
        const int cell   = P.cellBase + ( valid ? item : item0 );
        const bool fixed = P.boundary[cell] == 1;    // Dirichlet cell: uNew = u (expliciteuler.cpp:21-23)
        const bool live  = valid && !fixed;
        if( finish && valid && sub == 0 && P.finFlag[cell] ) {
            // finished by the previous update: this step's closure status
            P.status[cell]  = UQC_CELL_CONVERGED;
            P.iters[cell]   = 0;
            P.finFlag[cell] = 0;
        }
        if( far && item + stride < P.nWork ) {
            const size_t next = size_t( cell ) + stride;
            prefetch_cell( P.uQ + next * NS * P.nQ, NS * P.nQ, sub );
            prefetch_cell( P.uRe + next * ldc, ldc, sub );
            prefetch_line( sub == 0   ? (const void*)( P.nbr + next * NF )
                           : sub == 1 ? P.unitN + 2 * next * NF
                           : sub == 2 ? (const void*)( P.scaledN + 2 * next * NF )
                                      : P.level + next );
            prefetch_line( sub & 1 ? (const void*)( P.boundary + next ) : P.area + next );
        }
        const int nTj  = P.nTLevel[P.level[cell]];
        const int nMax = __reduce_max_sync( 0xffffffffu, nTj );
        double acc[NS][NTM];
#pragma unroll
        for( int i = 0; i < NTM; ++i )
#pragma unroll
            for( int s = 0; s < NS; ++s ) acc[s][i] = 0.0;
        const double* ua = P.uQ + size_t( cell ) * NS * P.nQ;
        if( live ) {
            const double* ub[NF];
            double nu[NF][2], sn[NF][2], len[NF];
#pragma unroll
            for( int f = 0; f < NF; ++f ) {
                const size_t at = size_t( cell ) * NF + f;
                ub[f]           = P.uQ + size_t( P.nbr[at] ) * NS * P.nQ;
                nu[f][0]        = P.unitN[2 * at];
                nu[f][1]        = P.unitN[2 * at + 1];
                sn[f][0]        = P.scaledN[2 * at];
                sn[f][1]        = P.scaledN[2 * at + 1];
                len[f]          = sqrt( sn[f][0] * sn[f][0] + sn[f][1] * sn[f][1] );
            }
            for( int k = sub; k < P.nQ; k += KN * LPC ) {
                const bool two = KN == 2 && k + LPC < P.nQ;
                const int kk[2] = {k, two ? k + LPC : k};
                double gs[KN][NS];
#pragma unroll
                for( int j = 0; j < KN; ++j ) {
                    double a[NS];
#pragma unroll
                    for( int s = 0; s < NS; ++s ) {
                        a[s]     = ua[s * P.nQ + kk[j]];
                        gs[j][s] = 0.0;
                    }
                    const typename Problem<CL>::Side sa = Problem<CL>::side( a, P.phys.gamma );
#pragma unroll
                    for( int f = 0; f < NF; ++f ) {
                        double b[NS], y[NS];
#pragma unroll
                        for( int s = 0; s < NS; ++s ) b[s] = ub[f][s * P.nQ + kk[j]];
                        Problem<CL>::flux( a, sa, b, nu[f], sn[f], len[f], y, P.phys );
#pragma unroll
                        for( int s = 0; s < NS; ++s ) gs[j][s] += y[s];
                    }
                }
                if( !two ) {
#pragma unroll
                    for( int s = 0; s < NS && KN == 2; ++s ) gs[KN - 1][s] = 0.0;
                }
                const double *w0 = phiWf + kk[0] * P.ld, *w1 = phiWf + kk[1] * P.ld;
#pragma unroll
                for( int i = 0; i < NTM; ++i ) {
                    if( i >= nMax ) break;
                    const double x0 = w0[i], x1 = KN == 2 ? w1[i] : 0.0;
#pragma unroll
                    for( int s = 0; s < NS; ++s ) {
                        acc[s][i] = fma( gs[0][s], x0, acc[s][i] );
                        if( KN == 2 ) acc[s][i] = fma( gs[KN - 1][s], x1, acc[s][i] );
                    }
                }
            }
        }
        __syncwarp();
        double r[NS][NB];
        exchange_moments<NS, NTM>( acc, nMax, sub, r );
        const double area = P.area[cell], c = dt / area;
        double sq = 0.0, u0 = 0.0;
#pragma unroll
        for( int b = 0; b < NB; ++b ) {
            const int i = LPC * b + sub;
            // a live cell's moments of its level (beyond it u stays zero); a fixed cell's all
            if( valid && i < ( fixed ? P.nT : nTj ) ) {
#pragma unroll
                for( int s = 0; s < NS; ++s ) {
                    const size_t at  = size_t( cell ) * ldc + s * P.nT + i;
                    const double old = P.uRe[at], v = fixed ? old : old - r[s][b] * c, d = old - v;
                    P.u[at]          = v;
                    sq               = fma( d, d, sq );
                    if( s == 0 && i == 0 ) {
                        u0 = v;
                        res += fabs( v - P.uOld0[cell] ) * area;
                    }
                }
            }
        }
        if( finish ) {
            // the next step's closure test (see k_update); a fixed cell passes
            sq              = cell_sum( sq );
            const bool pass = valid && ( fixed || sqrt( sq ) < P.eps );
            bool fin        = pass;
            if( P.nLevels > 1 ) {
                __syncwarp();    // the cell's new moments are written
                const int lev   = int( P.level[cell] );
                const double* u = P.u + size_t( cell ) * ldc;
                fin = pass && !fixed && level_rule( P, level_indicator( P, [&]( int i ) { return u[i]; }, lev, nTj ), lev ) == lev;
            }
            if( fin && sub == 0 ) finish_cell( P, cell, u0, dtNext );
            if constexpr( NS == 4 ) {
                // the gradient the mixed form's rounds start from (see test_next_step),
                // from the lane's own moments
                if( P.gStore && valid && !pass ) {
                    double* gs = P.gStore + size_t( cell ) * P.gStride;
                    for( int i = sub; i < nTj; i += LPC )
#pragma unroll
                        for( int s = 0; s < NS; ++s ) {
                            const size_t at  = size_t( cell ) * ldc + s * P.nT + i;
                            gs[s * nTj + i]  = P.uRe[at] - P.u[at];
                        }
                    if( sub == 0 ) gs[ldc] = sqrt( sq );
                }
            }
            warp_append( pass && !fin && sub == 0, cell, clist, ccount, lane );
            warp_append( valid && !pass && sub == 0, cell, nlist, ncount, lane );
        }
    }
    for( int o = 16; o > 0; o >>= 1 ) dtNext = fmin( dtNext, __shfl_xor_sync( 0xffffffffu, dtNext, o ) );
    if( lane == 0 && dtNext < 1e300 ) atomic_min_pos_double( &P.ctl->dtBitsNext, dtNext );
    update_epilogue( P, res, dt, finish );
}

}    // namespace uqc
