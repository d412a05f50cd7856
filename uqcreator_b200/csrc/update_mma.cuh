// Update of the 2-D Euler cells with the projection on the FP64 tensor cores
// (k_update_mma).
//
// k_update gives a warp one cell and projects its nodal flux sums with a lane
// per basis function: a table value and the node's four states from shared
// memory for every four FMAs, lanes beyond the basis functions idle, and with
// hundreds of nodes a table that is streamed from L2 for every cell (512 nodes, 35
// moments: 143 KB a cell) and flux buffers that fill shared memory. Here a warp
// takes two cells. Their four states are the eight rows of an mma (m8n8k4), the
// basis functions its columns: per four nodes one value a lane of the fluxes and
// one per eight functions of the table, for both cells. The fluxes are
// evaluated over (cell, node) slots, so that the lanes are full whatever the
// node count is modulo 32. Where the table does not stay in shared memory the
// CTA's warps go through the nodes together in chunks, the next chunk of the
// table arriving (cp.async) while they work.
//
// Bound by issue and latency of the fluxes (16 warps an SM, 128 registers). 200k
// cells, 21 moments, 100 nodes: 1150 -> 811 us; 262k cells, 35 moments, 512 nodes:
// 8.95 -> 5.02 ms.
#pragma once
#include "ipm_kernels.cuh"

namespace uqc {

// Column tiles of the instances (8 basis functions each), and a padded table row.
constexpr int UPD_TILES[3] = {3, 5, 8};
__host__ __device__ constexpr int upd_ld( int tiles ) { return 8 * tiles + 4; }    // 4 mod 8: fragments free of bank conflicts
constexpr int UPD_FACE = 16;    // doubles of a cell's face data

__host__ __device__ inline size_t update_mma_doubles( int nS, int nQ, int chunk, int tiles, int warps ) {
    const int rows = chunk >= nQ ? chunk : 2 * chunk;
    return size_t( rows ) * upd_ld( tiles ) + size_t( warps ) * 2 * ( size_t( chunk ) * nS + UPD_FACE );
}

template <int CL, bool FIN, int NT> __global__ void __launch_bounds__( 256, 2 ) k_update_mma( KParams P ) {
    constexpr int NS = Closure<CL>::NS, NF = 3, LD = upd_ld( NT );
    static_assert( NS == 4, "two cells' states are the eight rows of an mma" );
    const bool finish = FIN && P.finishInUpdate;
    extern __shared__ __align__( 16 ) double smem[];
    if( !P.ctl->active ) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
    const int gr = lane >> 2, t = lane & 3;    // accumulator row (cell gr / 4, state gr mod 4), column pair
    const int chunk  = P.updNodes;
    const bool whole = chunk >= P.nQ;
    double* tab = smem;    // the whole table, or two chunks of its rows
    double* Gs  = smem + size_t( whole ? chunk : 2 * chunk ) * LD + size_t( warp ) * 2 * ( chunk * NS + UPD_FACE );    // [cell][node][state]
    double* fd  = Gs + 2 * chunk * NS;    // per cell: unit normal, scaled normal, length of each face
    const int nQ4 = ( P.nQ + 3 ) & ~3;
    auto stage    = [&]( int buf, int k0 ) {
        const int len      = min( chunk, nQ4 - k0 ) * LD;    // rows are padded with zeros up to nQ4; even
        const double* from = P.phiWfP + size_t( k0 ) * LD;
        double* to         = tab + size_t( buf ) * chunk * LD;
        for( int e = 2 * threadIdx.x; e < len; e += 2 * blockDim.x )
            asm volatile( "cp.async.cg.shared.global [%0], [%1], 16;" ::"r"( unsigned( __cvta_generic_to_shared( to + e ) ) ), "l"( from + e )
                          : "memory" );
    };
    if( whole ) {
        stage( 0, 0 );
        asm volatile( "cp.async.wait_all;" ::: "memory" );
        __syncthreads();
    }
    const double dt  = __longlong_as_double( (long long)P.ctl->dtBits );
    const size_t ldc = size_t( NS ) * P.nT;
    double res = 0.0, dtNext = 1e300;
    NextLists N;
    if( finish ) N.open( P );
    const int end = P.cellBase + P.nWork;
    for( int first = P.cellBase + 2 * blockIdx.x * nWarps; first < end; first += 2 * gridDim.x * nWarps ) {
        const int c0 = first + 2 * warp;
        bool live[2];
#pragma unroll
        for( int c = 0; c < 2; ++c ) {
            const int cell  = c0 + c;
            const bool have = cell < end;
            live[c]         = have && P.boundary[cell] != 1;
            if( have && finish && lane == 0 && P.finFlag[cell] ) {
                // finished by the previous update: this step's closure status
                P.status[cell]  = UQC_CELL_CONVERGED;
                P.iters[cell]   = 0;
                P.finFlag[cell] = 0;
            }
            if( have && !live[c] ) {
                // Dirichlet cell: uNew = u (expliciteuler.cpp:21-23)
                for( int idx = lane; idx < int( ldc ); idx += 32 ) P.u[cell * ldc + idx] = P.uRe[cell * ldc + idx];
                if( lane == 0 ) {
                    const double u0 = P.uRe[cell * ldc];
                    res += fabs( u0 - P.uOld0[cell] ) * P.area[cell];
                    if( finish && P.nLevels == 1 ) finish_cell( P, cell, u0, dtNext );
                }
                if( finish && P.nLevels > 1 ) N.cbuf.push( lane, cell, N.clist, N.ccount );
            }
        }
        __syncwarp();    // the previous cells' face data is read
        if( lane < 2 * NF ) {
            const int c = lane / NF, f = lane - c * NF;
            if( live[c] ) {
                const size_t at = size_t( c0 + c ) * NF + f;
                const double a = P.scaledN[2 * at], b = P.scaledN[2 * at + 1];
                double* w      = fd + c * UPD_FACE + 5 * f;
                w[0]           = P.unitN[2 * at];
                w[1]           = P.unitN[2 * at + 1];
                w[2]           = a;
                w[3]           = b;
                w[4]           = sqrt( a * a + b * b );    // |n| of euler2d.cpp:84, once per face
            }
        }
        int nb[2][NF];
#pragma unroll
        for( int c = 0; c < 2; ++c )
#pragma unroll
            for( int f = 0; f < NF; ++f ) nb[c][f] = live[c] ? P.nbr[size_t( c0 + c ) * NF + f] : 0;
        double acc[NT][2];
#pragma unroll
        for( int n = 0; n < NT; ++n ) acc[n][0] = acc[n][1] = 0.0;
        __syncwarp();
        if( !whole ) stage( 0, 0 );
        for( int ch = 0, k0 = 0; k0 < P.nQ; ++ch, k0 += chunk ) {
            const int nn = min( chunk, P.nQ - k0 ), nn4 = ( nn + 3 ) & ~3;
            // fluxes over (cell, node) slots; the rows up to a multiple of four nodes are zero
            for( int j = lane; j < 2 * nn4; j += 32 ) {
                const int c = j >= nn4, k = j - ( c ? nn4 : 0 );
                double gs[NS];
#pragma unroll
                for( int s = 0; s < NS; ++s ) gs[s] = 0.0;
                if( ( c ? live[1] : live[0] ) && k < nn ) {
                    const double* q = P.uQ + k0 + k;
                    const double* f5 = fd + c * UPD_FACE;
                    double a[NS], b[NF][NS];
#pragma unroll
                    for( int s = 0; s < NS; ++s ) a[s] = q[( size_t( c0 + c ) * NS + s ) * P.nQ];
#pragma unroll
                    for( int f = 0; f < NF; ++f )
#pragma unroll
                        for( int s = 0; s < NS; ++s ) b[f][s] = q[( size_t( c ? nb[1][f] : nb[0][f] ) * NS + s ) * P.nQ];
                    const typename Problem<CL>::Side sa = Problem<CL>::side( a, P.phys.gamma );
#pragma unroll
                    for( int f = 0; f < NF; ++f ) {
                        double y[NS];
                        Problem<CL>::flux( a, sa, b[f], f5 + 5 * f, f5 + 5 * f + 2, f5[5 * f + 4], y, P.phys );
#pragma unroll
                        for( int s = 0; s < NS; ++s ) gs[s] += y[s];
                    }
                }
                double2* out = reinterpret_cast<double2*>( Gs + ( c * chunk + k ) * NS );
                out[0]       = make_double2( gs[0], gs[1] );
                out[1]       = make_double2( gs[2], gs[3] );
            }
            if( whole )
                __syncwarp();
            else {
                asm volatile( "cp.async.wait_all;" ::: "memory" );
                __syncthreads();    // the chunk has arrived; every warp is past the other buffer
                if( k0 + chunk < P.nQ ) stage( ( ch + 1 ) & 1, k0 + chunk );
            }
            // rhs(row, i) += sum_k G(row, k) phiWf(k, i)
            const double* A  = Gs + ( gr >> 2 ) * chunk * NS + t * NS + ( gr & 3 );
            const double* Bt = tab + size_t( whole ? 0 : ( ch & 1 ) ) * chunk * LD + t * LD + gr;
#pragma unroll 2
            for( int k = 0; k < nn4; k += 4 ) {
                const double a = A[k * NS];
#pragma unroll
                for( int n = 0; n < NT; ++n ) dmma_8x8x4( acc[n][0], acc[n][1], a, Bt[k * LD + 8 * n] );
            }
            __syncwarp();    // Gs is read
        }
        if( !whole ) __syncthreads();    // the last chunk is read before the next cells' first arrives
        // update: the lane's cell and state, moments 8 n + 2 t and the next
        const int mine  = gr >> 2, cell = c0 + mine, s = gr & 3;
        const bool on   = mine ? live[1] : live[0];
        const int nTj   = on ? P.nTLevel[P.level[cell]] : 0;
        double sq = 0.0, u00 = 0.0;
        if( on ) {
            const double area = P.area[cell], cf = dt / area;
            const size_t row  = cell * ldc + s * P.nT;
#pragma unroll
            for( int n = 0; n < NT; ++n )
#pragma unroll
                for( int h = 0; h < 2; ++h ) {
                    const int i = 8 * n + 2 * t + h;
                    if( i < nTj ) {
                        const double old = P.uRe[row + i], v = old - acc[n][h] * cf, gi = old - v;
                        P.u[row + i]     = v;
                        sq               = fma( gi, gi, sq );
                        if( s == 0 && i == 0 ) {
                            u00 = v;
                            res += fabs( v - P.uOld0[cell] ) * area;
                        }
                    }
                }
        }
        if( finish ) {
            for( int o = 8; o > 0; o >>= 1 ) sq += __shfl_xor_sync( 0xffffffffu, sq, o );    // over the cell's 16 lanes
#pragma unroll
            for( int c = 0; c < 2; ++c ) {
                const double sc = __shfl_sync( 0xffffffffu, sq, 16 * c ), uc = __shfl_sync( 0xffffffffu, u00, 16 * c );
                const int nc    = __shfl_sync( 0xffffffffu, nTj, 16 * c );
                if( live[c] ) test_next_step<NS>( P, lane, c0 + c, nc, sc, uc, N, dtNext );
            }
        }
        __syncwarp();
    }
    if( finish ) N.flush( lane );
    if( lane == 0 && dtNext < 1e300 ) atomic_min_pos_double( &P.ctl->dtBitsNext, dtNext );
    // every lane may hold a residual term: update_epilogue adds them per warp
    update_epilogue( P, res, dt, finish );
}

}    // namespace uqc
