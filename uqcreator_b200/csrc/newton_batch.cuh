// FP64 Newton closure (k_newton): several cells share a
// CTA and take their Newton iterations together.
//
// An iteration of Closure::SolveClosure (closure.cpp:133-193) on a cell of
// n = nS nT duals and nQ nodes needs the Hessian (pairs of basis functions x
// nodes x blocks, by far the most arithmetic), the solution of its system
// (little arithmetic, a long dependent chain) and a trial gradient. B cells per
// CTA ("slots", W / B warps each) iterate in step:
//
//   1. Hessian. Block (m, l) of a cell's Hessian is sum_k phi_ki phi_kj wt_k
//      DU_ml(Lambda_k) (closure.cpp:255-271), so the B cells' Hessians are one
//      product  [pairs x nodes] [nodes x (cell, block)]  of a constant matrix
//      with the cells' nodal DU. All warps of the CTA run it on the FP64 tensor
//      cores (mma.sync m8n8k4): a warp owns 8-pair row tiles over all columns,
//      forms its A values phi_ki phi_kj as it goes (one multiplication and two
//      loads per 8 x 4 fragment, used for every column tile) and keeps the
//      accumulators in registers over all nodes. The accumulators are then
//      scattered into the cells' packed triangles, which take the place of DU.
//   2. Block elimination by 8 x 8 tiles (eliminate_slot), a slot's warps
//      together, one barrier per tile column; back substitution by one warp.
//   3. The trial step, and the trial's nodal duals, U and DU in one pass (they
//      share the exponential, the logarithm and the division), gradient sums
//      split over (part, basis function) threads; DU goes where the Hessian was.
//      The line search and the tests are those of newton_cell (ipm_kernels.cuh).
//
// A slot that finishes takes the next cell from the work counter, so the CTA
// stays full until the list runs out.
//
// What bounds it: with 140 duals and 512 nodes the product (61 % of a cell's
// cycles, at 75 % of the FP64 rate); with 84 duals and 100 nodes the dependent
// chain of the elimination (40 %), which the other cells of the SM only partly
// cover (four cells fit: 41 KB each, 34 KB of it Hessian, and a 17 KB table per
// CTA); FP64 pipe 30-45 % busy. Cycles of one cell's iteration on an SM (its share
// of them): 43,000 in k_closure (four cells of two warps each) -> 21,000 with 84
// duals, 420,000 -> 140,000 with 140; 2-D Euler, 200k cells, closure phase of a step
// 10.2 -> 5.1 ms; 262k cells, three uncertainties, 88.5 -> 31 ms.
#pragma once
#include "chord.cuh"

namespace uqc {

// Shared memory of a slot (doubles): duals and moments at the finest stride nT
// (state-major), trial duals basis-major, moment sums of the last trial, the
// direction, nodal states node-major, reduction scratch; then one region that
// holds in turn DU (a column of duStride nodes per block) with the gradient's
// partial sums behind it, and the Hessian tiles with the right-hand side.
struct SlotLayout {
    int lam, lamI, uh, m, d, uk, red, hd, total;    // offsets in doubles
    int duStride;                                   // nodes per DU column: >= nQ, = 4 mod 8
};
__host__ __device__ inline SlotLayout slot_layout( int nS, int nT, int nQ, int NP, int threads ) {
    auto a4     = []( int x ) { return ( x + 3 ) & ~3; };
    const int n = nS * nT, parts = threads / nT > 0 ? threads / nT : 1;
    SlotLayout L;
    // DU columns of 4 mod 8 doubles: the eight columns of a B fragment start
    // in different bank groups
    L.duStride = ( ( nQ + 3 ) & ~3 ) | 4;
    int o = 0;
    L.lam  = o, o += a4( n );
    L.lamI = o, o += a4( n );
    L.uh   = o, o += a4( n );
    L.m    = o, o += a4( n );
    L.d    = o, o += a4( n );
    L.uk   = o, o += a4( nS * nQ );
    L.red  = o, o += 32;
    L.hd   = o;
    const int du = NP * L.duStride + parts * n, h = int( hess_doubles( n ) );
    o += a4( du > h ? du : h );
    L.total = o;
    return L;
}

// Tiles of k_newton: the block-packed upper triangle of linalg.cuh (htile, hrhs)
// with another order inside a tile, row-major with the 16-byte column pairs of
// a row permuted by the row: an mma accumulator (row, two columns) is one
// 16-byte access, and accumulators, operand fragments and whole rows read by
// consecutive lanes are all free of bank conflicts. (The column-major order of
// linalg.cuh costs two-way conflicts on each; the trailing update is bound by
// shared-memory cycles.)
__host__ __device__ __forceinline__ int rix( int r, int c ) { return ( r << 3 ) | ( ( ( ( c >> 1 ) ^ ( r >> 1 ) ) & 3 ) << 1 ) | ( c & 1 ); }
__host__ __device__ __forceinline__ int rblk( int r, int c ) { return htile( r >> 3, c >> 3 ) + rix( r & 7, c & 7 ); }

// Nodes per staged chunk of the basis table when it goes into the nodal states
// (nS nQ doubles a slot): the largest count of 4 mod 8 whose nT rows fit, 0 if none.
__host__ __device__ inline int newton_chunk( int nS, int nT, int nQ ) {
    const int fit = nS * nQ / nT;
    return fit < 4 ? 0 : fit - ( fit + 4 ) % 8;
}

// T <- -T^-1 for a symmetric positive definite 8 x 8 tile T held as an mma
// accumulator (lane 4 g + t: c0, c1 = row g, columns 2t and 2t + 1), by sweeps on
// the four 2 x 2 pivot blocks P (rows and columns p): A_pp -> -P^-1, A_rp -> A_rp
// P^-1, A_rc -> A_rc - A_rp P^-1 A_pc. With P^-1 = adj(P) / det(P) the products with
// the adjugate form beside the reciprocal, so a block costs the exchange by
// shuffles, the determinant, its reciprocal and one FMA of dependent latency:
// 820 cycles for the tile on an idle SM, against 1,020 for its element-wise
// Cholesky factor and triangular inverse in every lane's registers. This is the
// elimination's dependent chain. Returns false if a leading minor is not
// positive, or a block's determinant not within 2^+-1000.
__device__ __forceinline__ bool tile_sweep( double& c0, double& c1, int lane ) {
    const unsigned full = 0xffffffffu;
    const int g = lane >> 2, t = lane & 3;
    bool ok = true;
#pragma unroll
    for( int p = 0; p < 4; ++p ) {
        const double a = __shfl_sync( full, c0, 9 * p ), b = __shfl_sync( full, c1, 9 * p ), d = __shfl_sync( full, c1, 9 * p + 4 );
        const double u0 = __shfl_sync( full, c0, 4 * g + p ), u1 = __shfl_sync( full, c1, 4 * g + p );
        const double v00 = __shfl_sync( full, c0, 8 * p + t ), v01 = __shfl_sync( full, c1, 8 * p + t );
        const double v10 = __shfl_sync( full, c0, 8 * p + 4 + t ), v11 = __shfl_sync( full, c1, 8 * p + 4 + t );
        const double det = fma( a, d, -b * b );
        // a > 0 and 2^-1000 <= det < 2^1000 by the high words (beside the FP64 pipe; a NaN is
        // out of range)
        ok             = ok && __double2hiint( a ) > 0 && unsigned( __double2hiint( det ) - 0x01700000 ) < 0x7D000000u;
        const double r   = reciprocal( det );
        // A_rp adj(P); the pivot rows take -adj(P)
        const bool inRow = ( g >> 1 ) == p, inCol = t == p;
        const double q0  = inRow ? ( ( g & 1 ) ? b : -d ) : fma( u0, d, -u1 * b );
        const double q1  = inRow ? ( ( g & 1 ) ? -a : b ) : fma( u1, a, -u0 * b );
        const double s0  = inCol ? -q0 : fma( q0, v00, q1 * v10 );
        const double s1  = inCol ? -q1 : fma( q0, v01, q1 * v11 );
        c0               = fma( -s0, r, inRow || inCol ? 0.0 : c0 );
        c1               = fma( -s1, r, inRow || inCol ? 0.0 : c1 );
    }
    return ok;
}

// The sweep of S T S, S the powers of two that take T's diagonal entries to [1, 4):
// the determinants of entries beyond 2^+-500 leave the format's range (or the
// reciprocal's) although the entries do not. D <- -S (S T S)^-1 S. (A call that no usual
// state takes; its being there costs the others 0.5 %: closure phase of a warm step, 200k
// cells of 84 duals, 3.553 -> 3.570 ms; inlined 0.7 %, as a second round of a loop 3 %.)
static __device__ __noinline__ bool tile_sweep_scaled( double* D, double c0, double c1, int lane ) {
    const unsigned full = 0xffffffffu;
    const int g = lane >> 2, t = lane & 3;
    const double diag = ( g & 1 ) ? c1 : c0;    // of row g, in the lane that holds its column
    const double dg = __shfl_sync( full, diag, 4 * g + ( g >> 1 ) ), d0 = __shfl_sync( full, diag, 9 * t ), d1 = __shfl_sync( full, diag, 9 * t + 4 );
    if( __any_sync( full, !( dg > 0.0 ) || !isfinite( dg ) ) ) return false;
    const int e = -( ilogb( dg ) >> 1 ), e0 = e - ( ilogb( d0 ) >> 1 ), e1 = e - ( ilogb( d1 ) >> 1 );
    c0            = scalbn( c0, e0 );
    c1            = scalbn( c1, e1 );
    const bool ok = tile_sweep( c0, c1, lane );
    *reinterpret_cast<double2*>( D + rix( g, 2 * t ) ) = make_double2( scalbn( c0, e0 ), scalbn( c1, e1 ) );
    return ok;
}

// D <- -T^-1 (see tile_sweep); returns false if T is not positive definite.
__device__ __forceinline__ bool tile_sweep_inverse( double* D, double c0, double c1, int lane ) {
    double x0 = c0, x1 = c1;
    if( __builtin_expect( !tile_sweep( x0, x1, lane ), 0 ) ) return tile_sweep_scaled( D, c0, c1, lane );
    *reinterpret_cast<double2*>( D + rix( lane >> 2, 2 * ( lane & 3 ) ) ) = make_double2( x0, x1 );
    return true;
}

// B fragments (rows t and t + 4 of column g) of a tile held as an accumulator.
__device__ __forceinline__ void acc_to_b( double c0, double c1, int lane, double& b0, double& b1 ) {
    const unsigned full = 0xffffffffu;
    const int g = lane >> 2, t = lane & 3, src = 4 * t + ( g >> 1 );
    const double x0 = __shfl_sync( full, c0, src ), x1 = __shfl_sync( full, c1, src );
    const double z0 = __shfl_sync( full, c0, src + 16 ), z1 = __shfl_sync( full, c1, src + 16 );
    b0              = ( g & 1 ) ? x1 : x0;
    b1              = ( g & 1 ) ? z1 : z0;
}

// Block elimination H = L D L^T by 8 x 8 tiles, a slot's G warps together
// (block-packed tiles, right-hand side behind them; see linalg.cuh), one slot
// barrier per tile column. Step J, with N = -H_JJ^-1 in the diagonal tile's
// place: a warp takes whole tile columns C, forms W = N H_JC in registers and
// adds H_JR^T W to the column's tiles (R, C), J < R <= C; tile row J stays as it
// is (the back substitution reads it). Warp 0 takes the next diagonal tile
// alone, and its inverse, which is the dependent chain of the step; the last
// warp takes the right-hand side. Returns false if a pivot block is not
// positive definite (posv's info > 0). flag: two ints in shared memory, zero
// on entry, for the diagonal tiles of even and odd columns: step J's warps read
// tile J's after the step's barrier while warp 0 may already be writing tile
// J + 1's, and tile J + 2's is written only after the next barrier, which every
// reader of tile J's has reached. (With one flag for all, a warp that read it late
// could leave a step, and a barrier, before the others.) Warp 0 of every slot
// issues on the same scheduler (slots are a multiple of four warps apart), where
// its chain does not queue behind the other warps' products on the FP64 pipe.
template <int GROUP> __device__ bool eliminate_slot( const Grp<GROUP>& g, double* H, int nb, int* flag ) {
    constexpr int G = GROUP / 32;
    const int warp = g.r >> 5, lane = g.r & 31, gr = lane >> 2, t = lane & 3;
    const int o  = rix( gr, 2 * t );                         // accumulator place in a tile (16 bytes)
    const int f0 = rix( t, gr ), f1 = rix( t + 4, gr );      // fragment places
    double* rhs = H + hrhs( nb );
    auto invert = [&]( int J, double* D, double c0, double c1 ) {
        if( !tile_sweep_inverse( D, c0, c1, lane ) && lane == 0 ) flag[J & 1] = 1;
    };
    if( warp == 0 ) {
        // the first tile: only its upper half is filled
        const double c0 = H[gr <= 2 * t ? o : rix( 2 * t, gr )], c1 = H[gr <= 2 * t + 1 ? o + 1 : rix( 2 * t + 1, gr )];
        __syncwarp();
        invert( 0, H, c0, c1 );
    }
    for( int J = 0; J + 1 < nb; ++J ) {
        g.sync();    // the diagonal tile's inverse and all of row J's updates are in place
        if( flag[J & 1] ) return false;
        const int K     = J + 1;
        const double* N = H + htile( J, J );
        const double n0 = N[f0], n1 = N[f1];    // symmetric: also the A fragments
        // W = N H_JC as B fragments
        auto scaled = [&]( int C, double& b0, double& b1 ) {
            const double* A = H + htile( J, C );
            double w0 = 0.0, w1 = 0.0;
            dmma_8x8x4( w0, w1, n0, A[f0] );
            dmma_8x8x4( w0, w1, n1, A[f1] );
            acc_to_b( w0, w1, lane, b0, b1 );
        };
        if( warp == 0 ) {
            double b0, b1;
            scaled( K, b0, b1 );
            const double* A = H + htile( J, K );
            double* D       = H + htile( K, K );
            // the tile's lower half is not kept up: fill it by symmetry
            double c0 = D[gr <= 2 * t ? o : rix( 2 * t, gr )], c1 = D[gr <= 2 * t + 1 ? o + 1 : rix( 2 * t + 1, gr )];
            __syncwarp();
            dmma_8x8x4( c0, c1, A[f0], b0 );
            dmma_8x8x4( c0, c1, A[f1], b1 );
            invert( K, D, c0, c1 );
        }
        if( G == 1 || warp > 0 ) {
            const int worker = G == 1 ? 0 : warp - 1, workers = G == 1 ? 1 : G - 1;
            if( worker == workers - 1 ) {
                // b_R += H_JR^T (N b_J): lane c < 8 forms entry c of N b_J, then a lane per row
                double s0 = 0.0, s1 = 0.0;
                const int c = lane & 7;
#pragma unroll
                for( int k = 0; k < 8; k += 2 ) {
                    s0 = fma( N[rix( k, c )], rhs[J * 8 + k], s0 );
                    s1 = fma( N[rix( k + 1, c )], rhs[J * 8 + k + 1], s1 );
                }
                const double z = s0 + s1;
                double zk[8];
#pragma unroll
                for( int k = 0; k < 8; ++k ) zk[k] = __shfl_sync( 0xffffffffu, z, k );
                for( int r = K * 8 + lane; r < nb * 8; r += 32 ) {
                    const double* A = H + htile( J, r >> 3 );
                    s0 = rhs[r], s1 = 0.0;
#pragma unroll
                    for( int k = 0; k < 8; k += 2 ) {
                        s0 = fma( A[rix( k, r & 7 )], zk[k], s0 );
                        s1 = fma( A[rix( k + 1, r & 7 )], zk[k + 1], s1 );
                    }
                    rhs[r] = s0 + s1;
                }
            }
            for( int C = nb - 1 - worker; C > K; C -= workers ) {
                double b0, b1;
                scaled( C, b0, b1 );
                double* O = H + htile( K, C );
                // pairs of tiles, the next pair's operands loaded before this pair's results are stored
                int R = K;
                const double* A = H + htile( J, R );
                int step = ( R + 1 ) * 64;          // htile(J, R + 1) - htile(J, R)
                if( ( C - K ) % 2 == 0 ) {
                    double2 v = *reinterpret_cast<const double2*>( O + o );
                    dmma_8x8x4( v.x, v.y, A[f0], b0 );
                    dmma_8x8x4( v.x, v.y, A[f1], b1 );
                    *reinterpret_cast<double2*>( O + o ) = v;
                    ++R, O += 64, A += step, step += 64;
                }
                if( R < C ) {
                    double2 v0 = *reinterpret_cast<const double2*>( O + o ), v1 = *reinterpret_cast<const double2*>( O + 64 + o );
                    double x0 = A[f0], x1 = A[f1], y0 = A[step + f0], y1 = A[step + f1];
                    for( ;; ) {
                        dmma_8x8x4( v0.x, v0.y, x0, b0 );
                        dmma_8x8x4( v1.x, v1.y, y0, b0 );
                        dmma_8x8x4( v0.x, v0.y, x1, b1 );
                        dmma_8x8x4( v1.x, v1.y, y1, b1 );
                        R += 2;
                        if( R > C ) break;
                        A += 2 * step + 64, step += 128;
                        const double2 w0 = *reinterpret_cast<const double2*>( O + 128 + o ), w1 = *reinterpret_cast<const double2*>( O + 192 + o );
                        x0 = A[f0], x1 = A[f1], y0 = A[step + f0], y1 = A[step + f1];
                        *reinterpret_cast<double2*>( O + o )      = v0;
                        *reinterpret_cast<double2*>( O + 64 + o ) = v1;
                        v0 = w0, v1 = w1;
                        O += 128;
                    }
                    *reinterpret_cast<double2*>( O + o )      = v0;
                    *reinterpret_cast<double2*>( O + 64 + o ) = v1;
                }
            }
        }
    }
    g.sync();
    return !flag[( nb - 1 ) & 1];
}

// x = H^-1 b by one warp from eliminate_slot's tiles: x_J = -N_JJ b_J, then every
// row above takes its share H_RJ x_J (a lane per row, the next tile row first).
// The right-hand side is overwritten. (With the tile rows scaled beforehand,
// x_J = -N b_J + sum N H_JC x_C, the chain is 40 % shorter, but that pass over the
// tiles cost more than it gave.)
__device__ __forceinline__ void back_substitute( double* H, int nb, int n, double* x, int lane ) {
    double* y   = H + hrhs( nb );
    const int c = lane & 7;
    for( int J = nb - 1; J >= 0; --J ) {
        const double* N = H + htile( J, J );
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for( int k = 0; k < 8; k += 2 ) {
            const double2 v = *reinterpret_cast<const double2*>( y + J * 8 + k );
            s0              = fma( -N[rix( k, c )], v.x, s0 );
            s1              = fma( -N[rix( k + 1, c )], v.y, s1 );
        }
        const double xc = s0 + s1;
        if( lane < 8 && J * 8 + lane < n ) x[J * 8 + lane] = xc;
        double xv[8];
#pragma unroll
        for( int k = 0; k < 8; ++k ) xv[k] = __shfl_sync( 0xffffffffu, xc, k );
        for( int r = J * 8 - 1 - lane; r >= 0; r -= 32 ) {
            const double* A = H + htile( r >> 3, J );
            s0 = y[r], s1 = 0.0;
#pragma unroll
            for( int k = 0; k < 8; k += 2 ) {
                const double2 v = *reinterpret_cast<const double2*>( A + rix( r & 7, k ) );
                s0              = fma( -v.x, xv[k], s0 );
                s1              = fma( v.y, xv[k + 1], s1 );
            }
            y[r] = s0 - s1;
        }
        __syncwarp();
    }
}

// Where the value of pair p, block b (states m <= l) goes in the tiles of a
// level with T basis functions: (m T + j, l T + i) and, off the diagonal
// blocks, its mirror image (m T + i, l T + j).
__host__ __device__ inline void pair_places( int nS, int p, int b, int T, int* row, int* col ) {
    int i = 0, m = 0;
    while( ( i + 1 ) * ( i + 2 ) / 2 <= p ) ++i;
    const int j = p - i * ( i + 1 ) / 2;
    while( b >= nS - m ) {
        b -= nS - m;
        ++m;
    }
    const int l = m + b;
    row[0] = m * T + j, col[0] = l * T + i;
    row[1] = m < l ? m * T + i : row[0], col[1] = m < l ? l * T + j : col[0];
}
template <int NS> __device__ __noinline__ void scatter_value( double* H, int p, int b, int T, double v ) {
    if( p >= T * ( T + 1 ) / 2 ) return;    // a basis function beyond the level
    int row[2], col[2];
    pair_places( NS, p, b, T, row, col );
    H[rblk( row[0], col[0] )] = v;
    H[rblk( row[1], col[1] )] = v;
}

// B cells per CTA of W warps, MQ row tiles of 8 pairs per warp and pass.
template <int CL, int B, int W, int MQ, int CTAS>
__global__ void __launch_bounds__( 32 * W, CTAS ) k_newton( KParams P, int mode ) {
    constexpr int NS = Closure<CL>::NS, NP = Closure<CL>::NP, G = W / B, GROUP = 32 * G, NT = ( NP * B + 7 ) / 8;
    static_assert( B >= 2, "the table's chunks use two slots' nodal states" );
    extern __shared__ __align__( 16 ) double smem[];
    if( mode == 1 && !P.ctl->active ) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, slot = warp / G;
    Grp<GROUP> g{int( threadIdx.x ) - slot * GROUP, 1 + slot};
    const SlotLayout S = slot_layout( NS, P.nT, P.nQ, NP, GROUP );
    double* ws         = smem + size_t( slot ) * S.total;
    double *lam = ws + S.lam, *lamI = ws + S.lamI, *uh = ws + S.uh, *ms = ws + S.m, *dir = ws + S.d, *uk = ws + S.uk, *red = ws + S.red;
    double* H        = ws + S.hd;    // Hessian tiles; between iterations DU and the partial sums
    double* part     = H + NP * S.duStride;
    int* flag        = reinterpret_cast<int*>( red + 24 );    // two
    const size_t ldc = size_t( NS ) * P.nT;
    const int nQ4    = ( P.nQ + 3 ) & ~3;
    const double eps = P.eps;
    const bool guard = P.newtonMode != 0;
    const int pairs = P.nT * ( P.nT + 1 ) / 2, tiles = ( pairs + 7 ) / 8;
    // the node-contiguous basis table for the Hessian product, rows of 4 mod 8
    // doubles so that eight rows' fragments fall in different banks: whole when it
    // fits beside the slots, else chunks of nodes by turns in the first two
    // slots' nodal states, which nobody needs during the product
    double* tab         = smem + size_t( B ) * S.total + 4;
    const int chunk     = P.tabInSmem ? 0 : newton_chunk( NS, P.nT, P.nQ );
    const int tabStride = P.tabInSmem ? nQ4 | 4 : chunk;
    if( P.tabInSmem ) {
        for( int e = threadIdx.x; e < P.nT * nQ4; e += 32 * W ) {
            const int i = e / nQ4, k = e - i * nQ4;
            tab[i * tabStride + k] = P.phiT[size_t( i ) * P.ldT + k];
        }
        __syncthreads();
    }
    auto stage = [&]( int buf, int k0 ) {
        const int len = min( chunk, nQ4 - k0 ) / 2;    // 16-byte pieces of a row
        double* to    = smem + size_t( buf ) * S.total + S.uk;
        for( int e = threadIdx.x; e < P.nT * len; e += 32 * W ) {
            const int i = e / len, c = e - i * len;
            asm volatile( "cp.async.cg.shared.global [%0], [%1], 16;" ::"r"( smem_u32( to + i * chunk + 2 * c ) ),
                          "l"( P.phiT + size_t( i ) * P.ldT + k0 + 2 * c )
                          : "memory" );
        }
    };
    int* alist;
    unsigned* acount;
    step_list( P, 0, alist, acount );
    const int nWork = alist ? int( *acount ) : P.nWork;
    unsigned long long itSum = 0, lsSum = 0;
    int failSum = 0, activeSum = 0;
    double dtMin = 1e300;

    // the slot's cell
    int cell = -1, lev = 0, nTj = P.nT, iters = 0, ls = 0;
    double gn   = 0.0;
    bool first = true, active = false, more = true;

    // Lambda, U and wt DU at the trial duals lam + c d (lam itself for c = 0), the
    // moment sums m and the gradient norm (closure.cpp:205-213, 234-253)
    auto evaluate = [&]( double c ) {
        for( int idx = g.r; idx < NS * nTj; idx += GROUP ) {
            const int s = idx / nTj, i = idx - s * nTj;
            const double l0  = lam[s * P.nT + i];
            lamI[i * NS + s] = c == 0.0 ? l0 : fma( c, dir[idx], l0 );
        }
        g.sync();
        for( int k = g.r; k < nQ4; k += GROUP ) {
            if( k < P.nQ ) {
                double L[NS], u[NS], y[NP];
#pragma unroll
                for( int s = 0; s < NS; ++s ) L[s] = 0.0;
                const double* col = P.phiT + k;
                for( int i = 0; i < nTj; ++i, col += P.ldT ) {
                    const double r = __ldg( col );
                    double li[NS];
                    load_node<NS>( lamI, i, li );
#pragma unroll
                    for( int s = 0; s < NS; ++s ) L[s] = fma( li[s], r, L[s] );
                }
                closure_udu<CL>( L, u, y, P.phys );
                const double w = __ldg( P.wt + k );
#pragma unroll
                for( int s = 0; s < NS; ++s ) uk[k * NS + s] = u[s];
#pragma unroll
                for( int b = 0; b < NP; ++b ) H[b * S.duStride + k] = w * y[b];
            }
            else {
#pragma unroll
                for( int b = 0; b < NP; ++b ) H[b * S.duStride + k] = 0.0;
            }
        }
        g.sync();
        const int parts = GROUP / nTj > 0 ? min( GROUP / nTj, max( 1, GROUP / P.nT ) ) : 1;
        for( int e = g.r; e < parts * nTj; e += GROUP ) {
            const int p = e / nTj, i = e - p * nTj;
            double a[NS];
#pragma unroll
            for( int s = 0; s < NS; ++s ) a[s] = 0.0;
            const double* t = P.phiWf + size_t( p ) * P.ld + i;
#pragma unroll 2
            for( int k = p; k < P.nQ; k += parts, t += size_t( parts ) * P.ld ) {
                const double w = __ldg( t );
                double x[NS];
                load_node<NS>( uk, k, x );
#pragma unroll
                for( int s = 0; s < NS; ++s ) a[s] = fma( x[s], w, a[s] );
            }
#pragma unroll
            for( int s = 0; s < NS; ++s ) part[( p * NS + s ) * nTj + i] = a[s];
        }
        g.sync();
        double sq = 0.0;
        for( int idx = g.r; idx < NS * nTj; idx += GROUP ) {
            const int s = idx / nTj, i = idx - s * nTj;
            double m    = part[idx];
            for( int p = 1; p < parts; ++p ) m += part[p * NS * nTj + idx];
            ms[s * P.nT + i] = m;
            const double d   = m - uh[s * P.nT + i];
            sq               = fma( d, d, sq );
        }
        return sqrt( group_sum<GROUP>( g, sq, red ) );
    };
    // The cell is done: status, duals, and in step mode the epilogue [C]-[F]
    auto finish = [&]( int rc ) {
        if( g.r == 0 ) {
            P.status[cell] = rc;
            P.iters[cell]  = iters;
            itSum += iters;
            lsSum += ls;
            failSum += rc != 0;
            activeSum += iters > 0;
        }
        for( int idx = g.r; idx < int( ldc ); idx += GROUP ) P.lam[cell * ldc + idx] = lam[idx];
        if( mode == 1 ) {
            if( rc != UQC_CELL_CONVERGED ) evaluate( 0.0 );    // U at the duals it keeps
            g.sync();
            const double d = cell_epilogue<CL, GROUP, true>( g, P, P.phiWf, uh, uk, cell, lev, nTj, red, ms );
            dtMin          = d < dtMin ? d : dtMin;
        }
        g.sync();
        active = false;
    };

    for( ;; ) {
        // ---- a free slot takes cells until one needs an iteration
        while( !active && more ) {
            int item;
            if( first ) {
                // the first cells go to the CTAs in turn, so that a short list
                // spreads over the SMs
                item  = slot * int( gridDim.x ) + int( blockIdx.x );
                first = false;
            }
            else {
                if( g.r == 0 ) red[16] = double( atomicAdd( P.workCounter, 1u ) );
                g.sync();
                item = B * int( gridDim.x ) + int( red[16] );
                g.sync();
            }
            if( item >= nWork ) {
                more = false;
                break;
            }
            cell  = alist ? alist[item] : item;
            lev   = P.level ? int( P.level[cell] ) : P.nLevels - 1;
            nTj   = P.nTotalCell ? int( P.nTotalCell[cell] ) : P.nTLevel[lev];
            iters = ls = 0;
            bool bad   = false;
            for( int idx = g.r; idx < int( ldc ); idx += GROUP ) {
                const double a = P.lam[cell * ldc + idx], b = P.u[cell * ldc + idx];
                lam[idx]       = a;
                uh[idx]        = b;
                bad            = bad || !isfinite( a ) || !isfinite( b );
            }
            if( group_any<GROUP>( g, bad, red ) ) {
                g.sync();
                finish( UQC_CELL_NONFINITE );
                continue;
            }
            g.sync();
            gn = evaluate( 0.0 );
            if( gn < eps )
                finish( UQC_CELL_CONVERGED );
            else
                active = true;
        }
        if( !__syncthreads_or( active ) ) break;

        PT_BEGIN( tHess );
        // ---- Hessians of all slots: accumulators for MQ row tiles x NT column tiles
        const int gr = lane >> 2, t = lane & 3;
        int bOff[NT];
#pragma unroll
        for( int nt = 0; nt < NT; ++nt ) {
            // the last tile's padding columns repeat the last block
            const int col = min( 8 * nt + gr, NP * B - 1 ), sl = col / NP;
            bOff[nt] = sl * S.total + S.hd + ( col - sl * NP ) * S.duStride + t;
        }
        // (at most W MQ row tiles: the launch rule's condition)
        double acc[MQ][NT][2];
        int oi[MQ], oj[MQ];
#pragma unroll
        for( int q = 0; q < MQ; ++q ) {
            int j, i;
            unpack_pair( min( 8 * ( warp + W * q ) + gr, pairs - 1 ), j, i );
            oi[q] = i * tabStride + t;
            oj[q] = j * tabStride + t;
#pragma unroll
            for( int nt = 0; nt < NT; ++nt ) acc[q][nt][0] = acc[q][nt][1] = 0.0;
        }
        auto product = [&]( const double* tb, int kBeg, int kEnd ) {
#pragma unroll 2
            for( int k0 = kBeg; k0 < kEnd; k0 += 4 ) {
                double b[NT];
#pragma unroll
                for( int nt = 0; nt < NT; ++nt ) b[nt] = smem[bOff[nt] + k0];
                const double* tk = tb + ( k0 - kBeg );
#pragma unroll
                for( int q = 0; q < MQ; ++q ) {
                    if( warp + W * q < tiles ) {
                        const double a = tk[oi[q]] * tk[oj[q]];
#pragma unroll
                        for( int nt = 0; nt < NT; ++nt ) dmma_8x8x4( acc[q][nt][0], acc[q][nt][1], a, b[nt] );
                    }
                }
            }
        };
        if( P.tabInSmem )
            product( tab, 0, nQ4 );
        else {
            stage( 0, 0 );
            for( int c = 0, k0 = 0; k0 < nQ4; ++c, k0 += chunk ) {
                asm volatile( "cp.async.wait_all;" ::: "memory" );
                __syncthreads();    // this chunk is in place, the previous one is read
                if( k0 + chunk < nQ4 ) stage( ( c + 1 ) & 1, k0 + chunk );
                product( smem + size_t( c & 1 ) * S.total + S.uk, k0, min( k0 + chunk, nQ4 ) );
            }
        }
        __syncthreads();    // DU is read; the tiles take its place
        PT_END( tHess, 2 );
        PT_BEGIN( tScatter );
        // ---- scatter: value (pair (j, i), block (m, l)) of each slot
        const int n = NS * nTj, nb = hnb( n );
        {
            // with one moment count for all cells no slot needs another's (a free
            // slot's place takes what its columns held); else each slot's count is
            // published, zero for a free slot
            const bool uniform = P.nLevels == 1 && !P.nTotalCell;
            int* nTs           = reinterpret_cast<int*>( smem + size_t( B ) * S.total );
            if( !uniform ) {
                if( g.r == 0 ) nTs[slot] = active ? nTj : 0;
                __syncthreads();
            }
#pragma unroll
            for( int q = 0; q < MQ; ++q ) {
                const int p = 8 * ( warp + W * q ) + gr;
                if( p >= pairs ) continue;
#pragma unroll
                for( int nt = 0; nt < NT; ++nt ) {
                    // two adjacent columns: blocks of the same slot when NP is even
#pragma unroll
                    for( int h = 0; h < 2; ++h ) {
                        const int col = 8 * nt + 2 * t + h;
                        if( col >= NP * B ) continue;
                        const int sl = col / NP, b = col - sl * NP;
                        double* Hs   = smem + size_t( sl ) * S.total + S.hd;
                        if( uniform || nTs[sl] == P.nT ) {
                            // both places of the value from the table (the same one twice
                            // for a value that is not mirrored)
                            const unsigned o = __ldg( P.pairSlots + p * NP + b );
                            Hs[o & 0xFFFFu]  = acc[q][nt][h];
                            Hs[o >> 16]      = acc[q][nt][h];
                        }
                        else if( nTs[sl] > 0 )
                            scatter_value<NS>( Hs, p, b, nTs[sl], acc[q][nt][h] );
                    }
                }
            }
        }
        if( active ) {
            // identity padding of the last tile column, right-hand side g = m - u
            if( n & 7 ) {
                for( int e = g.r; e < nb * 64; e += GROUP ) {
                    const int R = e >> 6, col = ( nb - 1 ) * 8 + ( ( e >> 3 ) & 7 ), row = R * 8 + ( e & 7 );
                    if( col >= n && row <= col ) H[rblk( row, col )] = row == col ? 1.0 : 0.0;
                }
            }
            for( int idx = g.r; idx < nb * 8; idx += GROUP ) {
                const int s = idx / nTj, i = idx - s * nTj;
                H[hrhs( nb ) + idx] = idx < n ? ms[s * P.nT + i] - uh[s * P.nT + i] : 0.0;
            }
            if( g.r == 0 ) flag[0] = flag[1] = 0;
        }
        __syncthreads();
        PT_END( tScatter, 28 );
        PT_COUNT( 29 );
        if( !active ) continue;

        // ---- direction, line search, tests (newton_cell's iteration)
        PT_BEGIN( tChol );
        if( !eliminate_slot<GROUP>( g, H, nb, flag ) ) {
            g.sync();
            finish( UQC_CELL_NOT_PD );
            continue;
        }
        PT_END( tChol, 3 );
        PT_BEGIN( tBack );
        if( ( g.r >> 5 ) == 0 ) back_substitute( H, nb, n, dir, lane );
        g.sync();
        PT_END( tBack, 4 );
        ++iters;
        double step = 1.0;
        PT_BEGIN( tTrial );
        double gnN  = evaluate( -step );
        PT_END( tTrial, 5 );
        int refine = 0, rc = -1;
        while( gn < gnN || ( guard && !isfinite( gnN ) ) ) {
            step *= 0.5;
            ++ls;
            gnN = evaluate( -step );
            if( gnN < eps ) {
                rc = UQC_CELL_CONVERGED;
                break;
            }
            if( ++refine > 1000 ) {
                rc = UQC_CELL_LINE_SEARCH;
                break;
            }
        }
        if( rc != UQC_CELL_LINE_SEARCH ) {
            // accept the trial (its duals are in lamI)
            for( int idx = g.r; idx < n; idx += GROUP ) {
                const int s = idx / nTj, i = idx - s * nTj;
                lam[s * P.nT + i] = lamI[i * NS + s];
            }
            gn = gnN;
            if( gnN < eps )
                rc = UQC_CELL_CONVERGED;
            else if( iters >= P.maxIter )
                rc = UQC_CELL_MAX_ITER;
        }
        g.sync();
        if( rc >= 0 ) finish( rc );
    }
    if( g.r == 0 ) {
        if( itSum ) atomicAdd( &P.ctl->newtonIters, itSum );
        if( lsSum ) atomicAdd( &P.ctl->lineSearchTrials, lsSum );
        if( failSum ) atomicAdd( &P.ctl->failedCells, failSum );
        if( activeSum ) atomicAdd( &P.ctl->activeCells, activeSum );
        if( mode == 1 && dtMin < 1e300 ) atomic_min_pos_double( &P.ctl->dtBits, dtMin );
    }
}

}    // namespace uqc
