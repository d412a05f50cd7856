// Instantiation of every kernel of one closure kind (included once per kind
// by kernels_<kind>.cu) and the table of their addresses.
#pragma once
#include "chord.cuh"
#include "ipm_kernels.cuh"
#include "kernels.h"
#include "newton_batch.cuh"
#include "newton_tiny.cuh"
#include "small_cells.cuh"
#include "update_mma.cuh"

namespace uqc {

// The instances for few moments: NTM = 6, 10 or 16, as far as a lane's registers
// hold a cell's sums.
template <int CL, int NTM> void* small_kernel_of( int which ) {
    if constexpr( Closure<CL>::NS * NTM <= ( Closure<CL>::NS == 4 ? 24 : 32 ) ) {
        if constexpr( !Closure<CL>::LINEAR && Closure<CL>::NS < 4 )
            if( which == KERNEL_CHECK_SMALL ) return (void*)&k_check_small<CL, NTM>;
        if( which == KERNEL_UPDATE_SMALL ) return (void*)&k_update_small<CL, true, NTM>;
        if( which == KERNEL_UPDATE_SMALL_PLAIN ) return (void*)&k_update_small<CL, false, NTM>;
    }
    return nullptr;
}

template <int CL> void* kernel_of( int group, int which ) {
    if constexpr( Closure<CL>::LINEAR ) {
        // linear closures: no Newton, so no mixed, register-Newton or rounds kernels
        if( which == KERNEL_CLOSURE_MIXED || which == KERNEL_CLOSURE_TINY || which == KERNEL_CHORD || which == KERNEL_HESS_TC ||
            which == KERNEL_INVERT_RAW || which == KERNEL_INVERT || which == KERNEL_INVERT_SWEEP )
            return nullptr;
    }
    switch( which ) {
        case KERNEL_CLOSURE:
            if( group == 32 ) return (void*)&k_closure<CL, 32, double>;
            if( group == 64 ) return (void*)&k_closure<CL, 64, double>;
            if( group == 256 ) return (void*)&k_closure<CL, 256, double>;
            return nullptr;
        case KERNEL_CLOSURE_TINY:
            if constexpr( !Closure<CL>::LINEAR ) return group == SMALL_N ? (void*)&k_newton_tiny<CL, SMALL_N> : (void*)&k_newton_tiny<CL, TINY_N>;
            return nullptr;
        case KERNEL_CLOSURE_MIXED:
            if constexpr( !Closure<CL>::LINEAR ) {
                if( group == 32 ) return (void*)&k_closure<CL, 32, float>;
                if( group == 64 ) return (void*)&k_closure<CL, 64, float>;
            }
            return nullptr;
        case KERNEL_UPDATE: return (void*)&k_update<CL, true, false, false>;
        case KERNEL_UPDATE_PLAIN: return (void*)&k_update<CL, false, false, false>;
        case KERNEL_UPDATE_SPLIT: return (void*)&k_update<CL, true, false, true>;
        case KERNEL_UPDATE_PLAIN_SPLIT: return (void*)&k_update<CL, false, false, true>;
        case KERNEL_UPDATE_WALL:
            if constexpr( Closure<CL>::NS == 4 ) return (void*)&k_update<CL, true, true, false>;
            return nullptr;
        case KERNEL_UPDATE_PLAIN_WALL:
            if constexpr( Closure<CL>::NS == 4 ) return (void*)&k_update<CL, false, true, false>;
            return nullptr;
        case KERNEL_UPDATE_MMA:
        case KERNEL_UPDATE_MMA_PLAIN:
            if constexpr( CL == 1 ) {
                const bool fin = which == KERNEL_UPDATE_MMA;
                if( group == UPD_TILES[0] ) return fin ? (void*)&k_update_mma<CL, true, UPD_TILES[0]> : (void*)&k_update_mma<CL, false, UPD_TILES[0]>;
                if( group == UPD_TILES[1] ) return fin ? (void*)&k_update_mma<CL, true, UPD_TILES[1]> : (void*)&k_update_mma<CL, false, UPD_TILES[1]>;
                if( group == UPD_TILES[2] ) return fin ? (void*)&k_update_mma<CL, true, UPD_TILES[2]> : (void*)&k_update_mma<CL, false, UPD_TILES[2]>;
            }
            return nullptr;
        case KERNEL_INIT:
            if( group == 32 ) return (void*)&k_init<CL, 32>;
            if( group == 256 ) return (void*)&k_init<CL, 256>;
            return nullptr;
        case KERNEL_MEANVAR:
            if( group == 32 ) return (void*)&k_meanvar<CL, 32>;
            if( group == 256 ) return (void*)&k_meanvar<CL, 256>;
            return nullptr;
        case KERNEL_CHECK: return (void*)&k_check<CL>;
        case KERNEL_CHECK_SMALL:
        case KERNEL_UPDATE_SMALL:
        case KERNEL_UPDATE_SMALL_PLAIN:
            if( group == SMALL_NT[0] ) return small_kernel_of<CL, SMALL_NT[0]>( which );
            if( group == SMALL_NT[1] ) return small_kernel_of<CL, SMALL_NT[1]>( which );
            if( group == SMALL_NT[2] ) return small_kernel_of<CL, SMALL_NT[2]>( which );
            return nullptr;
        case KERNEL_PHASE_COUNTERS: {
#ifdef UQC_PHASE_TIMERS
            void* p = nullptr;
            return cudaGetSymbolAddress( &p, g_phaseCycles ) == cudaSuccess ? p : nullptr;
#else
            return nullptr;
#endif
        }
        case KERNEL_NEWTON_S4:
        case KERNEL_NEWTON_S2:
        case KERNEL_NEWTON_M2:
        case KERNEL_NEWTON_L2:
            if constexpr( CL == 1 ) {
                if( which == KERNEL_NEWTON_S4 ) return (void*)&k_newton<CL, 4, 4, 2, 4>;
                if( which == KERNEL_NEWTON_S2 ) return (void*)&k_newton<CL, 2, 4, 4, 4>;
                if( which == KERNEL_NEWTON_M2 ) return (void*)&k_newton<CL, 2, 8, 4, 2>;
                return (void*)&k_newton<CL, 2, 16, 5, 1>;
            }
            else if constexpr( !Closure<CL>::LINEAR ) {
                if( which == KERNEL_NEWTON_S4 ) return (void*)&k_newton<CL, 4, 4, 2, 4>;
                if( which == KERNEL_NEWTON_S2 ) return (void*)&k_newton<CL, 2, 4, 4, 4>;
            }
            return nullptr;
        case KERNEL_CHORD:
        case KERNEL_HESS_TC:
        case KERNEL_INVERT_RAW:
        case KERNEL_INVERT:
        case KERNEL_INVERT_SWEEP:
            if constexpr( CL == 1 ) {    // the mixed form in rounds serves the 2-D Euler closure
                if( which == KERNEL_CHORD ) return (void*)&k_chord<CL>;
                if( which == KERNEL_INVERT_SWEEP ) return (void*)&k_invert_sweep<CL>;
                if( which == KERNEL_HESS_TC ) return (void*)&k_hess_tc<CL>;
                if( which == KERNEL_INVERT_RAW ) return (void*)&k_invert<CL, true>;
                return (void*)&k_invert<CL, false>;
            }
            return nullptr;
        default: return nullptr;
    }
}

}    // namespace uqc
