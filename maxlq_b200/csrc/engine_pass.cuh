// engine_pass.cuh -- the pass launchers of Engine<T> specialised for one grid
// size, as explicit instantiations: engine_pass.cu defines those of one
// (T, N) per object file, so that the sizes compile in parallel, and the
// engine's own translation units declare them all extern.
#pragma once
#include "engine_impl.cuh"

// every functor an x stage runs, as X(prefix, T, N, functor)
#define MLQ_XFWD_FUNCTORS(X, P, T, N)                                                                             \
    X(P, T, N, FCopy) X(P, T, N, FMul) X(P, T, N, FSq3) X(P, T, N, FGSq) X(P, T, N, FGPow) X(P, T, N, FRProd)     \
    X(P, T, N, FRProdE) X(P, T, N, FRE) X(P, T, N, FUGradU) X(P, T, N, FDot3) X(P, T, N, FEDot)                   \
    X(P, T, N, FRTrial<false>) X(P, T, N, FRTrial<true>) X(P, T, N, FRTrialE) X(P, T, N, FG1) X(P, T, N, FG2) X(P, T, N, FG2E) X(P, T, N, FG2T)    \
    X(P, T, N, FG3<false>) X(P, T, N, FG3<true>) X(P, T, N, FC3) X(P, T, N, FLSS) X(P, T, N, FLSS12)              \
    X(P, T, N, FLSW<0>) X(P, T, N, FLSW<1>) X(P, T, N, FLSQG) X(P, T, N, FLSA) X(P, T, N, FAPow)           \
    X(P, T, N, FLSE) X(P, T, N, FLSTrial<false>) X(P, T, N, FLSTrial<true>)                               \
    X(P, T, N, FLSTrialE) X(P, T, N, FLSC2) X(P, T, N, FLSPC6) X(P, T, N, FLSPC8A) X(P, T, N, FLSPC8B)            \
    X(P, T, N, FLSUV) X(P, T, N, FLSS32)
#define MLQ_PASS_X(P, T, N, F) P template void Engine<T>::xfwd_c<N, F>(XFwdArgs<T>&, const F&);

// P: `extern` (declaration) or nothing (definition)
#define MLQ_PASS_UNIT(P, T, N)                                          \
    P template void Engine<T>::xinv_c<N>(XInvArgs<T>&, int);            \
    P template void Engine<T>::y_c<N>(YArgs<T>&, int, int);             \
    P template void Engine<T>::zfwd_c<N>(ZFwdArgs<T>&, int);            \
    P template void Engine<T>::zinv_c<N>(ZInvArgs<T>&, int);            \
    P template void Engine<T>::zinv_multi_c<N>(ZInvMultiArgs<T>&, int); \
    MLQ_XFWD_FUNCTORS(MLQ_PASS_X, P, T, N)

// the sizes of dispatch_n
#define MLQ_PASS_EXTERN(T)                                                                                     \
    MLQ_PASS_UNIT(extern, T, 16)                                                                               \
    MLQ_PASS_UNIT(extern, T, 32)                                                                               \
    MLQ_PASS_UNIT(extern, T, 48)                                                                               \
    MLQ_PASS_UNIT(extern, T, 64)                                                                               \
    MLQ_PASS_UNIT(extern, T, 96)                                                                               \
    MLQ_PASS_UNIT(extern, T, 128)                                                                              \
    MLQ_PASS_UNIT(extern, T, 192)                                                                              \
    MLQ_PASS_UNIT(extern, T, 256)                                                                              \
    MLQ_PASS_UNIT(extern, T, 384)                                                                              \
    MLQ_PASS_UNIT(extern, T, 512)                                                                              \
    MLQ_PASS_UNIT(extern, T, 768)                                                                              \
    MLQ_PASS_UNIT(extern, T, 1024)
