// uw_state.cuh -- the thread-private state of one column in the FP64 column code at the implicit-CIN
// branch of iteration 2, as lists, and its copy to and from a hand-off buffer.
//
// The worklist pass runs in two launches: UW_MODE_LIST1 computes iteration 1 of the implicit-CIN
// loop and iteration 2 up to the CIN decision; a column taking the implicit branch restores its
// iteration-1 state there (uwshcu.F90:1759-1889), stores it here, and UW_MODE_RESUME continues it in
// warps sorted by updraft depth.  Stored is what the rest of iteration 2 reads and cannot rebuild:
//   - the profiles of UW_ST_FULL: the Exner functions, the wet-bulb humidity and the virtual potential
//     temperatures at the layer edges (pow, findsp and conden results); UW_MODE_RESUME rebuilds the
//     other environment profiles from the inputs with the set-up's operations, and every other
//     profile is written by the sections after this point before they read it;
//   - the source air (tracers included), the cloud base and the closure's inputs;
//   - the scalars that a section may read without having set them (the updraft's when no level is left
//     for it, and the roots, which keep their last values where a quadratic has none).
// So the second launch computes exactly what a single launch would.  (With the 14 further profiles, the
// k = 0 elements and the 60 scalars that nothing reads, a slot took 6 kB at 30 levels and 5 tracers
// instead of 1.6 kB.)
//
// Buffer layout: word w of slot s at state[w * cap + s] (consecutive slots of a warp are
// consecutive doubles).  Integers are exact in a double.
#pragma once
#include <cstddef>

#define UW_ST_FULL(X) X(exn0) X(exns0) X(qw0) X(thv0bot) X(thv0top)
#define UW_ST_VEC(X) X(trsrc)
#define UW_ST_DBL(X)                                                                                      \
    X(cin) X(cinlcl) X(plcl) X(plfc) X(exlcl) X(tkeavg) X(qtsrc) X(thlsrc) X(usrc) X(vsrc) X(thv0lcl)   \
    X(cush) X(thlu_top) X(qtu_top) X(exntop) X(drage) X(bogbot) X(bogtop) X(rho0j) X(wtwb) X(wtw)       \
    X(xs1) X(xs2) X(xc1) X(xc2)
#define UW_ST_INT(X) X(xflags) X(lflags) X(kinv) X(klcl) X(klfc)

#define UW_ST_ONE(x) +1
// words of one slot: the lists above, plus tscaleh and errbits
__host__ __device__ inline size_t uw_state_words(int mkx, int ncnst)
{
    const size_t lv = (size_t)mkx + 1;
    return (0 UW_ST_FULL(UW_ST_ONE)) * lv + (0 UW_ST_VEC(UW_ST_ONE)) * (size_t)ncnst + (0 UW_ST_DBL(UW_ST_ONE)) +
           (0 UW_ST_INT(UW_ST_ONE)) + 2;
}

// One scalar to / from the buffer, whatever its type (every integer and float is exact in a double).
#if defined(__CUDACC__)
__device__ __forceinline__ void uw_st_put(double* st, size_t& w, size_t cs, double x) { st[w++ * cs] = x; }
__device__ __forceinline__ void uw_st_put(double* st, size_t& w, size_t cs, float x) { st[w++ * cs] = (double)x; }
__device__ __forceinline__ void uw_st_put(double* st, size_t& w, size_t cs, int x) { st[w++ * cs] = (double)x; }
__device__ __forceinline__ void uw_st_put(double* st, size_t& w, size_t cs, unsigned int x) { st[w++ * cs] = (double)x; }
__device__ __forceinline__ void uw_st_get(const double* st, size_t& w, size_t cs, double& x) { x = st[w++ * cs]; }
__device__ __forceinline__ void uw_st_get(const double* st, size_t& w, size_t cs, float& x) { x = (float)st[w++ * cs]; }
__device__ __forceinline__ void uw_st_get(const double* st, size_t& w, size_t cs, int& x) { x = (int)st[w++ * cs]; }
__device__ __forceinline__ void uw_st_get(const double* st, size_t& w, size_t cs, unsigned int& x)
{
    x = (unsigned int)st[w++ * cs];
}
#endif

// Column code only (names mkx, ncnst, errbits and the listed variables in scope).
#define UW_SV_FULL(a) _Pragma("unroll 4") for (int k_ = 0; k_ <= mkx; k_++) st_[(w_ + k_) * cs_] = a[k_]; w_ += mkx + 1;
#define UW_SV_VEC(a) _Pragma("unroll 1") for (int m_ = 0; m_ < ncnst; m_++) st_[(w_ + m_) * cs_] = a[m_]; w_ += ncnst;
#define UW_SV_ONE(x) uw_st_put(st_, w_, cs_, x);
#define UW_SAVE_STATE(ST, CS, TSCALEH)                                                                    \
    do {                                                                                                  \
        double* const st_ = (ST);                                                                         \
        const size_t cs_ = (CS);                                                                          \
        size_t w_ = 0;                                                                                    \
        UW_ST_FULL(UW_SV_FULL) UW_ST_VEC(UW_SV_VEC)                                                       \
        UW_ST_DBL(UW_SV_ONE) UW_ST_INT(UW_SV_ONE) UW_SV_ONE(TSCALEH) UW_SV_ONE(errbits)                  \
    } while (0)

#define UW_LD_FULL(a) _Pragma("unroll 4") for (int k_ = 0; k_ <= mkx; k_++) a[k_] = st_[(w_ + k_) * cs_]; w_ += mkx + 1;
#define UW_LD_VEC(a) _Pragma("unroll 1") for (int m_ = 0; m_ < ncnst; m_++) a[m_] = st_[(w_ + m_) * cs_]; w_ += ncnst;
#define UW_LD_ONE(x) uw_st_get(st_, w_, cs_, x);
#define UW_LOAD_STATE(ST, CS, TSCALEH)                                                                    \
    do {                                                                                                  \
        const double* const st_ = (ST);                                                                   \
        const size_t cs_ = (CS);                                                                          \
        size_t w_ = 0;                                                                                    \
        UW_ST_FULL(UW_LD_FULL) UW_ST_VEC(UW_LD_VEC)                                                       \
        UW_ST_DBL(UW_LD_ONE) UW_ST_INT(UW_LD_ONE) UW_LD_ONE(TSCALEH) UW_LD_ONE(errbits)                  \
    } while (0)
