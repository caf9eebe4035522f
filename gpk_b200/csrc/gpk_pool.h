// gpk_pool.h — words taken from a pool that the blocks of a launch share.
#pragma once

#ifdef __CUDACC__
#define GPK_POOL_FN __host__ __device__ __forceinline__
#else
#define GPK_POOL_FN inline
#endif

// Takes `need` words of a pool of `pool` words; `at` becomes the first of
// them.  False where they do not fit.  The counter never goes back, so no word
// is given twice, whatever the order in which requests of different sizes
// arrive.  (Taking an addition back where the request did not fit gives words
// twice: the subtraction may follow another block's successful addition.)  A
// request that does not fit adds nothing, unless another one came between its
// reading and its addition: then the counter stays past the end.
// One addition, not a compare-and-exchange: of those, one succeeds per round
// trip to the L2, 5.5 ms for the geometry of 2000 x 2000 cells (7875 tiles)
// instead of 0.28, and 9.55 ms for a 256^3 FP32 step instead of 8.15.
//   Counter::load()    the count, 64 bits wide (additions past the end never wrap it)
//   Counter::add(v)    adds v; returns the count before
template <class Counter>
GPK_POOL_FN bool pool_take(Counter& c, unsigned need, unsigned pool, unsigned& at) {
    if (c.load() + need > pool) return false;
    const unsigned long long old = c.add(need);
    at = (unsigned)old;
    return old + need <= pool;
}
