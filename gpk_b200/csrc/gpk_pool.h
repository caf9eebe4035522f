// gpk_pool.h — words taken from a pool that the blocks of a launch share.
#pragma once

#ifdef __CUDACC__
#define GPK_POOL_FN __host__ __device__ __forceinline__
#else
#define GPK_POOL_FN inline
#endif

// Takes `need` words of a pool of `pool` words; `at` becomes the first of
// them.  False where they do not fit.  The counter moves only with a request
// that fits, and never back: no word is given twice, whatever the order in
// which requests of different sizes arrive.  (Adding first and subtracting
// where the request did not fit gives words twice: a subtraction may follow
// another block's successful addition.)  The loop repeats only where another
// request was granted in between.
//   Counter::load()               the words taken so far
//   Counter::exchange(old, next)  writes next where the value is old; returns
//                                 the value found
template <class Counter>
GPK_POOL_FN bool pool_take(Counter& c, unsigned need, unsigned pool, unsigned& at) {
    unsigned old = c.load();
    while (old <= pool && pool - old >= need) {
        const unsigned found = c.exchange(old, old + need);
        if (found == old) {
            at = old;
            return true;
        }
        old = found;
    }
    return false;
}
