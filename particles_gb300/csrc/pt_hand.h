/*
 * pt_hand.h -- slots of the hand-over list (PtHand), reserved by many warps at
 * once.  Host- and device-compilable; no dependencies.
 */
#ifndef PT_HAND_H
#define PT_HAND_H

#if defined(__CUDACC__)
#define PT_HAND_FN __host__ __device__ __forceinline__
#else
#define PT_HAND_FN static inline
#endif

/* Reserves n consecutive slots of a list of cap: returns the first of them, or
 * cap if fewer than n are left.  cas(expected, wanted) compares and swaps the
 * list's count and returns what it held; seen is any value the count has held.
 * A reservation that does not fit leaves the count alone.  (Adding first and
 * subtracting when it did not fit lets another warp reserve above the sum in
 * between: the count then ends below slots that are written, and slots below
 * it are not.)  So the count never exceeds cap and every slot below it belongs
 * to exactly one reservation. */
template <class CAS>
PT_HAND_FN unsigned long long pt_hand_reserve(unsigned long long seen, unsigned long long n,
                                              unsigned long long cap, CAS cas)
{
    while (n <= cap && seen <= cap - n) {
        const unsigned long long was = cas(seen, seen + n);
        if (was == seen) return seen;
        seen = was;
    }
    return cap;
}

#endif /* PT_HAND_H */
