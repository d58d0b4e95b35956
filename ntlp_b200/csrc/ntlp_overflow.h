/*
 * ntlp_overflow.h -- the list of deposition tiles that hold more droplets
 * than their stage, left by the tiled kernels to the overflow kernels: a
 * count, ntiles tile indices and a slot that is never read, in an array of
 * 2 + ntiles ints.
 *
 * The tiled kernel appends, the overflow kernel reads, and the last kernel of
 * a deposition clears the count, so the list is empty between depositions.
 * A deposition whose later launches were refused leaves its entries behind:
 * OverflowState remembers that, and the next deposition clears the list
 * before its first kernel.  No entry is ever written or read past the array,
 * whatever the count.
 */
#ifndef NTLP_OVERFLOW_H
#define NTLP_OVERFLOW_H

#ifdef __CUDACC__
#define NTLP_OVF_HD __host__ __device__ __forceinline__
#else
#define NTLP_OVF_HD inline
#endif

namespace ntlp {

/* Appends a tile; add(p) adds one to *p and returns what it held (atomicAdd).
 * What does not fit goes to the last slot: with a branch around the store
 * k_deposit64 took 1.2% longer (1 M droplets on 128^3: 0.3798, not 0.3752 ms). */
template <class Add>
NTLP_OVF_HD void overflow_put(int *list, int ntiles, int tile, Add add) {
    const unsigned at = (unsigned)add(list), end = (unsigned)ntiles;
    list[1 + (at < end ? at : end)] = tile;
}

/* entries that may be read */
NTLP_OVF_HD int overflow_count(const int *list, int ntiles) {
    const int n = list[0];
    return n < 0 ? 0 : (n < ntiles ? n : ntiles);
}

/* host side, one per list: whether its last deposition was launched whole */
struct OverflowState {
    bool unfinished = false;
    /* clear() queues the clearing of the count and returns 0 if it could */
    template <class Clear>
    int ready(Clear clear) {
        if (!unfinished) return 0;
        const int rc = clear();
        if (rc == 0) unfinished = false;
        return rc;
    }
    void begin() { unfinished = true; }   /* before a deposition's first launch */
    void end() { unfinished = false; }    /* when all its launches were accepted */
};

}  // namespace ntlp

#endif
