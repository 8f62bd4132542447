// How decode attention splits a group's keys over CTAs.  Plain host code, so that the rules can be tested without a device.
#pragma once

struct DecodeSplit {
    // grid.x = max_clusters clusters of cl_size CTAs (up to 8); a sequence of `len` keys uses the first
    // ceil(len / cluster_keys) clusters (all of them when cluster_keys == 0)
    int cl_size, max_clusters, cluster_keys;
};

// How a group's keys are split over CTAs.  slots: CTAs of the kernel that are resident at once; groups: (sequence, K/V
// head group) pairs; keys: largest number of keys of a sequence, 0 = unknown (position on the device).
//  * whole grid resident at once: cl_size * max_clusters * groups <= slots (a partial second wave would nearly double
//    the time);
//  * up to 8 CTAs of a group (any number, so that 6 per group fill 444 slots where 4 would leave a third of them empty) form
//    a cluster, merged by asynchronous stores into one another's shared memory; pass_keys = keys that a CTA's warps
//    take in one tile each: a CTA is not given less than one such pass;
//  * further clusters join in (merge through global memory, about 2 us) only for sequences with more than 4 passes per
//    CTA of the first; the kernel decides that per sequence from its actual length;
//  * clusters of five to eight CTAs share one GPC and leave an eighth of its slots empty, so they are counted against 7/8
//    of them (3 fp32 sequences of 32540 keys as 54 clusters of 8 took a second wave: 43 us against 36.5 as 74 splits);
//  * ranges of four and more tiles per warp use clusters of one: any number of splits then fits the machine (9 per group fill
//    296 slots where 8 would leave a tenth of them empty), and the merge is small against the stream.
inline DecodeSplit plan_splits(long long slots, long long groups, long long keys, int pass_keys) {
    DecodeSplit P;
    long long want = slots / groups;
    if (want < 1) want = 1;
    if (want > 256) want = 256;
    const bool known = keys > 0;
    if (known && keys / want >= 4LL * pass_keys) {
        P.cl_size = 1;
        P.max_clusters = (int)want;
        P.cluster_keys = pass_keys;
        return P;
    }
    const long long fit = slots * 7 / 8;
    int c = want < 8 ? (int)want : 8;
    if (c > 4) c = fit / groups > 8 ? 8 : fit / groups < 4 ? 4 : (int)(fit / groups);
    if (known && c > (keys + pass_keys - 1) / pass_keys) c = (int)((keys + pass_keys - 1) / pass_keys);
    P.cl_size = c;
    P.cluster_keys = 4 * c * pass_keys;
    long long k = (c > 4 ? fit / groups : want) / c;
    if (known && k > (keys + P.cluster_keys - 1) / P.cluster_keys) k = (keys + P.cluster_keys - 1) / P.cluster_keys;
    if (!known && k > 4) k = 4;
    P.max_clusters = (int)(k < 1 ? 1 : k);
    return P;
}

// fp32 cache, CTAs of eight warps that have an SM to themselves.  fit[c]: clusters of c such CTAs that the device holds at once,
// by its own count: how many GPCs have room for another cluster of seven or eight does not follow from the number of SMs (148 of
// them hold 15; as 16, or as 17 and 18 of seven, they took a second wave).  False: the four-warp plan.
// us a call, position on the device, at 500 / 4000 / 16000 / 32000 keys; four-warp CTAs | eight-warp CTAs in one cluster of eight | this:
//   12/12 heads  3.7  8.7 12.4 35.3 | 3.2 5.4 16.2 30.9 | as the second           32/8  3.8  9.0 12.1 25.8 | 3.4 6.3 15.7 28.7 | 3.8 8.3 12.6 24.6
//   32/4         4.3 10.1 16.8 27.6 | 4.1 8.5 12.7 18.7 | as the second           72/9  4.7 12.1 22.5 39.6 | 4.2 8.5 23.1 41.7 | 4.6 9.4 18.5 31.6
// (16 groups and more: the four-warp plan, 16/16 4.1 8.9 25.9 44.4.)  Unknown length, more than two query heads a group: clusters of
// eight that leave a fifth of the SMs empty make way for smaller ones, up to 16 CTAs a group, the warps of the four-warp plan: up to
// 8000 keys they lose to the cluster of eight, beyond them they win as much.  With one or two heads the cluster of eight stays: smaller
// ones win at 16000 keys only (12/12 3.5 7.5 14.6 33.0, 16/8 3.6 7.5 10.9 24.2 against 3.2 5.5 12.9 24.9).
inline bool plan_wide(DecodeSplit &P, const int *fit, long long groups, int heads, long long keys, int pass_keys) {
    const bool known = keys > 0;
    int c = known && keys <= 7LL * pass_keys ? (int)((keys + pass_keys - 1) / pass_keys) : 8;
    if (fit[c] < groups) return false;
    int k = 1;
    if (!known) {
        int best = 0;
        for (int n = 8; n >= (heads > 2 ? 4 : 8); --n) {
            const int m = fit[n] / groups < 4 ? (int)(fit[n] / groups) : 4;
            if (n * m > best && (best == 0 || (best < 16 && best * groups * 5 < 4LL * fit[1]))) best = n * m, c = n, k = m;
        }
    }
    P.cl_size = c;
    P.cluster_keys = 4 * c * pass_keys;
    P.max_clusters = k;
    return true;
}
