// Sums over the lanes of a warp that share a key (a tet), before an atomic.
#pragma once

namespace mp {

// Sums v[0..N) over the lanes that share `key` (one tet), leaving the sums in
// the group's lowest lane.  All 32 lanes must call it.  Returns true for the
// lanes that hold a group sum.
//
// Pointer jumping over each group's member list: every lane starts pointing at
// the next member above it and holds the sum of the members from itself up to
// (not including) the one it points at; each round adds the pointed-to
// lane's partial sum and takes over its pointer, so ceil(log2(group size))
// rounds leave the whole group's sum in its lowest lane.  A round of four FP64
// sums is one vote, nine shuffles and four adds, and groups need not be contiguous (particles
// that hopped since the last tet sort sit between their tet's others).  This
// replaced a tree over group ranks that located the rank r + s member with a
// bit search each round: FP64 push 0.0905 -> 0.0868 ms, mixed 0.0660 ->
// 0.0592 ms on 2M ions sorted every 10 steps.  Summing runs of adjacent equal
// keys instead (no match) was slower (0.14 ms): a tet's lanes split into
// several runs once particles hop, and every run issues its own atomics.
template <typename T, int N>
__device__ __forceinline__ bool group_sum(int key, T (&v)[N]) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(FULL, key);
    const unsigned above = peers & (0xfffffffeu << lane);  // members above this lane
    int nxt = above ? __ffs(above) - 1 : -1;
    while (__any_sync(FULL, nxt >= 0)) {
        const int src = nxt >= 0 ? nxt : lane;
        T t[N];
#pragma unroll
        for (int i = 0; i < N; i++) t[i] = __shfl_sync(FULL, v[i], src);
        const int n2 = __shfl_sync(FULL, nxt, src);
        if (nxt >= 0) {
#pragma unroll
            for (int i = 0; i < N; i++) v[i] += t[i];
            nxt = n2;
        }
    }
    return (peers & ((1u << lane) - 1u)) == 0;
}

}  // namespace mp
