// How many tokens' rows the workspace of a portion gets (engine.cu, stack.cu).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cuda_runtime_api.h>

namespace cq {

// `have` rows stand, a portion wants `need` (at most `most`, what a cache or a cut of a portion allows).  Growing takes twice the rows that stand, so that a
// chat's ever longer portions do not allocate each time; where the device has no room for those, the rows of this portion; and then
// half as many again and again: a portion longer than its workspace goes through the layers in pieces.  bytes(r): memory of r rows.
// take(r): gives the old rows back and takes r new ones, false when the device refused.  What stands is given back only for
// something larger that fits beside what other programs hold.  Returns the rows that stand afterwards, 0 when there is room for none.
template <class Bytes, class Take>
int portion_rows(int have, int need, int most, Bytes bytes, Take take) {
    if (need <= have) return have;
    auto whole = [&](int r) { return std::min(most, (r + 255) / 256 * 256); };
    size_t held = bytes(have);
    for (int r = std::max(whole(need), std::min(most, 2 * have)); r > have;) {
        size_t room = 0, total = 0;
        if (cudaMemGetInfo(&room, &total) != cudaSuccess) { cudaGetLastError(); room = (size_t)-1 / 2; }
        if (bytes(r) <= room + held) {
            if (take(r)) return r;
            cudaGetLastError();                 // an allocation that was refused is no error of a later launch
            have = 0; held = 0;
        }
        const int next = r > whole(need) ? whole(need) : whole((r + 1) / 2);
        if (next >= r) break;                   // 256 rows did not fit
        r = next;
    }
    return have;
}

}  // namespace cq
