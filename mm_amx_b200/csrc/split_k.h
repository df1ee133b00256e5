// How the K of a tile is cut into chains of sums.  Plain C++.
#pragma once

namespace b200fc {

// Parts that each of the S CTAs (or pairs) sharing a tile's K of `stages` stored pieces sums one after the other, so that K is summed in
// `chains` chains at least.  even: where a CTA has several, none is longer than K / chains (or one piece), by its longest share; the kernel
// gives part q of a share of n pieces those from n * q / parts on.
inline int parts_of_share(int stages, int S, int chains, bool even) {
    const int share = (stages + S - 1) / S;
    int parts = (chains + S - 1) / S;
    while (even && parts > 1 && parts < share && (long long)((share + parts - 1) / parts) * chains > stages) parts++;
    return parts;
}

}  // namespace b200fc
