// Packs reaction networks for the SSA's packed form (stoch_device.cuh, PackedReaction).
#pragma once
#include <cmath>
#include <cstring>
#include <vector>
#include "stoch_device.cuh"

namespace gpgmp {

// False where a reaction does not fit the packed form: more than two reactant molecules, a
// species named twice among the reactants (its hazard is then A * A, and counts may turn
// negative), a stoichiometry outside 0..kPackedChange (the changes are kept as the upper half
// of a float, exact up to 256) or more than four changed species, a negative or non-finite rate
// (the running sums must not fall).  *nnet: the most species that one reaction changes.
inline bool pack_network(const gpgmp_reaction* r, int R, int S, PackedReaction* out, int* nnet) {
    *nnet = 1;
    for (int k = 0; k < R; ++k) {
        const gpgmp_reaction& a = r[k];
        PackedReaction& o = out[k];
        if (!(a.rate >= 0.0f) || !std::isfinite(a.rate)) return false;
        o.rate = a.rate;
        o.sub = 0.0f;
        o.s1 = o.s2 = 0;
        int molecules = 0, change[MAX_SPECIES] = {};
        for (int j = 0; j < a.num_reactants; ++j) {
            const int sp = a.reactant_species[j], st = a.reactant_stoich[j];
            if (st < 1 || st > 2) return false;
            for (int i = 0; i < j; ++i)
                if (a.reactant_species[i] == sp) return false;
            for (int m = 0; m < st; ++m, ++molecules) {
                if (molecules == 0) o.s1 = sp + 1;
                else if (molecules == 1) { o.s2 = sp + 1; o.sub = (float)m; }
                else return false;
            }
            change[sp] -= st;
        }
        for (int j = 0; j < a.num_products; ++j) {
            if (a.product_stoich[j] < 0 || a.product_stoich[j] > kPackedChange) return false;
            change[a.product_species[j]] += a.product_stoich[j];
        }
        int n = 0;
        for (int s = 0; s < S; ++s) {
            if (change[s] == 0) continue;
            if (n == 4 || change[s] > kPackedChange) return false;
            const float f = (float)change[s];
            uint32_t bits;
            std::memcpy(&bits, &f, 4);
            o.net[n++] = ((uint32_t)(s + 1) << 16) | (bits >> 16);
        }
        if (n > *nnet) *nnet = n;
        for (; n < 4; ++n) o.net[n] = 0u;
    }
    return true;
}

}  // namespace gpgmp
