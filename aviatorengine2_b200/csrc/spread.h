// spread.h - how a launch with few rays lays them out over its warps.  Plain
// C++, so that the rules can be tested without a GPU.
#pragma once
#include <stdint.h>

#include "ae_math.h"

namespace ae {

// The share of each of half the warps (at least one) when `count` rays meet a
// launch's `warps`; for any two numbers.
AE_HD uint32_t spread_share(uint32_t count, uint32_t warps) {
    const uint32_t half = warps > 1u ? warps / 2u + (warps & 1u) : 1u;
    return count / half + (count % half ? 1u : 0u);
}

// How many lanes of each warp take rays: all 32, or, with few rays, so few
// that the rays occupy about half of the warps.  Lanes that diverge then wait
// for fewer neighbours, which is what a small launch's time is made of (it
// lasts as long as its slowest rays), and idle warps cost nothing.  Random rays
// through 200 instances, one ray a thread / step-wise walk, all lanes ->
// spread: 500 rays 165 -> 65 / 155 -> 100 us, 8,000 rays 193 -> 115 / 184 -> 135
// us, 20,000 rays 197 -> 149 / 175 -> 172 us.  From a quarter of the lanes on,
// full warps issue less and win (50,000 rays: 199 -> 213 us on the walk), hence
// the limit of 16.  Launches that can walk a ray by four lanes ask spread_quads
// first and come here above its range, for 9 to 16 lanes.
AE_HD uint32_t spread_lanes(uint32_t count, uint32_t warps) {
    const uint32_t l = spread_share(count, warps);
    return l > 16u ? 32u : (l ? l : 1u);
}

// How many quads of each warp take a ray (quad_walk.cuh), or 0 where eight in
// half of the warps do not reach (20,000 rays: 149 us either way).
AE_HD uint32_t spread_quads(uint32_t count, uint32_t warps) {
    const uint32_t q = spread_share(count, warps);
    return q > 8u ? 0u : (q ? q : 1u);
}

}  // namespace ae
