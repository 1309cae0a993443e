// How many layers of a step one launch of the push channel carries.
#pragma once
#include <algorithm>
#include <cstddef>

namespace kvx {

// Both caches on one GPU: half of the layers that are left, at least what makes 4 MiB and at most 128 MiB; the sender waits
// until they are recorded.  A launch costs 5 us on the host, and two to three times that, for both, beside a forward thread
// that records events.  Halving keeps the last launches one layer long, so that nothing but the last layer (or 4 MiB) follows
// the forward pass, and the cap starts a large step with its first layers.  us a step, one launch a layer / this rule: 7 chunks of
// 3001 tokens, 4 heads, 32 layers 339 / 211, 80 fp8 layers of 6005 tokens 883 / 323, 61 MLA layers of 20011 tokens 716 / 420,
// 12 hybrid layers of 30011 tokens 345 / 323, 8192 tokens 470 / 443.
inline size_t layers_per_local_launch(size_t remaining, size_t bytes_per_layer) {
  const size_t per = std::max<size_t>(1, bytes_per_layer);
  const size_t least = std::max<size_t>(1, (4u << 20) / per), most = std::max<size_t>(1, (128u << 20) / per);
  return std::min({remaining, most, std::max(least, (remaining + 1) / 2)});
}

// Towards another GPU no layer is held back for the ones behind it: 128 MiB are 190 us of the link, which a launch of 5 us does
// not pay for.  The attention kernel goes layer by layer, a walk takes what has been recorded meanwhile, up to eight.
inline size_t layers_per_remote_launch(size_t recorded, bool walk) { return walk ? std::min<size_t>(recorded, 8) : 1; }

}  // namespace kvx
