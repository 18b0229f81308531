// Rows of a step of the config.json families: what buffers hold and what launches ask for.  Plain arithmetic, the same for every family.
#pragma once
#include <algorithm>

namespace b200 {

constexpr int KX_MAX_STEP = 2048;              // tokens of a step
constexpr int KX_MAX_OUT_ROWS = 512;           // logits rows of a step

// rows of a step's launches: powers of two up to 512 (one graph each), whole tiles of 256 beyond
inline int kx_bucket(int n) {
    for (int b = 8; b <= 512; b *= 2)
        if (n <= b) return b;
    return (n + 255) / 256 * 256;
}
// the next smaller bucket
inline int kx_bucket_below(int b) { return b > 512 ? b - 256 : b / 2; }

// tokens of a portion
inline int kx_portion(int chunk) { return chunk > 256 ? 512 : (chunk > 128 ? 256 : 128); }

// tokens of a step: sixteen chunks (f32-exact models: one portion)
inline int kx_step_tokens(int chunk, bool exact) { return exact ? std::min(chunk, kx_portion(chunk)) : (int)std::min<long long>(16ll * chunk, KX_MAX_STEP); }

// rows every buffer of a step holds: a step's tokens and a whole portion at least, and a bucket itself, since launches cover the bucket of a step's tokens (operands
// are packed and tensor maps encoded with that many rows a group)
inline int kx_max_rows(int chunk, bool exact) { return kx_bucket(std::max(kx_portion(chunk), kx_step_tokens(chunk, exact))); }

}  // namespace b200
