// Host stand-in for the kernels' programmatic launch hooks: one CTA runs alone.
#pragma once
namespace sfntt {
inline void pdl_trigger() {}
inline void pdl_wait() {}
inline void pdl_enter() {}
}  // namespace sfntt
