// bvh_layout.h -- constants of the wide-node layout shared by the builders
// (host and device) and the traversal kernels.
#pragma once

#include <cstdint>

namespace vkptc {

// Child ref of an unused wide-node slot.  A leaf ref is ~((first << 3) |
// (count - 1)); INT32_MIN = ~0x7FFFFFFF would be the leaf of 8 triangles
// starting at 2^28 - 1, which no scene below kMaxTriangles has.
constexpr int32_t kEmptyChild = INT32_MIN;
// Most triangles in a leaf of the SAH traversal tree.  A triangle test costs
// about as much as testing a node's four boxes, so small leaves pay as long as
// they do not double the nodes.  On the 1,046,904-triangle sphere (camera rays /
// rays from hit points / random rays, G/s) leaves of 1: 4.13 / 2.58 / 3.96,
// 2: 4.29 / 2.68 / 4.56, 3: 4.25 / 2.61 / 4.60, 4: 3.95 / 2.47 / 4.69; on the
// 2,064,386-triangle grid 1: 5.15 / 2.58 / 8.52, 2: 5.47 / 2.80 / 9.28,
// 3: 5.48 / 2.83 / 9.17, 4: 5.17 / 2.64 / 8.04.
constexpr uint32_t kSahLeafMax = 2;
constexpr uint64_t kMaxTriangles = (1ull << 28) - 8u;

}  // namespace vkptc
