// The node steps a ray through a mesh is expected to take (expectedNodeSteps in
// albedo_b200/csrc/host/flatten.cpp), on trees small enough to do by hand. Prints
// one line per tree.
#include "host/flatten.hpp"

#include <cstdio>
#include <vector>

using namespace albedo_b200;

namespace {

struct Box {
    float x0, x1, y0, y1, z0, z1;
};

void add(DevNode& n, const Box& b, std::uint32_t child)
{
    const std::uint32_t c{n.count++};
    n.lo_x[c] = b.x0;
    n.hi_x[c] = b.x1;
    n.lo_y[c] = b.y0;
    n.hi_y[c] = b.y1;
    n.lo_z[c] = b.z0;
    n.hi_z[c] = b.z1;
    n.child[c] = child;
}

constexpr std::uint32_t kLeaf{kLeafBit | 5u};

} // namespace

int main()
{
    // Another mesh's node, which counts for nothing here.
    DevNode other{};
    add(other, {0, 100, 0, 100, 0, 100}, 0);
    std::printf("empty %.9g\n", expectedNodeSteps({other}, 1, kEmptyChild));

    DevNode leaf{};
    add(leaf, {0, 1, 0, 2, 0, 3}, kLeaf);
    std::printf("leaf %.9g\n", expectedNodeSteps({other, leaf}, 1, 1));

    // A root of 2 x 2 x 1 (half its surface: 8), in it a node of 1 x 1 x 1 (3), in
    // that one of 1 x 1 x 1/2 (2): 1 + 3/8 + 2/8.
    DevNode root{};
    add(root, {0, 2, 0, 1, 0, 1}, kLeaf);
    add(root, {0, 1, 1, 2, 0, 1}, 2);
    DevNode middle{};
    add(middle, {0, 1, 1, 2, 0.5f, 1}, kLeaf);
    add(middle, {0, 1, 1, 2, 0, 0.5f}, 3);
    add(middle, {0, 1, 1, 1.5f, 0, 1}, kLeaf);
    DevNode low{};
    add(low, {0, 1, 1, 2, 0, 0.5f}, kLeaf);
    std::printf("tree %.9g\n", expectedNodeSteps({other, root, middle, low}, 1, 1));

    // Four children that all fill the root: every ray enters all of them.
    DevNode full{};
    for (std::uint32_t c{0}; c < 4; ++c) {
        add(full, {-1, 1, -1, 1, -1, 1}, 2 + c);
    }
    DevNode end{};
    add(end, {-1, 1, -1, 1, -1, 1}, kLeaf);
    std::printf("full %.9g\n", expectedNodeSteps({other, full, end, end, end, end}, 1, 1));

    // A mesh without extent has no area to compare with.
    DevNode point{};
    add(point, {1, 1, 1, 1, 1, 1}, kLeaf);
    std::printf("point %.9g\n", expectedNodeSteps({other, point}, 1, 1));
    return 0;
}
