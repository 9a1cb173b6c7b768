// host_blocks_check.cpp -- which host ranges count as lying in one block
// (csrc/host_blocks.hpp): edges, neighbours, freed blocks.
#include <cstdio>

#include "host_blocks.hpp"

static int bad = 0;
static void expect(bool got, bool want, const char *what)
{
    if (got != want) {
        std::printf("%s: %d\n", what, got);
        bad = 1;
    }
}

int main()
{
    static char mem[4096];
    msosm::HostBlocks b;
    expect(b.covers(mem, 1, 5), false, "no blocks");
    b.add(mem + 1000, 100, 5);
    b.add(mem + 1100, 50, 5);  // a direct neighbour is another block
    expect(b.covers(mem + 1000, 100, 5), true, "whole block");
    expect(b.covers(mem + 1040, 60, 5), true, "to its end");
    expect(b.covers(mem + 1040, 61, 5), false, "one byte past its end, into the neighbour");
    expect(b.covers(mem + 999, 10, 5), false, "from before it");
    expect(b.covers(mem + 1100, 50, 5), true, "the neighbour");
    expect(b.covers(mem + 1150, 1, 5), false, "behind both");
    expect(b.covers(mem + 1040, (size_t)-1, 5), false, "a length that wraps");
    expect(b.covers(mem + 1000, 100, 6), false, "a block of another context");
    b.remove(mem + 1000);
    expect(b.covers(mem + 1000, 1, 5), false, "freed");
    expect(b.covers(mem + 1100, 1, 5), true, "the neighbour stays");
    if (!bad)
        std::printf("ok\n");
    return bad;
}
