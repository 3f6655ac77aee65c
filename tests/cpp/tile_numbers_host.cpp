// Prints, for the tiles of the matrix-free operators, whether the number of the last tile of the
// longest accepted side survives its field: name, tiles a side, stored number of the last one.
#include <cstdio>

#include "matfree.cuh"

int main() {
    using namespace mg;
    auto last = [](int own) { return (kMaxSide + own - 1) / own - 1; };  // kMaxSide nodes at most
    MfCol c{};
    c.cx = (decltype(c.cx))last(kCX);
    c.cy = (decltype(c.cy))last(kCY);
    c.cz = (decltype(c.cz))last(kCZ);
    std::printf("col_x %d %d\n", last(kCX), (int)c.cx);
    std::printf("col_y %d %d\n", last(kCY), (int)c.cy);
    std::printf("col_z %d %d\n", last(kCZ), (int)c.cz);
    return 0;
}
