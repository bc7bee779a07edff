// Blocks of batch members' row steps: "named linear cells block" lines in, the
// member's block out, for a schedule of 128 threads.
#include <cstdint>
#include <iostream>

#include "ops3d.h"

int main() {
    bool named = false, linear = false;
    uint64_t cells = 0;
    while (std::cin >> named >> linear >> cells) {
        std::cout << orr::row_block(128u, named, linear, cells) << "\n";
    }
}
