// Device state of one block-RPCholesky round, shared by the round kernels.
#pragma once

#include <cstdint>

namespace kevd {

struct RoundState {
    int64_t rank;    // columns of F written
    int64_t r_old;   // rank before this round's update
    int32_t nacc;    // accepted this round
    int32_t done;    // set once the factorisation has stopped
    int32_t rounds;  // rounds executed
    int32_t cur;     // index of the round being worked on
    double total;    // sum of d after the last update
};

}  // namespace kevd
