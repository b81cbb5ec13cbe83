// jt_batchmix_params.cuh -- a batch step of jt_batchmix.cuh.
#pragma once

#include "jt_bluemix.cuh"

namespace jt {

struct BatchMix {
    MixParams f, g;           // g: the inverse passes of a step with a turn
    const float2 *twf, *twg;
    const float2 *Bp;         // turn: the chirp's spectrum, a row per line number modulo n1
    int n1;
    int cols_in, cols_out;    // walk lines first
    int inv, turn;
    int chirp_in, chirp_out;  // 1: rows, 2: columns of the n1 x n2 view
    MixBlue bl;
};

}  // namespace jt
