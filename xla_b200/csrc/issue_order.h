// When the two MMA issuers of tmem_gemm.cu may take the folds in turn.  (Plain C++, without CUDA: the host asks before a launch.)
#pragma once

namespace qmm {

// Step j of the K loop uses barrier j % n of a ring of n, and waits for its phase by parity.  Parity tells a phase from the one
// before it only, so whoever waits for step j has to know already that step j - n has been complete: else it takes the phase
// before that for its own, and the MMA reads an operand that is not there yet.  An issuer knows it of
//   * the steps it waited for itself: those of every second fold;
//   * the steps of all folds that were drained before the last accumulator it waited for.  There are two accumulators and the drain
//     goes in order: the fold two before that one, and all before.
// fu: steps per fold; a_slots, b_slots: the rings; acc_last: a fold's accumulator is waited for after its first step's operands.
constexpr bool issuers_may_alternate(int fu, int a_slots, int b_slots, bool acc_last) {
  for (int q = 0; q < fu; ++q)
    for (int ring = 0; ring < 2; ++ring) {
      const int n = ring ? b_slots : a_slots;
      const int folds_back = n > q ? (n - q + fu - 1) / fu : 0;  // of step q - n of the fold
      const int drained = acc_last && q == 0 ? 4 : 2;
      if (folds_back % 2 != 0 && folds_back < drained) return false;
    }
  return true;
}

}  // namespace qmm
