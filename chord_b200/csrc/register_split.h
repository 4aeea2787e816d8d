// Whether a kernel's warps can divide its registers: plain C++, so that a host without a GPU can check it
// too.
#pragma once

namespace chord {

// Registers a thread has when a kernel is compiled to `num_regs` (the hardware hands them out in
// eights).
constexpr int allocated_registers(int num_regs) { return (num_regs + 7) / 8 * 8; }

// Whether warps can divide their registers anew (setmaxnreg): what a CTA's warps take afterwards has to
// come out of what it was launched with.  Otherwise the warps that ask for more wait for ever.
constexpr bool register_split_fits(int num_regs, int less_warps, int less_regs, int more_warps, int more_regs) {
  return less_warps * less_regs + more_warps * more_regs <= (less_warps + more_warps) * allocated_registers(num_regs) &&
         less_regs <= allocated_registers(num_regs) && more_regs >= allocated_registers(num_regs);
}

}  // namespace chord
