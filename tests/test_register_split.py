"""Register split of the step kernels (setmaxnreg): every instantiation is
compiled to the registers a thread that its split counts on, as the compiler
reported them when the library was built.  Fewer would leave setmaxnreg.inc
waiting for registers that the launch never had."""
import os
import re

import pytest

from fletcher_petrobras_gb300.build import OUT

# (kernel, tile rows, extended form) -> registers a thread: Regs, RegsH and
# kLaunchRegs of the sources.
LAUNCH = {("fp32", 16): 168, ("fp32", 12): 168, ("fp32", 8): 128, ("d1d1", 16): 168,
          ("half", 16, 0): 96, ("half", 16, 1): 80, ("half", 12, 0): 128, ("half", 12, 1): 128,
          ("half", 8, 0): 168, ("half", 8, 1): 168}


@pytest.mark.parametrize("source", ["propagate_fp32", "propagate_d1d1", "propagate_half"])
def test_launch_registers(source, lib):
    kind = source.split("_")[1]
    log = open(os.path.join(OUT, source + ".cu.o.log")).read()
    found = re.findall(r"Compiling entry function '\S*k_propagate_%s(\S*)'.*?Used (\d+) registers" % kind, log, re.S)
    assert found
    for name, regs in found:
        # Template arguments: TY, S, ISO, EXT, ... (16-bit forms), TY, S, ISO, ... (FP32).
        args = [int(v) for v in re.findall(r"L[ib](\d+)E", name.split("EEv")[0] + "E")]
        key = (kind, 16) if kind == "d1d1" else (kind, args[0], args[3]) if kind == "half" else (kind, args[0])
        assert int(regs) >= LAUNCH[key], (name, regs)
