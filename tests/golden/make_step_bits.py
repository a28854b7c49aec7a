"""Golden file of test_gpu_step_bits.py, made on a GPU: step_bits.json, the
CRC-32 of the fields of every class after two steps.  It was made by the library
as it stood before the step of one component had a kernel body of its own; make
it again where a change of rounding is meant, or with another compiler."""
import json
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [os.path.dirname(os.path.dirname(HERE)), os.path.dirname(HERE)]

import step_bits  # noqa: E402

if __name__ == "__main__":
    with open(os.path.join(HERE, "step_bits.json") if len(sys.argv) < 2 else sys.argv[1], "w") as f:
        json.dump({step_bits.name(c): step_bits.crc(c) for c in step_bits.classes()}, f, indent=0, sort_keys=True)
        f.write("\n")
