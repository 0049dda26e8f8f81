"""A kernel may be resident while the launch before it still runs (programmatic dependent launch), so what a forward writes must not be read
through the read-only path, which promises that nobody writes it for the kernel's whole life."""
import re
from pathlib import Path

import fxfusion_b200

KERNELS = Path(fxfusion_b200.__file__).parent / "csrc" / "kernels"
# prepared when the engine is built: bounds of weights, biases of weights in split form (constants of the graph)
CONSTANT = {"p.w_bound", "p.w_bound + 1", "p.v_bound", "p.v_bound + 1", "p.bias + c", "p.bias + grow"}


def test_read_only_loads_are_of_constants():
    seen = 0
    for path in sorted(KERNELS.glob("*.cu*")):
        text = re.sub(r"//.*", "", path.read_text())
        assert "ld.global.nc" not in text, path.name
        args = re.findall(r"__ldg\(([^()]*)\)", text)
        assert len(args) == text.count("__ldg("), path.name
        assert set(args) <= CONSTANT, (path.name, set(args) - CONSTANT)
        seen += len(args)
    assert seen > 0
