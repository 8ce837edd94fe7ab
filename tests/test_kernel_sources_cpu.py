"""What the kernels' sources must not do, whatever a compiler makes of it today."""
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "parm_gb300" / "csrc"


def test_participation_masks_come_from_data():
    """__activemask() tells which lanes happen to run together, not which lanes take part: a shuffle under it may miss
    its source lane."""
    for f in sorted(CSRC.glob("*.cu*")):
        assert "__activemask" not in f.read_text(), f.name
