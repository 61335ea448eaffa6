"""Memory order of the device BVH's bottom-up pass (sol_b200/csrc/kernels/lbvh.cu), read from its source.

One lane's atomic and fence acquire a node's subtree, and then all lanes of the
warp read it.  Votes and shuffles order no memory between lanes, so warp
barriers have to stand at the hand-overs; a missing one gives right results on
most runs, which is why the source is checked."""
import re
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "sol_b200" / "csrc" / "kernels" / "lbvh.cu"


def _bottom_up():
    text = SRC.read_text()
    body = text[text.index("bottom_up(Tree t, int n"):]
    body = re.sub(r"//[^\n]*", "", body[:body.index("\n}\n")])
    at = [(m.start(), m.group(1)) for m in re.finditer(
        r"(atomicAdd|__threadfence|__syncwarp|t\.leaf\[node\] =|__ballot_sync|restructure)", body)]
    return [name for _, name in at]


def test_every_lane_is_ordered_after_the_arrival():
    seq = _bottom_up()
    # release, arrive, acquire, publish the node, barrier, vote, treelet, fence by every writer, barrier
    assert seq == ["__threadfence", "atomicAdd", "__threadfence", "t.leaf[node] =", "__syncwarp", "__ballot_sync",
                   "restructure", "__threadfence", "__syncwarp"]
