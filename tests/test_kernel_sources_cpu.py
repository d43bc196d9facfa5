"""What a launch on this machine cannot show: rules that every kernel source keeps."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "flex_shard_b200" / "csrc"


def _kernels(path):
    text = re.sub(r"//[^\n]*", "", path.read_text())
    return text.split("__global__")[1:]


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.stem)
def test_a_kernel_waits_for_its_cluster_before_it_addresses_a_peer(path):
    """The shared memory of another CTA of a cluster may be used only once that CTA is known to have started, so a
    cluster barrier comes before the first address in a peer's shared memory."""
    for body in _kernels(path):
        uses = [body.find(s) for s in ("map_to_cta(", "mapa.", "st.shared::cluster", "st.async") if s in body]
        waits = [body.find(s) for s in ("cluster_sync_all(", "cluster_wait(") if s in body]
        assert not uses or (waits and min(waits) < min(uses)), body[:120]
