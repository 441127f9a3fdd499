"""Rules of the CUDA programming model that a run cannot show to be broken, read off the kernel sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).parents[1] / "param_decomp_b200" / "ops" / "csrc"


def _kernels(path: Path) -> dict[str, str]:
    parts = re.split(r"(?=__global__)", path.read_text())[1:]
    return {re.search(r"(\w+_kernel)\(", p).group(1): p for p in parts}


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu")))
def test_cluster_barrier_before_a_peers_shared_memory(source):
    """A CTA of a cluster may touch another one's shared memory only once that one is known to run: a cluster barrier stands
    before the first address mapped to a peer."""
    for name, body in _kernels(CSRC / source).items():
        mapped, barrier = body.find("mapa_shared("), body.find("cluster_sync_all()")
        assert mapped < 0 or 0 <= barrier < mapped, name


def test_generic_stores_into_bulk_copy_targets_are_fenced():
    """vocab_kl writes over the columns past V in a buffer that the next row's bulk copy overwrites: the writing thread's
    proxy fence follows each such store."""
    body = _kernels(CSRC / "vocab_kl.cu")["vocab_kl_rows_kernel"]
    stores = [m.end() for m in re.finditer(r"ta\[k\] = tb\[k\] = [^;]*;", body)]
    assert stores and all("fence_proxy_async_smem();" in body[at : at + 60] for at in stores)
