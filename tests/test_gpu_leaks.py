"""A context gives back what it took."""
import pytest

pytestmark = pytest.mark.gpu


def test_tangents_then_shared_memory_systems(edmd):
    """Both use the context's second stream: a lost one keeps ~0.5 MB of the GPU."""
    import torch
    s = edmd.hex_start(60, 0.5, 3)
    s["desc"] = edmd.default_desc(s["N"], s["Lx"], s["Ly"])

    def use(n):
        for _ in range(n):
            eng = edmd.Engine([s], engine=edmd.ENGINE_WARP)
            eng.tangent(1, 4, 2)
            eng.advance(max_coll=3, flags=edmd.F_SMEM)
            eng.close()

    use(20)
    free = torch.cuda.mem_get_info()[0]
    use(80)
    assert free - torch.cuda.mem_get_info()[0] < 16 << 20
