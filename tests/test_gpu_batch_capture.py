"""A batch's search recorded into a caller's CUDA graph at its first call."""
import numpy as np
import pytest

from nbodylib_gb300 import BatchedDensity
from nbodylib_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mapping", [0, 1])
def test_first_search_under_capture(gpu, mapping):
    import torch
    pos, _, mass, off = syn.plummer_groups(np.array([20, 1, 333, 0, 2049, 40]), seed=5)
    dpos, dmass, doff = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (pos, mass, off))
    batch = BatchedDensity(dpos, dmass, doff, bucket_size=16, device=True)
    batch.set_query_mapping(mapping)
    stream = torch.cuda.Stream()
    batch.set_stream(stream)
    out = torch.zeros(len(mass), dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        batch.density(32, use_graph=False, out=out)
    graph.replay()
    torch.cuda.synchronize()
    want = batch.density(32, use_graph=False)
    torch.cuda.synchronize()
    np.testing.assert_allclose(out.cpu().numpy(), want.cpu().numpy(), rtol=1e-13)
    batch.close()
