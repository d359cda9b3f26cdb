"""A batch member stepped by itself inside a caller's graph capture: nothing may
be uploaded or synchronised there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# a domain that steps in tiles, and marches of four and of two levels, whose plans are uploaded by the first step
@pytest.mark.parametrize("shape", [(120, 90), (600, 500), (1100, 900)])
@pytest.mark.parametrize("storage", ["f64", "f32"])
def test_first_steps_of_a_member_under_capture(pkg, shape, storage):
    import torch
    spec = dict(nx=shape[0], ny=shape[1], Ra=1e4, coords=pkg.mesh_box(*shape, 0, 1.0, shape[1] / shape[0], 1.0, "tanh", 1.3))
    b = pkg.Batch(2, [spec], storage=storage)
    c = pkg.Cavity(2, *shape, Ra=1e4, coords=spec["coords"], storage=storage, kernel="direct")
    b.initial()
    c.initial()
    m = b.members[0]
    stream = torch.cuda.ExternalStream(b.stream_ptr())
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        m.step(8)
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    c.step(8)
    m.step(20)  # and outside it
    c.step(20)
    for x, y in zip(m.populations(), c.populations()):
        assert np.array_equal(x, y)
    del graph
    b.close()
    c.close()
