"""The lanes that the Python sample calls return: what the library wrote, or zeros where it wrote
nothing, whatever the diagnostic says."""

import ctypes as C

import numpy as np
import pytest

from rypath_b200 import abi, native, renderer


class Library:
    """A library whose sample calls write `rows` (None: nothing) and report `status`."""

    def __init__(self, status, text, rows):
        self.status, self.text, self.rows = status, text, rows

    def sample(self, handle, request, out, capacity, diag, cap):
        if self.rows is not None:
            assert capacity == len(self.rows)
            C.memmove(out, self.rows.ctypes.data, self.rows.nbytes)
        diag.value = self.text
        return self.status

    rp_cuda_sample = rp_cuda_sample_scalar = sample

    def rp_cuda_scene_destroy(self, handle):
        pass


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("status,text,written", [
    (abi.RP_SUCCESS, b"", True), (abi.RP_FAILURE, b"lane 2 failed with status 4", True),
    (abi.RP_FAILURE, b"CUDA error out of memory in cudaMallocAsync", False),
    (abi.RP_INVALID_ARGUMENT, b"Render request pixels exceed the film", False)])
def test_lanes_are_the_librarys_or_zeros(monkeypatch, scalar, status, text, written):
    rows = np.zeros(12, abi.scalar_dtype() if scalar else abi.packet_dtype())
    rows["pixel"] = np.arange(12)
    rows["radiance"] = 0.5
    rows["status"][2::3] = 4 if status == abi.RP_FAILURE else 0  # the last lane too
    library = Library(status, text, rows if written else None)
    monkeypatch.setattr(native, "lib", lambda: library)
    scene = renderer.CudaRenderScene(1)
    request = renderer.RenderRequest(4, 3)
    result = scene.sample_scalar(request) if scalar else scene.sample(request)
    scene.close()
    lanes = result.samples if scalar else result.packet_samples
    assert result.status == status and result.diagnostic == text.decode()
    assert lanes.tobytes() == (rows if written else np.zeros_like(rows)).tobytes()
