"""What the benchmark counts: rays traced, kernels launched, bytes moved."""
import bench
from nostrum_pray_gb300 import denoise


def test_shared_camera_rays_are_not_counted_as_traced():
    # two pixels of 4 samples, one bounce each: 8 paths, 16 segments, 2 camera rays
    assert bench.traced_rays(16, [(2, 4)], True) == 10
    assert bench.traced_rays(16, [(2, 4)], False) == 16
    assert bench.traced_rays(100, [(10, 1), (5, 3)], True) == 90


def test_inference_counts():
    """A convolution's epilogue does the pooling, concatenation, residual and
    output transform on the tensor cores at every size, and stores the radiance
    only (3 floats per pixel)."""
    assert denoise.inference_launches() == 20
    assert denoise.inference_launches(False) == 30 == denoise.denoise_launches(128, 128, tensor_cores=False)
    assert denoise.inference_launches() <= denoise.denoise_launches(128, 128)
    assert denoise.inference_bytes(512, 512, 2) == denoise.forward_bytes(512, 512, 2) - 2 * 512 * 512 * 3 * 4
