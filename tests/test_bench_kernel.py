"""The benchmark's roofline entry names the kernel that the choice runs."""
import bench


def test_kernel_label_follows_the_choice(slsf):
    kernels = {"resident": "k_resident", "cluster": "k_cluster", "stream": "k_stream", "grid": "grid-wide"}
    assert set(kernels) == set(slsf.KERNEL_KINDS)
    for kind, name in kernels.items():
        assert bench.kernel_label({"kind": kind, "cluster": 2, "threads": 256}).startswith(name)
