"""Which products of a few dozen rows go to the kernel that splits the reduction over a cluster."""
import pytest

from pretrained_rstr_b200.parts.linear import cluster_product


@pytest.mark.parametrize("n_out,n_in", [(2304, 768), (3072, 768), (4096, 1024), (4096, 256), (4736, 512)])
def test_wide_outputs_up_to_32_rows(n_out, n_in):
    assert [m for m in range(1, 130) if cluster_product(m, n_out, n_in, 148)] == list(range(17, 33))


@pytest.mark.parametrize("n_out,n_in", [(4737, 512), (4864, 768), (5400, 768), (8192, 512), (32768, 64)])
def test_outputs_whose_tiles_fill_the_device_do_not(n_out, n_in):
    """Nothing is split there: the tensor-memory kernel is up to five times as fast (32,768 x 64)."""
    assert not any(cluster_product(m, n_out, n_in, 148) for m in range(1, 130))


@pytest.mark.parametrize("n_out,n_in", [(768, 768), (768, 3072), (2048, 1600), (1600, 6400), (2560, 10240)])
def test_narrow_outputs_and_long_reductions_up_to_64_rows(n_out, n_in):
    assert [m for m in range(1, 130) if cluster_product(m, n_out, n_in, 148)] == list(range(17, 65))
