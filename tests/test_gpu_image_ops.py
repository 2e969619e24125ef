"""Reconstruct / SampleParticles (particles <-> dense image) on the GPU against the numpy restatement,
plus the reference's own relational pins: gradcheck and sample(reconstruct(x)) == x
(pyapr/tests/test_aprnet.py:248-285)."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle():
    import apr_oracle
    apr_oracle.build()
    return apr_oracle


def _arrays(name):
    if name == "long":                      # rows of 1101 cells: more than a warp holds at a time (512), odd extents, cells of up to 8^3
        from pyapr import synthetic
        gen = torch.Generator().manual_seed(21)
        return synthetic.apr_from_level_map(torch.randint(8, 12, (3, 4, 551), generator=gen).to(torch.int16), (5, 7, 1101))
    return H.arrays(name) if name in H.APR_CASES else H.blob_arrays()


def _apr(name):
    import pyapr
    a = _arrays(name)
    apr = pyapr.apr_from_arrays(a, name)
    apr.init_cuda()
    return a, apr


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 1e-6)])
@pytest.mark.parametrize("name", ["blob", "odd", "odd2", "plane", "ref_shape", "long"])
def test_image_ops_match_oracle(name, dtype, tol, oracle):
    from _pyaprwrapper.data_containers import APRPtrVector
    from _pyaprwrapper.aprnet import cuda as C
    a, apr = _apr(name)
    o = oracle.OracleAPR(a)
    dev = torch.device("cuda:0")
    rng = np.random.RandomState(1)
    for dl in range(0, H.max_dl(a) + 1):
        n = o.number_parts(dl)
        ld = torch.full((1,), dl, dtype=torch.int32)
        x = rng.rand(3, n)
        xt = torch.from_numpy(x).to(dev, dtype)[None].contiguous()
        img = C.reconstruct_forward(APRPtrVector([apr]), xt, ld)
        want = oracle.reconstruct_forward(a, x, dl)
        assert tuple(img.shape[2:]) == want.shape[1:]
        assert H.rel_err(H.t2n(img[0]), want) <= tol, (name, dl)
        g = rng.randn(*want.shape)
        gt = torch.from_numpy(g).to(dev, dtype)[None].contiguous()
        assert H.rel_err(H.t2n(C.reconstruct_backward(APRPtrVector([apr]), gt, ld)[0]), oracle.reconstruct_backward(a, g, dl, n)) <= tol * 64
        assert H.rel_err(H.t2n(C.sample_particles_forward(APRPtrVector([apr]), gt, ld)[0]), oracle.sample_particles_forward(a, g, dl, n)) <= tol * 64
        assert H.rel_err(H.t2n(C.sample_particles_backward(APRPtrVector([apr]), xt, ld)[0]), oracle.sample_particles_backward(a, x, dl)) <= tol


@pytest.mark.parametrize("name", ["blob", "odd", "ref_shape"])
def test_sample_of_reconstruction_is_identity(name):
    from pyapr.aprnet import cuda as aprnet
    a, apr = _apr(name)
    dev = torch.device("cuda:0")
    recon, sample = aprnet.Reconstruct(), aprnet.SampleParticles()
    for dl in range(0, H.max_dl(a) + 1):
        n = int(apr.number_parts(dl)) if hasattr(apr, "number_parts") else None
        import pyapr
        n = int(pyapr.aprnet.utils.number_particles(apr, dl))
        x = torch.rand(2, 4, n, device=dev, dtype=torch.float64)
        ld = torch.full((2,), dl, dtype=torch.int32)
        y = sample(recon(x, [apr, apr], ld), [apr, apr], ld)
        assert torch.allclose(x, y, rtol=0, atol=1e-13)


@pytest.mark.parametrize("name", ["odd", "cube16"])
def test_image_ops_gradcheck(name):
    import pyapr
    from pyapr.aprnet import cuda as aprnet
    from torch.autograd import gradcheck
    a, apr = _apr(name)
    dev = torch.device("cuda:0")
    dl = min(1, H.max_dl(a))
    n = int(pyapr.aprnet.utils.number_particles(apr, dl))
    ld = torch.full((1,), dl, dtype=torch.int32)
    x = torch.rand(1, 2, n, device=dev, dtype=torch.float64, requires_grad=True)
    assert gradcheck(lambda t: aprnet.Reconstruct()(t, [apr], ld.clone()), (x,), eps=1e-6, atol=1e-7)
    img = aprnet.Reconstruct()(x.detach(), [apr], ld.clone())
    im = torch.rand_like(img).requires_grad_(True)
    assert gradcheck(lambda t: aprnet.SampleParticles()(t, [apr], ld.clone()), (im,), eps=1e-6, atol=1e-7)


@pytest.mark.parametrize("channels", [1, 2, 3])
@pytest.mark.parametrize("shape", [(16, 24, 32), (8, 8, 516), (9, 7, 1030)])
def test_image_rows_at_any_alignment(shape, channels):
    """Rows are read in pairs of voxels and stored in 16-byte pieces where their addresses allow it: an image that starts one element further gives the same
    particles bit for bit, and whole, ragged and several pieces of a row give back each cell's value (all of it copies)."""
    from _pyaprwrapper.data_containers import APRPtrVector
    from _pyaprwrapper.aprnet import cuda as C
    import pyapr
    from pyapr import synthetic
    arrays = synthetic.random_apr(shape, 3, density=0.02)
    apr = pyapr.apr_from_arrays(arrays)
    apr.init_cuda()
    ld = torch.zeros(1, dtype=torch.int32)
    torch.manual_seed(5)
    for dtype in (torch.float32, torch.float64):
        flat = torch.randn(1 + channels * shape[0] * shape[1] * shape[2], device="cuda", dtype=dtype)
        shifted = flat[1:].view(1, channels, *shape)
        aligned = shifted.clone()
        parts = C.sample_particles_forward(APRPtrVector([apr]), aligned, ld)
        assert torch.equal(C.sample_particles_forward(APRPtrVector([apr]), shifted, ld), parts)
        image = C.reconstruct_forward(APRPtrVector([apr]), parts, ld)
        fine = C.sample_particles_forward(APRPtrVector([apr]), image, ld)
        assert torch.allclose(fine, parts, rtol=1e-5 if dtype == torch.float32 else 1e-13, atol=0)
        assert torch.equal(image, C.reconstruct_forward(APRPtrVector([apr]), parts, ld))


@pytest.mark.parametrize("dtype,short,long", [(torch.float32, (64, 256, 512), (64, 128, 1024)), (torch.float64, (64, 256, 256), (64, 128, 512))])
@pytest.mark.parametrize("channels", [1, 2, 3])
def test_long_rows_are_painted_as_fast(dtype, short, long, channels):
    """The same volume cut into rows that a warp holds and into rows twice as long: as many voxels, cells and bytes, so about the same time."""
    from _pyaprwrapper.data_containers import APRPtrVector
    from _pyaprwrapper.aprnet import cuda as C
    import pyapr
    from pyapr import synthetic
    took, ld = [], torch.zeros(1, dtype=torch.int32)
    for shape in (short, long):
        apr = pyapr.apr_from_arrays(H.blob_arrays(shape, 80, 7))
        apr.init_cuda()
        x = torch.randn(1, channels, int(pyapr.aprnet.utils.number_particles(apr, 0)), device="cuda", dtype=dtype)
        best = []
        for _ in range(9):
            C.reconstruct_forward(APRPtrVector([apr]), x, ld)
            torch.cuda.synchronize()
            C.profile_enable(True)
            try:
                C.reconstruct_forward(APRPtrVector([apr]), x, ld)
                torch.cuda.synchronize()
                best.append(C.profile_read()["cells_to_image"][1])
            finally:
                C.profile_enable(False)
        took.append(min(best) / x.shape[2])
    assert took[1] < 1.35 * took[0], took


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(3, 5, 256), (3, 5, 257), (3, 5, 511), (3, 5, 513), (2, 9, 1024), (2, 9, 1025), (4, 4, 2100)])
@pytest.mark.parametrize("channels", [1, 2, 5])
def test_rows_around_the_lengths_that_a_warp_holds(shape, channels, dtype):
    """Each voxel is a copy of the value of the cell that covers it, for cells of all sizes, those that reach over several pieces of a row included."""
    from _pyaprwrapper.data_containers import APRPtrVector
    from _pyaprwrapper.aprnet import cuda as C
    import pyapr
    from pyapr import synthetic
    import apr_oracle
    arrays = synthetic.random_apr(shape, 11, density=0.05)
    apr = pyapr.apr_from_arrays(arrays)
    apr.init_cuda()
    for dl in range(2):
        x = torch.randn(1, channels, int(pyapr.aprnet.utils.number_particles(apr, dl)), device="cuda", dtype=dtype)
        got = C.reconstruct_forward(APRPtrVector([apr]), x, torch.full((1,), dl, dtype=torch.int32))[0]
        assert np.array_equal(H.t2n(got), apr_oracle.reconstruct_forward(arrays, H.t2n(x[0]), dl).astype(H.t2n(got).dtype))


def test_more_channels_than_a_grid_has_rows_of_blocks():
    """131,073 channels: painted two at a time they are one more than 65,535 rows of blocks hold."""
    from _pyaprwrapper.data_containers import APRPtrVector
    from _pyaprwrapper.aprnet import cuda as C
    import pyapr
    from pyapr import synthetic
    apr = pyapr.apr_from_arrays(synthetic.apr_from_level_map(torch.full((2, 2, 2), 2, dtype=torch.int16), (4, 4, 4)))
    apr.init_cuda()
    channels, ld = 131073, torch.zeros(1, dtype=torch.int32)
    x = torch.randn(1, channels, 64, device="cuda")
    image = C.reconstruct_forward(APRPtrVector([apr]), x, ld)
    assert torch.equal(C.sample_particles_forward(APRPtrVector([apr]), image, ld), x)


@pytest.mark.parametrize("name", ["reconstruct_forward", "sample_particles_backward"])
def test_painting_allocates_its_result_only(name):
    from _pyaprwrapper.data_containers import APRPtrVector
    from _pyaprwrapper.aprnet import cuda as C
    a = H.blob_arrays((64, 128, 128), 40, 11)
    import pyapr
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    x, ld = torch.randn(1, 8, a.n_particles, device="cuda"), torch.zeros(1, dtype=torch.int32)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    image = getattr(C, name)(APRPtrVector([apr]), x, ld)
    assert torch.cuda.max_memory_allocated() - before <= image.numel() * 4 + 4096
