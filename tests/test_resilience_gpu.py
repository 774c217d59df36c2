"""Failure detection without a GPU fault, and checkpoint/resume.

* A bounded wait that nothing completes gives up, records its code in the workspace error
  word and returns; the host reads the word and raises; the context stays usable.
* Optimiser state saved to disk and loaded into a new optimiser continues bit-identically.
* Each SvbrdfOptim.optim call starts a fresh Adam, as the reference's does."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _mats(svb, n=3):
    from oracle import microfacet_ref as R
    return svb.scenes.batched_scenes(n=n, resolutions=(16, 32), vmin=3, vmax=7,
                                     render_fn=lambda *a: R.render(*a, dtype=torch.float32))


def test_bounded_wait_times_out_and_reports(svb, cuda):
    N = svb._native
    L = N.lib()
    ws = torch.zeros(16, dtype=torch.uint8, device=cuda)
    N.check(L.svbrdf_selftest_wait_timeout(ws.data_ptr(), ws.numel(), 2000, N.stream_handle(cuda)))
    torch.cuda.synchronize()
    w = ws.view(torch.int32).cpu().tolist()
    assert w[1] == 1  # "copy never landed"
    assert w[2] == 1 and w[3] == 0  # the completed wait, the one that ran out
    # the context is still usable: a batched run afterwards is healthy
    b = svb.BatchedOptim(_mats(svb, 2), device=cuda, config=svb.BatchConfig(480, 960, 0, 3))
    b.run(3)
    b.check()
    assert b.device_error() == 0


def test_host_turns_the_error_word_into_an_exception(svb, cuda):
    """The word a timed-out launch leaves (set here from the host) fails the next check."""
    N = svb._native
    b = svb.BatchedOptim(_mats(svb, 2), device=cuda, config=svb.BatchConfig(480, 960, 0, 2))
    b.run(2)
    b.check()
    off = N.WORKSPACE_ERROR_OFFSET
    b.ws[off:off + 4].view(torch.int32).fill_(2)
    assert b.device_error() == 2
    with pytest.raises(svb.SvbrdfError):
        b.check()


@pytest.mark.parametrize("variant", [1, 2, 3, 4])
def test_launch_under_a_set_error_word_returns(svb, cuda, variant):
    """Every wait of a launch whose workspace holds an error code may give up at once, with copies in
    flight: the launch drains them, returns and keeps the code, and the next plan is healthy."""
    off = svb._native.WORKSPACE_ERROR_OFFSET
    cfg = svb.BatchConfig({1: 480, 2: 480, 3: 480, 4: 512}[variant], {1: 480, 4: 1024}.get(variant, 960), 0, variant)
    b = svb.BatchedOptim(_mats(svb), device=cuda, config=cfg, hist_len=4)
    b.ws[off:off + 4].view(torch.int32).fill_(2)
    b.run(4)
    assert b.device_error() == 2
    runs = []
    for _ in range(2):
        c = svb.BatchedOptim(_mats(svb), device=cuda, config=cfg, hist_len=4)
        c.run(4)
        c.check()
        runs.append(c)
    assert torch.equal(runs[0].loss_hist, runs[1].loss_hist) and torch.isfinite(runs[0].loss_hist).all()
    assert all(torch.equal(x, y) for x, y in zip(runs[0].tex, runs[1].tex))


@pytest.mark.parametrize("gram", [True, False])
def test_tensor_core_launches_under_a_set_error_word_return(svb, cuda, gram):
    """The waits of the tensor-core kernels may give up in any warp while the error word is set: the
    launches wait for their loads, return and keep the code, and the next descriptor and
    convolutions are healthy."""
    N = svb._native
    gen = torch.Generator().manual_seed(5)
    tgt, cur = (torch.rand(2, 3, 256, 256, generator=gen).to(cuda) for _ in range(2))
    make = lambda: svb.descriptor.VGGDescriptor(cuda, seed=2, mode="config" if gram else "reference")
    d = make()
    d.load(tgt)
    d.err.fill_(41)
    for _ in range(3):
        d._loss_and_grad_eager(cur)
    assert d.device_error() == 41
    x, w = (torch.rand(*s, generator=gen).to(cuda) for s in ((2, 64, 64, 64), (64, 9 * 64)))
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    outs = []
    for code in (41, 0, 0):
        err.fill_(code)
        y = torch.zeros_like(x)
        N.check(N.lib().svbrdf_gen_conv_tf32(x.data_ptr(), w.data_ptr(), y.data_ptr(), 2, 64, 64, 64, 64, 3, 1,
                                             err.data_ptr(), N.stream_handle(cuda)))
        assert int(err.item()) == code
        outs.append(y)
    assert torch.equal(outs[1], outs[2]) and bool((outs[1] > 0).all())
    runs = []
    for _ in range(2):
        e = make()
        e.load(tgt)
        runs.append(e._loss_and_grad_eager(cur))
        assert e.device_error() == 0
    assert all(torch.equal(a, b) and torch.isfinite(a).all() for a, b in zip(*runs))


@pytest.mark.parametrize("ctas", [0, 5])
@pytest.mark.parametrize("variant,light", [(2, True), (3, True), (2, False), (3, False)])
def test_workspace_is_usable_again_once_the_word_is_zeroed(svb, cuda, variant, light, ctas):
    """A launch that gave up (here because its workspace held an error code: with a learnable light
    the CTAs of variant 2 leave at their first wait for one another, with iterations to go) leaves
    no count behind: with the word zeroed and the fit reset, the same plan runs as a fresh one."""
    off = svb._native.WORKSPACE_ERROR_OFFSET
    make = lambda: svb.BatchedOptim(_mats(svb), device=cuda, config=svb.BatchConfig(480, 960, ctas, variant),
                                    hist_len=9, optim_light=light)
    b = make()
    word = b.ws[off:off + 4].view(torch.int32)
    for iters in (5, 1, 9):
        word.fill_(2)
        b.run(iters)
        assert b.device_error() == 2
        word.zero_()
        assert int(b.ws[:4].view(torch.int32).item()) == 0  # the completion counter
    b.reset(inits=[m.init for m in _mats(svb)])
    b.run(9)
    b.check()
    c = make()
    c.run(9)
    c.check()
    assert torch.equal(b.loss_hist, c.loss_hist)
    for i in range(b.n):
        assert torch.equal(b.tex[i], c.tex[i]) and torch.equal(b.light_pow(i), c.light_pow(i))


@pytest.mark.parametrize("variant", [2, 3])
def test_batched_checkpoint_resume_is_exact(svb, cuda, tmp_path, variant):
    mats = _mats(svb)
    cfg = svb.BatchConfig(480, 960, 0, variant)
    a = svb.BatchedOptim(mats, device=cuda, config=cfg, hist_len=20)
    a.run(5)
    a.save(tmp_path / "ck.pt")
    a.run(7)
    b = svb.BatchedOptim(mats, device=cuda, config=cfg, hist_len=20)
    b.load(tmp_path / "ck.pt")
    b.run(7)
    for i in range(len(mats)):
        assert torch.equal(a.tex[i], b.tex[i])
        assert torch.equal(a.m1[i], b.m1[i]) and torch.equal(a.m2[i], b.m2[i])
    assert torch.equal(a.loss_hist, b.loss_hist)
    assert int(b.step_dev.item()) == 12 and b.step_count == 12
    other = svb.BatchedOptim(_mats(svb, 2), device=cuda, config=cfg, hist_len=20)
    with pytest.raises(ValueError):
        other.load(tmp_path / "ck.pt")


def test_fused_optim_calls_start_fresh_adam_and_checkpoint(svb, cuda, tmp_path):
    """Two optim calls follow the reference's two loops, each with a new Adam; the maps
    saved after them load into a new optimiser unchanged."""
    from oracle import microfacet_ref as R
    sc = svb.scenes.single_scene(res=64, seed=1014)
    svb.scenes.add_targets(sc, lambda *a: R.render(*a, dtype=torch.float32))
    r = svb.Microfacet(64, 9, sc.size, [t.to(cuda) for t in sc.cl], cuda)
    o = svb.SvbrdfOptim(cuda, r, loss="log1p")
    o.load_targets(sc.targets.to(cuda))
    o.init_from_tex(sc.init.to(cuda))
    o.optim(3, 0.01, None, False)
    o.optim(4, 0.01, None, False)
    ref = R.optim_loop(sc.init, sc.targets, sc.camera_pos, sc.light_pos, sc.light_pow, sc.size, 3, 0.01, "log1p",
                       False, torch.float64)
    ref = R.optim_loop(ref["textures"], sc.targets, sc.camera_pos, sc.light_pos, sc.light_pow, sc.size, 4, 0.01,
                       "log1p", False, torch.float64)
    assert rel_l2(o.textures.detach(), ref["textures"]) <= 2e-5
    assert rel_l2(o.exp_avg_sq, ref["exp_avg_sq"]) <= 1e-4
    o.save(tmp_path / "perpixel.pt")
    o2 = svb.SvbrdfOptim(cuda, r, loss="log1p")
    o2.load(tmp_path / "perpixel.pt")
    assert torch.equal(o2.textures.detach(), o.textures.detach())
    assert o2._step == 4 and o2.loss_image_list == o.loss_image_list


def test_latent_save_and_resume(svb, cuda, tmp_path):
    gen = svb.materialgan.StyleGAN2Generator(resolution=32, fmap_max=32, seed=0)
    sc = svb.scenes.single_scene(res=32, seed=1015)
    r = svb.Microfacet(32, 9, sc.size, [t.to(cuda) for t in sc.cl], cuda)
    o = svb.materialgan.MaterialGANOptim(cuda, r, gen)
    o.load_targets(torch.rand(9, 3, 32, 32).to(cuda))
    o.init_from(batch=1, seed=3, noise="random")
    o.save_latent(tmp_path / "optim_latent.pt", tmp_path / "optim_noise.pt")
    t0 = o.latent_to_textures().detach()
    o2 = svb.materialgan.MaterialGANOptim(cuda, r, gen)
    o2.load_targets(torch.rand(9, 3, 32, 32).to(cuda))
    o2.init_from(batch=1, seed=99)
    o2.load_latent(tmp_path / "optim_latent.pt", tmp_path / "optim_noise.pt")
    assert torch.equal(o2.latent_to_textures().detach(), t0)
