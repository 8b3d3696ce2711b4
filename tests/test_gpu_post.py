"""Tonemapping and denoising on the GPU.  kgr_tonemap against the oracle's
restatement of include/cuda/color.cuh: ACES bit for bit; sRGB within one
8-bit step (powf's last bit differs between the device and the host C
library; at least 99% of channels equal).  The denoiser against its NumPy
restatement (rtol 1e-4: expf/powf ulps through five passes), and on a
path-traced frame: the denoised 4-spp image is closer to the 1024-spp
reference than the raw one."""
import numpy as np
import pytest

from artemis_gb300 import kgr
from oracle import post_ref, pyoracle
from tests import helpers

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [kgr.TONEMAP_ACES, kgr.TONEMAP_SRGB])
def test_tonemap_matches_oracle(mode):
    rng = np.random.default_rng(mode)
    h, w = 23, 37  # not multiples of the 16 x 16 block
    hdr = np.zeros((h, w, 4), np.float32)
    hdr[..., :3] = (10.0 ** rng.uniform(-4, 2, (h, w, 3))).astype(np.float32)
    hdr[0, 0, :3] = [0.0, 0.0031308, 1e6]
    d_hdr = torch.from_numpy(hdr).cuda()
    d_ldr = torch.zeros((h, w), dtype=torch.int32, device="cuda")
    kgr.tonemap(d_hdr.data_ptr(), d_ldr.data_ptr(), w, h, mode)
    got = d_ldr.cpu().numpy().view(np.uint32)
    ref = pyoracle.tonemap(hdr, mode)
    if mode == kgr.TONEMAP_ACES:
        np.testing.assert_array_equal(got, ref)
    else:
        ch = lambda a: np.stack([(a >> s) & 0xFF for s in (0, 8, 16, 24)], -1).astype(np.int32)
        diff = np.abs(ch(got) - ch(ref))
        assert diff.max() <= 1 and (diff == 0).mean() >= 0.99


def render_with_aovs(g, sc, w, h, spp, frame):
    cam = kgr.camera(g.eye, g.target, g.fov, w / h)
    bufs = helpers.device_buffers(torch, w * h)
    att = kgr.Attachment("path_tracer")
    att.attach(w, h)
    att.load()
    att.set_option("spp", spp)
    att.set_option("russian_roulette", True)
    att.render(helpers.launch(cam, w, h, bufs, frame=frame, max_depth=6), sc)
    torch.cuda.synchronize()
    att.close()
    return bufs


def result_array(dn, w, h):
    """The denoiser's result buffer (device) as a (w*h, 4) array."""
    return dn.copy_result(np.zeros((w * h, 4), np.float32))


@pytest.mark.parametrize("guides", [kgr.DENOISE_NORMAL | kgr.DENOISE_ALBEDO | kgr.DENOISE_POSITION,
                                    kgr.DENOISE_NORMAL, kgr.DENOISE_NONE])
def test_denoiser_matches_oracle(guides):
    g, sc, _ = helpers.both("box4k", 1)
    w, h = 72, 56
    bufs = render_with_aovs(g, sc, w, h, 2, 3)
    dn = kgr.Denoiser(w, h, guides)
    dn.denoise(bufs[0].data_ptr(), bufs[1].data_ptr(), bufs[2].data_ptr(), bufs[3].data_ptr())
    torch.cuda.synchronize()
    cpu = [b.cpu().numpy().reshape(h, w, 4) for b in bufs]
    got = result_array(dn, w, h).reshape(h, w, 4)
    ref = post_ref.denoise(cpu[0], cpu[1], cpu[2], cpu[3], guides)
    np.testing.assert_allclose(got, ref, rtol=1e-4, atol=1e-6)
    dn.close()


def test_denoising_lowers_relmse():
    g, sc, _ = helpers.both("box4k", 1)
    w, h = 128, 128
    ref = np.zeros((w * h, 3))
    n_ref = 64
    for f in range(n_ref):
        ref += render_with_aovs(g, sc, w, h, 16, 1000 + f)[0].cpu().numpy()[:, :3]
    ref /= n_ref
    bufs = render_with_aovs(g, sc, w, h, 4, 7)
    dn = kgr.Denoiser(w, h)
    dn.denoise(bufs[0].data_ptr(), bufs[1].data_ptr(), bufs[2].data_ptr(), bufs[3].data_ptr())
    rel = lambda x: float(np.mean((x - ref) ** 2 / (ref ** 2 + 1e-2)))
    raw, den = rel(bufs[0].cpu().numpy()[:, :3]), rel(result_array(dn, w, h)[:, :3])
    print(f"relMSE 4 spp: raw {raw:.4f}, denoised {den:.4f}")
    assert den < 0.5 * raw
    dn.close()


@pytest.mark.parametrize("power", [0.0, 1.0, 2.0, 32.0, 63.5, 64.0, 1024.0])
def test_every_normal_power_matches_oracle(power):
    """Powers of two go by squaring, 64 by a loop of its own, others by powf."""
    g, sc, _ = helpers.both("box4k", 1)
    w, h = 37, 21
    bufs = render_with_aovs(g, sc, w, h, 2, 3)
    guides = kgr.DENOISE_NORMAL | kgr.DENOISE_POSITION
    dn = kgr.Denoiser(w, h, guides)
    dn.denoise(bufs[0].data_ptr(), bufs[1].data_ptr(), None, bufs[3].data_ptr(), iterations=3, normal_power=power)
    torch.cuda.synchronize()
    cpu = [b.cpu().numpy().reshape(h, w, 4) for b in bufs]
    got = result_array(dn, w, h).reshape(h, w, 4)
    ref = post_ref.denoise(cpu[0], cpu[1], cpu[2], cpu[3], guides, iterations=3, normal_power=power)
    np.testing.assert_allclose(got, ref, rtol=1e-4, atol=1e-6)
    dn.close()


def test_infinite_and_nan_pixels_stay_where_they_are():
    """A non-finite colour reaches only the taps of its own kind (hit or miss)."""
    w, h = 33, 9
    color = torch.rand((h, w, 4), device="cuda")
    normal = torch.zeros((h, w, 4), device="cuda")
    normal[:, :16, 2] = 1.0
    color[4, 20, 0], color[2, 25, 1] = float("nan"), float("inf")
    dn = kgr.Denoiser(w, h, kgr.DENOISE_NORMAL)
    dn.denoise(color.data_ptr(), normal.data_ptr(), iterations=2)
    torch.cuda.synchronize()
    got = result_array(dn, w, h).reshape(h, w, 4)
    assert np.isfinite(got[:, :16]).all()
    assert np.isnan(got[4, 20, 0]) and not np.isfinite(got[2, 25, 1])
    dn.close()


@pytest.mark.parametrize("w,h", [(2, 262140), (2, 262141), (1, 600001), (3000001, 1)])
def test_narrow_images_of_many_rows_or_columns(w, h):
    """More rows than a grid's second dimension holds blocks of, and one row
    of many columns: every extent that the creation accepts is filtered."""
    rng = np.random.default_rng(h)
    color = rng.uniform(0.1, 2.0, (h, w, 4)).astype(np.float32)
    normal = np.zeros((h, w, 4), np.float32)
    normal[..., 2] = 1.0
    bufs = [torch.from_numpy(b).cuda() for b in (color, normal)]
    dn = kgr.Denoiser(w, h, kgr.DENOISE_NORMAL)
    dn.denoise(bufs[0].data_ptr(), bufs[1].data_ptr(), iterations=2)
    torch.cuda.synchronize()
    got = result_array(dn, w, h).reshape(h, w, 4)
    ref = post_ref.denoise(color, normal, None, None, kgr.DENOISE_NORMAL, iterations=2)
    np.testing.assert_allclose(got, ref, rtol=1e-4, atol=1e-6)
    dn.close()


def pairs(n, tap_normals, tap_colors, tap_positions=None):
    """n pairs of pixels that only meet each other: three rows apart, sky
    between them.  The left pixel of a pair is black, at the origin, its
    normal (0, 0, 1).  (color, normal, position), float32 (3 n, 2, 4)."""
    bufs = [np.zeros((3 * n, 2, 4), np.float32) for _ in range(3)]
    bufs[0][::3, 1, :3] = np.asarray(tap_colors, np.float32)[:, None]
    bufs[1][::3, 0, 2] = 1.0
    bufs[1][::3, 1, :3] = tap_normals
    if tap_positions is not None:
        bufs[2][::3, 1, :3] = tap_positions
    return bufs


def tap_weight(bufs, guides, **params):
    """The weight of a pair's right pixel in the left one's mean, from the
    filter's result in double precision: r = w c / (9/64 + w)."""
    dev = [torch.from_numpy(b).cuda() for b in bufs]
    h = len(bufs[0])
    dn = kgr.Denoiser(2, h, guides)
    dn.denoise(dev[0].data_ptr(), dev[1].data_ptr(), None, dev[2].data_ptr(), iterations=1, **params)
    torch.cuda.synchronize()
    r = result_array(dn, 2, h).reshape(h, 2, 4)[::3, 0, 0].astype(np.float64)
    dn.close()
    c = bufs[0][::3, 1, 0].astype(np.float64)
    return r * (9.0 / 64.0) / (c - r)


@pytest.mark.parametrize("power", [64.0, 32.0, 2.0])
def test_normal_weight_is_good_to_a_few_ulp(power):
    """The cosine is the tap normal's z itself.  Roundings: the power 1 ulp,
    its product with the spline, the sum's product, the sum of weights and
    the mean half an ulp each: 3 ulp, of 2^-23 relative at most.  Cosines
    whose power is below 2^-18, so that w + 9/64 does not feel w's error."""
    rng = np.random.default_rng(int(power))
    z = (rng.uniform(2.0 ** -60, 2.0 ** -18, 4096) ** (1.0 / power)).astype(np.float32)
    normals = np.stack([np.sqrt(1.0 - z.astype(np.float64) ** 2), np.zeros(len(z)), z], 1).astype(np.float32)
    bufs = pairs(len(z), normals, np.ones(len(z)))
    got = tap_weight(bufs, kgr.DENOISE_NORMAL, normal_power=power, sigma_color=1e30)
    want = 3.0 / 32.0 * z.astype(np.float64) ** power
    assert np.abs(got / want - 1.0).max() <= 3.0 * 2.0 ** -23


def test_normals_longer_than_one_overflow_as_a_power_does():
    """A cosine above 1 whose power exceeds the largest float: the weight is
    infinite and the mean not a number, as with powf."""
    normals = np.tile(np.array([[0.0, 0.0, 100.0]], np.float32), (4, 1))
    bufs = pairs(4, normals, np.ones(4))
    got = [tap_weight(bufs, kgr.DENOISE_NORMAL, normal_power=p, sigma_color=1e30) for p in (64.0, 65.0)]
    assert np.isnan(got[0]).all() and np.isnan(got[1]).all()


def test_color_weight_is_good_to_its_argument():
    """The argument x = l / (sigma l / 2 + 1e-4) has three rounded steps
    (2^-24 relative each; the luminance's own rounding cancels but for the
    1e-4); the exponential may be 2 ulp off, the other steps 2 ulp."""
    rng = np.random.default_rng(3)
    sigma = 2.0 / 64.0
    c = rng.uniform(0.5, 8.0, 4096).astype(np.float32)
    normals = np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (len(c), 1))
    got = tap_weight(pairs(len(c), normals, c), kgr.DENOISE_NONE, sigma_color=sigma)
    k = [float(np.float32(v)) for v in (0.2126, 0.7152, 0.0722)]
    lum = c.astype(np.float64) * sum(k)
    x = lum / (0.5 * sigma * lum + float(np.float32(1e-4)))
    want = 3.0 / 32.0 * np.exp(-x)
    # the luminance's rounding (3 ulp at most) changes x by 1e-4 / (sigma l / 2) of itself
    bound = x * (3.0 * 2.0 ** -24 + 3.0 * 2.0 ** -23 * 1e-4 / (0.5 * sigma * lum)) + 4.0 * 2.0 ** -23
    assert (np.abs(got / want - 1.0) <= bound).all()


def test_position_weight_is_good_to_its_argument():
    """The argument d / sigma: the squared length (two rounded steps, half of
    them through the root), the quotient over the root (3.5), the rate and
    its product: 6.5 x 2^-24 relative; the exponential and the rest 4 ulp."""
    rng = np.random.default_rng(4)
    n, sigma = 4096, 1.0 / 64.0
    q = np.zeros((n, 3), np.float32)
    q[:, 0], q[:, 2] = rng.uniform(0.5, 2.0, n), rng.uniform(0.2, 1.0, n)
    normals = np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (n, 1))
    got = tap_weight(pairs(n, normals, np.ones(n), q), kgr.DENOISE_POSITION, sigma_color=1e30, sigma_position=sigma)
    v = q.astype(np.float64)
    x = v[:, 2] / np.sqrt((v * v).sum(1)) / sigma
    want = 3.0 / 32.0 * np.exp(-x)
    assert (np.abs(got / want - 1.0) <= x * 6.5 * 2.0 ** -24 + 4.0 * 2.0 ** -23).all()


@pytest.mark.parametrize("sigma_position", [1e-39, 1e-30, 1e30])
def test_extreme_sigmas_and_values(sigma_position):
    """Taps in the centre's plane weigh 1 whatever the sigma; positions and
    colours whose squares or sums leave the range of a float, and negative
    colours that make a denominator 0, give what the formula gives."""
    n = 4
    normals = np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (n, 1))
    q = np.array([[1.0, 0, 0], [1e-30, 0, 0], [1e25, 0, 0], [3e38, 0, 0]], np.float32)
    got = tap_weight(pairs(n, normals, np.ones(n), q), kgr.DENOISE_POSITION, sigma_color=1e30,
                     sigma_position=sigma_position)
    np.testing.assert_allclose(got, 3.0 / 32.0, rtol=1e-6)
    # luminances of 3e38 (their sum is infinite, the weight 1), and of -1e-4 with sigma 2 (the denominator 0,
    # the weight exp(-inf))
    for color, sigma, weight in ((3e38, 2.0, 3.0 / 32.0), (-1e-4, 2.0, 0.0)):
        bufs = pairs(n, normals, np.full(n, color, np.float32))
        if color > 0:
            bufs[0][::3, 0, :3] = 1e38
        dev = [torch.from_numpy(b).cuda() for b in bufs]
        dn = kgr.Denoiser(2, 3 * n, kgr.DENOISE_NONE)
        dn.denoise(dev[0].data_ptr(), dev[1].data_ptr(), iterations=1, sigma_color=sigma)
        torch.cuda.synchronize()
        r = result_array(dn, 2, 3 * n).reshape(3 * n, 2, 4)[::3, 0, 0]
        dn.close()
        c0, c1 = float(bufs[0][0, 0, 0]), float(np.float32(color))
        np.testing.assert_allclose(r, (c0 * 9 / 64 + weight * c1) / (9 / 64 + weight), rtol=1e-5)


@pytest.mark.parametrize("own_result", [False, True])
@pytest.mark.parametrize("iterations", [1, 2, 4, 5])
def test_albedo_guide_at_every_parity_of_the_passes(iterations, own_result):
    """The demodulated image goes where the first pass does not write, scratch
    or result by the number of passes; the colour may be the denoiser's own
    result buffer."""
    g, sc, _ = helpers.both("box4k", 1)
    w, h = 53, 35
    bufs = render_with_aovs(g, sc, w, h, 2, 9)
    dn = kgr.Denoiser(w, h)
    cpu = [b.cpu().numpy().reshape(h, w, 4) for b in bufs]
    color = bufs[0].data_ptr()
    if own_result:
        dn.denoise(*[b.data_ptr() for b in bufs], iterations=3)
        torch.cuda.synchronize()
        cpu[0] = result_array(dn, w, h).reshape(h, w, 4).copy()
        color = dn.result()
    dn.denoise(color, *[b.data_ptr() for b in bufs[1:]], iterations=iterations)
    torch.cuda.synchronize()
    got = result_array(dn, w, h).reshape(h, w, 4)
    ref = post_ref.denoise(*cpu, 7, iterations=iterations)
    np.testing.assert_allclose(got, ref, rtol=1e-4, atol=1e-6)
    dn.close()
