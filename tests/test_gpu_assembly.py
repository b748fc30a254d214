"""Laplacian assembly on the GPU: the reference-arithmetic kernel is
bit-identical to the reference's hostLevinLaplacian (golden fixtures), the
FP64 kernel matches the FP64 oracle to one rounding."""
import numpy as np
import pytest

from conftest import golden_cases, load_golden
from gpu_util import bands25_f32, oracle_problem, torch_cuda
from gpumatting_b200.synth import make_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", golden_cases())
def test_reference_arithmetic_bit_exact(case):
    torch = torch_cuda()
    from gpumatting_b200 import api

    g = load_golden(case)
    im = torch.from_numpy(g["im4"]).cuda()
    sc = torch.from_numpy(g["scribbles"]).cuda()
    a, b = api.levin_bands25(im, sc, eps=float(g["lam"]), gamma_value=1.0, arithmetic="reference")
    assert np.array_equal(a.cpu().numpy().view(np.uint32), g["a"].view(np.uint32))
    assert np.array_equal(b.cpu().numpy().view(np.uint32), g["b"].view(np.uint32))


@pytest.mark.parametrize("case", ["s37x29", "data05", "s3x3"])
def test_hostLevinLaplacian_dropin(case):
    torch_cuda()
    from gpumatting_b200 import api

    g = load_golden(case)
    H, W = g["scribbles"].shape
    a = np.zeros((25, W * H), np.float32)
    b = np.zeros(W * H, np.float32)
    api.hostLevinLaplacian(a, b, float(g["lam"]), g["im4"], g["scribbles"], W, H)
    assert np.array_equal(a.view(np.uint32), g["a"].view(np.uint32))
    assert np.array_equal(b, g["b"])


def _row_diag(w, g, W, H):
    """gamma + sum over the 24 stencil neighbours of the stored affinities."""
    d = g.reshape(H, W).copy()
    wp = w.reshape(12, H, W)
    for k in range(1, 13):
        dv = (k + 2) // 5
        du = k - 5 * dv
        d += wp[k - 1]
        # lower neighbour (u - du, v - dv) holds w_k for the pair
        sh = np.zeros((H, W))
        v0, u0 = dv, max(0, du)
        u1 = min(W, W + du)
        sh[v0:, u0:u1] = wp[k - 1][: H - dv, u0 - du:u1 - du]
        d += sh
    return d.ravel()


def _ulp_close(x, ref, dtype, ulps=1):
    r = ref.astype(dtype).astype(np.float64)
    x = x.astype(np.float64)
    sp = np.spacing(np.abs(r).astype(dtype)).astype(np.float64)
    return np.all(np.abs(x - r) <= ulps * sp + 1e-30)


@pytest.mark.parametrize("W,H,prec,fmt", [(64, 48, "fp16", "rgb8"), (37, 29, "bf16", "rgb8"),
                                          (101, 7, "fp32", "rgba"), (5, 40, "fp16", "rgba")])
def test_fp64_assembly_matches_oracle(orc, W, H, prec, fmt):
    torch = torch_cuda()
    from gpumatting_b200 import api

    p, w, g, b = oracle_problem(orc, W, H, seed=9)
    img = torch.from_numpy(p.image).cuda() if fmt == "rgb8" else torch.from_numpy(
        np.concatenate([p.image.astype(np.float64) / 255.0, np.ones((H, W, 1))], axis=2).astype(np.float32)).cuda()
    if fmt == "rgba":  # the float image is the reference (rounded) one
        w = orc.levin_sym64(img.cpu().numpy()[..., :3].astype(np.float64), p.eps)
    sc = torch.from_numpy(p.scribbles).cuda()
    st = api.LevinStore(W, H, prec)
    Lm = api.DeviceBandedMatrix(torch.zeros((25, W * H), device="cuda"), torch.tensor(orc.levin_offsets(W)).cuda(),
                                W * H)
    b25 = torch.zeros(W * H, device="cuda")
    st.assemble(img, sc, eps=p.eps, gamma_value=100.0, bands25=Lm, b25=b25)
    torch.cuda.synchronize()
    w32 = st.planes("w32")[:, :, :W].reshape(12, -1).cpu().numpy()
    assert _ulp_close(w32, w, np.float32)
    wl = st.planes("w")[:, :, :W].reshape(12, -1).float().cpu().numpy()
    dt = {"fp16": np.float16, "fp32": np.float32}.get(prec)
    if dt is not None:
        assert _ulp_close(wl, w, dt)
    else:  # bf16: compare against the FP32 rounding at bf16 spacing
        assert np.all(np.abs(wl - w) <= np.abs(w) * 2.0 ** -8 + 1e-30)
    assert np.array_equal(st.planes("gamma")[:, :W].cpu().numpy().ravel(), g.astype(np.float32))
    # diagonal planes: gamma + row sum of exactly the rounded weights
    for dname, wp in (("d32", w32), ("d", wl)):
        exp = _row_diag(wp.astype(np.float64), g, W, H).astype(np.float32)
        got = st.planes(dname)[:, :W].cpu().numpy().ravel()
        assert np.all(np.abs(got.astype(np.float64) - exp) <= np.spacing(np.abs(exp)) + 1e-30), dname
    assert np.array_equal(st.planes("b")[:, :W].cpu().numpy().ravel(), b.astype(np.float32))
    a25 = Lm.a.cpu().numpy()
    ref = bands25_f32(orc, w, g, W, H)
    assert np.abs(a25 - ref).max() <= 2e-6 * np.abs(ref).max()
    assert np.array_equal(b25.cpu().numpy(), b.astype(np.float32))


def test_assembly_per_pixel_gamma_maps(orc):
    torch = torch_cuda()
    from gpumatting_b200 import api

    W, H = 33, 21
    p = make_problem(W, H, 12)
    rng = np.random.default_rng(3)
    gam = rng.uniform(0, 50, size=(H, W)).astype(np.float32)
    s = rng.uniform(0, 1, size=(H, W)).astype(np.float32)
    st = api.LevinStore(W, H, "fp16")
    st.assemble(torch.from_numpy(p.image).cuda(), None, eps=1e-4, gamma_map=torch.from_numpy(gam).cuda(),
                s_map=torch.from_numpy(s).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(st.planes("gamma")[:, :W].cpu().numpy(), gam)
    assert np.array_equal(st.planes("b")[:, :W].cpu().numpy(), gam * s)


@pytest.mark.parametrize("W,H,prec,fmt", [(1, 9, "fp16", "rgb8"), (9, 2, "fp32", "rgba"), (3, 3, "bf16", "rgb8"),
                                          (125, 5, "fp16", "rgba"), (126, 41, "fp16", "rgb8"), (127, 4, "fp32", "rgb8"),
                                          (128, 3, "bf16", "rgba"), (253, 37, "fp32", "rgba"),
                                          (1241, 130, "fp16", "rgb8")])
def test_fp64_assembly_at_strip_and_run_edges(orc, W, H, prec, fmt):
    """Widths around the kernel's 126-column strips, runs of 2 rows up to
    several, images without a window.  Couplings within one FP32 ulp of the
    oracle's plus what FP64 rounding allows either side: an error of 2^-53 in
    81 Sigma (entries up to 81) over its smallest eigenvalue, at least 9 eps.
    The diagonals are the FP64 sums of the stored weights, rounded once;
    25-band output included."""
    torch = torch_cuda()
    from gpumatting_b200 import api

    rng = np.random.default_rng(W * 1000 + H)
    base = rng.integers(0, 256, size=(H // 4 + 2, W // 4 + 2, 3)).repeat(4, 0).repeat(4, 1)[:H, :W]
    image = np.clip(base + rng.integers(-6, 7, size=(H, W, 3)), 0, 255).astype(np.uint8)
    scr = rng.choice(np.array([0, 128, 255], np.uint8), size=(H, W), p=[0.1, 0.8, 0.1])
    img = torch.from_numpy(image).cuda()
    ref_in = image.astype(np.float64) / 255.0
    if fmt == "rgba":
        img = torch.from_numpy(np.concatenate([ref_in, np.ones((H, W, 1))], axis=2).astype(np.float32)).cuda()
        ref_in = img.cpu().numpy()[..., :3].astype(np.float64)
    w = orc.levin_sym64(np.ascontiguousarray(ref_in), 1e-5).reshape(12, H, W)
    st = api.LevinStore(W, H, prec)
    Lm = api.DeviceBandedMatrix(torch.zeros((25, W * H), device="cuda"), torch.tensor(orc.levin_offsets(W)).cuda(),
                                W * H)
    st.assemble(img, torch.from_numpy(scr).cuda(), eps=1e-5, gamma_value=100.0, bands25=Lm)
    w32 = st.planes("w32")[:, :, :W].cpu().numpy()
    sp = np.spacing(np.abs(w).astype(np.float32)).astype(np.float64)
    assert np.all(np.abs(w32 - w) <= sp + 81 * 2.0 ** -53 / (9 * 1e-5))
    wl = st.planes("w")[:, :, :W].float().cpu().numpy()
    assert np.all(np.abs(wl - w) <= np.abs(w) * {"fp16": 2.0 ** -10, "bf16": 2.0 ** -7, "fp32": 2.0 ** -22}[prec] + 1e-7)
    g = np.where(scr != 128, 100.0, 0.0)
    for name, wp in (("d32", w32), ("d", wl)):
        s = _row_diag(wp.astype(np.float64), g.ravel(), W, H)
        got = st.planes(name)[:, :W].cpu().numpy().ravel()
        assert np.all(np.abs(got - s) <= 0.5 * np.spacing(np.abs(s).astype(np.float32)) * (1 + 1e-6) + 1e-30), name
    a = Lm.a.cpu().numpy().reshape(25, H, W)
    for k in range(1, 13):
        dv = (k + 2) // 5
        du = k - 5 * dv
        assert np.array_equal(a[12 + k], -w32[k - 1])
        u0, u1 = max(0, du), min(W, W + du)
        if u1 > u0 and H > dv:
            assert np.array_equal(a[12 - k][dv:, u0:u1], -w32[k - 1][: H - dv, u0 - du:u1 - du])
    a2, b2 = api.levin_bands25(img, torch.from_numpy(scr).cuda(), eps=1e-5, gamma_value=100.0, arithmetic="fp64")
    assert np.array_equal(a2.cpu().numpy().view(np.uint32), Lm.a.cpu().numpy().view(np.uint32))
    assert np.array_equal(b2.cpu().numpy().reshape(H, W), np.where(scr == 255, 100.0, 0.0).astype(np.float32))


@pytest.mark.parametrize("W,H,prec", [(140, 37, "fp16"), (140, 37, "fp32"), (126, 5, "bf16"), (9, 3, "fp32")])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_nonfinite_colours_stay_in_their_windows(orc, W, H, prec, bad):
    """A non-finite colour of a float image reaches the couplings of the 3x3
    windows that hold it and nothing else: couplings out of the image are zero
    whatever its border holds.  The couplings of the others are the bits of the
    image without it."""
    torch = torch_cuda()
    from gpumatting_b200 import api

    rng = np.random.default_rng(W)
    base = np.ones((H, W, 4), np.float32)
    base[..., :3] = rng.random((H, W, 3))

    def planes(image):
        st = api.LevinStore(W, H, prec).assemble(torch.from_numpy(image).cuda(), eps=1e-5)
        return [st.planes(n)[..., :W].float().cpu().numpy() for n in ("w32", "w", "d32", "d")]

    clean = planes(base)
    for x, y in [(0, 0), (W - 1, 0), (0, H - 1), (W - 1, H - 1), (1, H // 2), (W - 2, 1), (W // 2, H - 2), (W - 1, H // 2)]:
        image = base.copy()
        image[y, x, 1] = bad
        fin = np.isfinite(orc.levin_sym64(np.ascontiguousarray(image[..., :3].astype(np.float64)), 1e-5).reshape(12, H, W))
        rows = _row_diag((~fin).astype(np.float64), np.zeros(W * H), W, H).reshape(H, W) == 0.0
        for name, got, ref in zip(("w32", "w", "d32", "d"), planes(image), clean):
            ok = np.isfinite(got)
            assert np.array_equal(ok, fin if name[0] == "w" else rows), (name, x, y)
            assert np.array_equal(got[ok], ref[ok]), (name, x, y)


def _limit_couplings(image):
    """Couplings (12, H, W) of whole-number colours (H, W, 3) for eps -> 0, FP64:
    (1 + D_i^T N^+ D_j) / 9 per 3x3 window, N = 9 sum(x x^T) - S S^T, D = 9 x - S.  And the
    smallest nonzero eigenvalue of any N."""
    x = image.astype(np.float64)
    H, W, _ = x.shape
    win = np.stack([x[j:H - 2 + j, i:W - 2 + i] for j in range(3) for i in range(3)], axis=2)  # (h, w, 9, 3)
    S = win.sum(2)
    D = 9.0 * win - S[:, :, None, :]
    N = 9.0 * np.einsum("hwqa,hwqb->hwab", win, win) - S[..., :, None] * S[..., None, :]  # whole numbers, exact
    lam, vec = np.linalg.eigh(N)
    real = lam > 1e-9 * np.maximum(lam[..., -1:], 1.0)
    inv = np.where(real, 1.0 / np.where(real, lam, 1.0), 0.0)
    y = np.einsum("hwqa,hwab->hwqb", D, vec)
    t = (1.0 + np.einsum("hwpb,hwb,hwqb->hwpq", y, inv, y)) / 9.0
    w = np.zeros((12, H, W))
    for p in range(9):
        for q in range(9):
            k = (q % 3 - p % 3) + 5 * (q // 3 - p // 3)
            if k > 0:
                w[k - 1, p // 3:p // 3 + H - 2, p % 3:p % 3 + W - 2] += t[:, :, p, q]
    return w, lam[real].min()


@pytest.mark.parametrize("eps", [0.0, 1e-300, 1e-20])
@pytest.mark.parametrize("prec,fmt", [("fp32", "rgb8"), ("fp16", "rgb8"), ("fp32", "rgba"), ("bf16", "rgba")])
def test_assembly_of_singular_windows(prec, fmt, eps):
    """eps = 0 and next to nothing on flat, white, black, grey, two-channel and
    one-line patches (windows of rank 0, 1 and 2) beside noise: the limit of small
    eps.  An addition of e to N moves the nine terms of a window by at most 8 e / lam
    of the smallest nonzero eigenvalue lam; e is 2^-26 for bytes, and for floats
    x = byte / 255 it is 9 2^-47 sum(x x) <= 243 2^-47, with three times that for the
    rounding of the 24-bit colours' sums; FP32's rounding of the sum comes on top."""
    torch = torch_cuda()
    from gpumatting_b200 import api

    W, H = 150, 40
    rng = np.random.default_rng(5)
    image = rng.integers(0, 256, size=(H, W, 3))
    image[:, 20:32] = (77, 200, 30)
    image[:, 32:44] = 255
    image[:, 44:56] = 0
    image[:, 60:76] = rng.integers(0, 256, size=(H, 16, 1))
    image[:, 80:96, 2] = image[:, 80:96, 1]
    image[:, 96:110, 0] = 9
    image[:, 112:128] = (np.arange(16) * 3)[None, :, None]
    image[:, 130:, 0] = 40
    image[:, 130:, 1] = 41
    want, lam = _limit_couplings(image)
    img = torch.from_numpy(image.astype(np.uint8)).cuda()
    e = 2.0 ** -26
    if fmt == "rgba":
        f = np.ones((H, W, 4), np.float32)
        # bytes / 256: exact, so that windows have the ranks of the bytes' own
        f[..., :3] = image / 256.0
        img = torch.from_numpy(f).cuda()
        e, lam = 3 * 243 * 2.0 ** -47, lam / 256.0 ** 2
    st = api.LevinStore(W, H, prec).assemble(img, eps=eps)
    got = st.planes("w32")[:, :, :W].double().cpu().numpy()
    tol = np.spacing(np.abs(want).astype(np.float32)).astype(np.float64) + 9 * 8 * e / lam
    assert np.all(np.abs(got - want) <= tol), np.nanmax(np.abs(got - want) / tol)
    for n in ("w", "d", "d32"):
        assert torch.isfinite(st.planes(n)[..., :W].float()).all()
