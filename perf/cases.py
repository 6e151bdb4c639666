"""The work whose speed is measured: what a user of cnncrf has it do, through its public entry points.

Kinds of case (`kind`), each with the sizes this repository's configurations, tests and benchmark use:

  crf     one CRF solve on a cost volume and edge weights the caller owns (crf_solve)
  net     StereoNet.predict: the feature and pairwise nets and the fused cost volume of one pair
  stereo  one image pair through Stereo: matching, CRF and, where asked for, a refinement
  tv      the TV/Huber primal-dual iterations on fields the caller owns (tv_iterate)
  batch   many pairs through one StereoBatch, replayed as a graph
  train   one training step (Trainer.step) and its gradients
"""
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cnn-crf-stereo_gb300"))

import cnncrf  # noqa: E402
from cnncrf import api  # noqa: E402
from cnncrf.train import Trainer  # noqa: E402

# the CRF of the repository's own nets (truncated linear) and the command line's defaults (step)
LINEAR = dict(L1=0.5, L2=1.5, delta=3, shape="linear")
STEP = dict(L1=1.0, L2=12.0, delta=2, shape="step")


def listed():
    return [
        # a thumbnail-sized solve with the solver's default options: latency and launches
        dict(name="crf_256x192_d32", kind="crf", W=256, H=192, D=32, iters=4, **STEP),
        # a ragged size whose labels leave lanes partly empty
        dict(name="crf_619x271_d75", kind="crf", W=619, H=271, D=75, iters=8, **LINEAR),
        # the reference's 7-layer topology and its softmax unary on a KITTI-sized pair, exact FP32
        dict(name="net_fp32_kitti", kind="net", W=1242, H=375, D=128, precision="fp32", topology="ref", layers=7,
             unary="softmax"),
        # the all-3x3 net on a KITTI-sized pair on the tensor cores
        dict(name="net_bf16_kitti", kind="net", W=1242, H=375, D=128, precision="bf16", topology="all3x3", layers=7,
             unary="dot"),
        # the small grey configuration, whole pipeline in FP32
        dict(name="stereo_gray_256x192", kind="stereo", W=256, H=192, D=32, match="gray", precision="fp32", iters=5,
             refine="none", **LINEAR),
        # one KITTI-sized pair at a time: the latency of an online user
        dict(name="stereo_bf16_kitti", kind="stereo", W=1242, H=375, D=128, match="color", precision="bf16", iters=8,
             refine="none", **LINEAR),
        # the Middlebury-quarter-sized FP32 configuration with its TV refinement
        dict(name="stereo_tv_720x480", kind="stereo", W=720, H=480, D=96, match="color", precision="fp32", iters=5,
             refine="tv", **LINEAR),
        # the command line's defaults: census matching, image-gradient weights, QuadDirect
        dict(name="stereo_census_720x480", kind="stereo", W=720, H=480, D=128, match="census", precision="fp32",
             iters=4, refine="quad", **STEP),
        # the refinement alone on a 4K field, larger than the L2
        dict(name="tv_4096x2160", kind="tv", W=4096, H=2160, iters=10),
        # throughput: eight KITTI-sized pairs in two pipelined groups
        dict(name="batch_kitti8", kind="batch", shapes="1242x375x128", per=8, group=4, iters=8, **LINEAR),
        # throughput on mixed sizes and disparity ranges (four shapes, two pairs of each)
        dict(name="batch_uneven", kind="batch", shapes="480x320x64,720x480x96,1242x375x128,1440x960x192", per=2,
             group=2, iters=8, **LINEAR),
        # training: four crops, forward, loss-augmented CRF, adjoints, SGD
        dict(name="train_4x512x256", kind="train", W=512, H=256, D=128, n=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["crf", "crf", "net", "stereo", "stereo", "tv", "batch", "train"])
    crf = rng.choice([LINEAR, STEP, dict(L1=0.7, L2=2.0, delta=1, shape="step"),
                      dict(L1=0.4, L2=2.5, delta=4, shape="linear")])
    W = _log(rng, 96, 1242)
    H = _log(rng, 64, 480)
    D = rng.choice([_log(rng, 8, 256), 32, 64, 96, 128, 192])
    while W * H * D > 1242 * 375 * 128:
        D = max(8, D // 2)
    if kind == "crf":
        return dict(kind=kind, W=W, H=H, D=D, iters=rng.randint(2, 9), **crf)
    if kind == "net":
        return dict(kind=kind, W=W, H=H, D=min(D, W // 2), precision=rng.choice(["fp32", "bf16"]),
                    topology=rng.choice(["ref", "all3x3"]), layers=rng.choice([3, 5, 7]),
                    unary=rng.choice(["softmax", "dot"]))
    if kind == "stereo":
        match = rng.choice(["gray", "color", "color", "census"])
        refine = rng.choice(["none", "quad"] if match == "census" else ["none", "tv"])
        precision = "fp32" if match != "color" or refine == "tv" else rng.choice(["fp32", "bf16"])
        if match == "census":
            W, H = min(W, 720), min(H, 480)
        return dict(kind=kind, W=W, H=H, D=min(D, W // 2), match=match, precision=precision,
                    iters=rng.randint(2, 8), refine=refine, **crf)
    if kind == "tv":
        return dict(kind=kind, W=_log(rng, 128, 4096), H=_log(rng, 96, 2160), iters=rng.randint(2, 20))
    if kind == "batch":
        shapes = {(W, H, min(D, W // 2))}
        if rng.random() < 0.5:
            shapes.add((_log(rng, 96, 800), _log(rng, 64, 400), rng.choice([32, 48, 64, 96])))
        labels = sum(w * h * d for w, h, d in shapes)
        per = max(1, min(rng.randint(2, 8), int(8 * 1242 * 375 * 128 / labels)))
        return dict(kind=kind, shapes=",".join("%dx%dx%d" % s for s in sorted(shapes)), per=per,
                    group=rng.choice([0, max(1, per // 2)]), iters=rng.randint(3, 8), **LINEAR)
    return dict(kind=kind, W=rng.randint(96, 512), H=rng.randint(64, 256), D=rng.choice([32, 64, 96, 128]),
                n=rng.randint(1, 4))


# ------------------------------------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 2654435761 % (1 << 62))


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda")


def _texture(g, n, H, W):
    """n RGB images of band-limited noise in [0, 1], (n, 3, H, W)."""
    t = 0.0
    for k, a in ((1, 0.25), (3, 0.35), (7, 0.4)):
        x = _rand(g, n, 3, H + k - 1, W + k - 1)
        t = t + a * k * F.avg_pool2d(x - 0.5, k, stride=1)
    return (t + 0.5).clamp(0.0, 1.0)


def _disparity(g, rng, n, H, W, D):
    """Ground planes with boxes in front, (n, H, W), in 0..D-1."""
    y = torch.linspace(0.0, 0.85 * (D - 1), H, device="cuda").view(1, H, 1)
    d = (y * (0.6 + 0.4 * _rand(g, n, 1, 1))).repeat(1, 1, W)
    for i in range(n):
        for k in range(12):
            w, h = rng.randint(max(2, W // 30), max(3, W // 5)), rng.randint(max(2, H // 12), max(3, H // 3))
            x0, y0 = rng.randint(0, max(1, W - w)), rng.randint(0, max(1, H - h))
            d[i, y0:y0 + h, x0:x0 + w] = float(rng.uniform(0.1, 0.95) * (D - 1)) if k % 3 else float(rng.randint(0, D))
    return d.clamp(0.0, D - 1.0)


def _scene(seed, n, H, W, D, gray=False):
    """n stereo pairs as RGBA in [0, 1], (n, H, W, 4) each, and the left disparities."""
    g, rng = _gen(seed), np.random.RandomState(seed % (1 << 31))
    right = _texture(g, n, H, W)
    if gray:
        right = right.mean(1, keepdim=True).repeat(1, 3, 1, 1)
    disp = _disparity(g, rng, n, H, W, D)
    x = torch.arange(W, device="cuda").view(1, 1, W) - disp.round().long()
    hidden = x < 0
    left = torch.gather(right, 3, x.clamp(0, W - 1).unsqueeze(1).expand(-1, 3, -1, -1))
    left = torch.where(hidden.unsqueeze(1), _texture(g, n, H, W), left)
    out = []
    for im in (left, right):
        im = im + 0.008 * torch.randn(im.shape, generator=g, device="cuda")
        if gray:
            im = im[:, :1].repeat(1, 3, 1, 1)
        a = torch.ones((n, H, W, 4), device="cuda")
        a[..., :3] = im.clamp(0.0, 1.0).permute(0, 2, 3, 1)
        out.append(a)
    return out[0], out[1], disp


def _cost(seed, W, H, D):
    """A cost volume as a matcher makes it (colour differences over the disparities, noise) and edge weights
    that fall with the image gradient."""
    left, right, _ = _scene(seed, 1, H, W, D)
    l, r = left[0, :, :, :3], right[0, :, :, :3]
    cost = torch.ones((H, W, D), device="cuda")
    for d in range(min(D, W)):
        cost[:, d:, d] = (l[:, d:] - r[:, :W - d]).abs().mean(2)
    cost += 0.05 * _rand(_gen(seed + 77), H, W, D)
    gray = l.mean(2)
    wx, wy = torch.zeros((H, W), device="cuda"), torch.zeros((H, W), device="cuda")
    wx[:, :-1] = 0.4 * torch.exp(-20.0 * (gray[:, 1:] - gray[:, :-1]).abs())
    wy[:-1] = 0.4 * torch.exp(-20.0 * (gray[1:] - gray[:-1]).abs())
    return cost, wx, wy


def _net_dims(c):
    """(kernel sizes per feature layer, padding)"""
    ks = [3] + [3 if c["topology"] == "all3x3" else 2] * (c["layers"] - 1)
    return ks, sum(k - 1 for k in ks) // 2


def _net_params(c, seed):
    """Filters and biases of the feature net and the pairwise net in the parameter file's order."""
    rng = np.random.RandomState((seed * 31 + 7) % (1 << 31))
    ks, _ = _net_dims(c)
    out, cin = [], 3

    def conv(co, ci, k):
        lim = math.sqrt(6.0 / (k * k * (ci + co)))
        return rng.uniform(-lim, lim, (co, ci, k, k)).astype(np.float32)

    for k in ks:
        out += [conv(100, cin, k), rng.uniform(-0.05, 0.05, 100).astype(np.float32)]
        cin = 100
    out += [conv(64, 3, 3), rng.uniform(-0.05, 0.05, 64).astype(np.float32)]
    out += [conv(64, 64, 3), rng.uniform(-0.05, 0.05, 64).astype(np.float32), conv(2, 64, 1)]
    return out


def _net_images(c, seed):
    _, pad = _net_dims(c)
    l, r, _ = _scene(seed, 1, c["H"] + 2 * pad, c["W"] + 2 * pad, c["D"])
    return l[0].contiguous(), r[0].contiguous()


def _tv_fields(c, seed):
    H, W = c["H"], c["W"]
    g = _gen(seed)
    _, _, disp = _scene(seed, 1, H, W, 128)
    u0 = disp[0].round()
    qf = torch.stack([2.0 * (_rand(g, H, W) - 0.5), 4.0 * _rand(g, H, W)], 2).contiguous()
    wx, wy = (0.02 + 0.5 * _rand(g, H, W) for _ in range(2))
    return u0, qf, wx, wy


def _shapes(c):
    return [tuple(int(v) for v in s.split("x")) for s in c["shapes"].split(",")]


def _rho(c):
    return cnncrf.RHO_LINEAR if c["shape"] == "linear" else cnncrf.RHO_STEP


def prepare(c, seed):
    kind = c["kind"]
    s = dict(c=c)
    if kind == "crf":
        s["cost"], s["wx"], s["wy"] = _cost(seed, c["W"], c["H"], c["D"])
    elif kind == "net":
        _, pad = _net_dims(c)
        net = api.StereoNet(c["layers"], 1, 3, c["H"] + 2 * pad, c["W"] + 2 * pad,
                            topology=cnncrf.TOPO_ALL3X3 if c["topology"] == "all3x3" else cnncrf.TOPO_REF,
                            unary=cnncrf.UNARY_ONE_MINUS_DOT if c["unary"] == "dot" else cnncrf.UNARY_NEG_SOFTMAX,
                            precision=cnncrf.BF16 if c["precision"] == "bf16" else cnncrf.FP32, with_pairwise=True)
        net.init_net(0.0, float(c["D"] - 1), 1.0)
        for i, p in enumerate(_net_params(c, seed)):
            net.set_param(i, p)
        s["net"], (s["left"], s["right"]) = net, _net_images(c, seed)
    elif kind == "stereo":
        st = api.Stereo(precision=cnncrf.BF16 if c["precision"] == "bf16" else cnncrf.FP32,
                        unary=cnncrf.UNARY_ONE_MINUS_DOT, topology=cnncrf.TOPO_ALL3X3, ref_depth_rounding=False,
                        crf_shape=_rho(c), huber_eps=0.01)
        st.initialize(c["W"], c["H"], 0.0, 1.0, float(c["D"] - 1))
        st.set_matching_function({"gray": cnncrf.MATCH_GRAYCNN_PAIRWISE, "color": cnncrf.MATCH_COLORCNN_PAIRWISE,
                                  "census": cnncrf._lib.MATCH_CENSUS}[c["match"]])
        if c["match"] == "census":
            st.set_filter_size(7)
        else:
            st.set_num_layers(7)
            st.set_xavier_seed(0)
        l, r, _ = _scene(seed, 1, c["H"], c["W"], c["D"], gray=c["match"] == "gray")
        s["st"], s["left"], s["right"] = st, l[0], r[0]
    elif kind == "tv":
        s["u0"], s["qf"], s["wx"], s["wy"] = _tv_fields(c, seed)
    elif kind == "batch":
        b = api.StereoBatch(crf_shape=_rho(c), graph=True, group_size=c["group"])
        s["pairs"] = []
        for j, (W, H, D) in enumerate(_shapes(c)):
            l, r, _ = _scene(seed * 8 + j, c["per"], H, W, D)
            for i in range(c["per"]):
                b.add_pair(W, H, 0.0, 1.0, float(D - 1))
                s["pairs"].append((l[i], r[i]))
        for i, (l, r) in enumerate(s["pairs"]):
            b.set_images(i, l, r)
        b.autotune(c["L1"], c["L2"], c["delta"], c["iters"])  # once per deployment: tiles and launch forms
        s["b"] = b
    else:
        t = Trainer(c["n"], c["W"], c["H"], disp_max=float(c["D"] - 1))
        t.init_xavier(0)
        s["left"], s["right"], disp = _scene(seed, c["n"], c["H"], c["W"], c["D"])
        s["gt"] = disp.round().clamp(0, c["D"] - 1).to(torch.int32)
        t.forward(s["left"], s["right"])
        t.autotune()  # once per deployment
        s["t"], s["np"] = t, t.num_params()
    return s


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "crf":
        labels, lb = api.crf_solve(s["cost"], s["wx"], s["wy"], c["L1"], c["L2"], c["delta"], c["iters"], _rho(c))
        return dict(labels=labels, bound=lb)
    if kind == "net":
        vol = s["net"].predict(s["left"], s["right"])
        return dict(volume=vol, pairwise=s["net"].pairwise_out)
    if kind == "stereo":
        st = s["st"]
        st.set_color_images(s["left"], s["right"])
        census = c["match"] == "census"
        st.compute_slack_propagation(c["L1"], c["L2"], c["delta"], c["iters"], 20.0 if census else 0.0,
                                     0.8 if census else 0.0, 0.4 if census else 1.0)
        out = dict(labels=st.labels_device().clone(), bound=st.lower_bound())
        if c["refine"] == "tv":
            st.fuse_thuber_quad_fit(1.0, 1.5, 4, 1)
        elif c["refine"] == "quad":
            st.fuse_quad_fit_direct()
        out["disparity"] = st.output_device().clone()
        return out
    if kind == "tv":
        u, u_, p, q = api.tv_iterate(s["u0"], s["u0"], s["qf"], s["wx"], s["wy"], 1.5, 0.01, 1.0, c["iters"])
        return dict(u=u, u_=u_, p=p, q=q)
    if kind == "batch":
        b = s["b"]
        for i, (l, r) in enumerate(s["pairs"]):
            b.set_images(i, l, r)
        b.run(c["L1"], c["L2"], c["delta"], c["iters"])
        n = len(s["pairs"])
        return dict(labels=[b.labels_device(i).clone() for i in range(n)],
                    disparity=[b.output_device(i).clone() for i in range(n)])
    t = s["t"]
    loss = t.step(s["left"], s["right"], s["gt"], lr=1e-3, momentum=0.9)
    return dict(loss=loss, grads=[t.grad_tensor(i) for i in range(s["np"])])


# ------------------------------------------------------------------------------------------------ work

def _crf_work(W, H, D, c):
    # the volume and the weights in, the labels out; per label and pass a forward and a backward message (delta
    # offsets each: one add, two minima) and the slack hand-over
    n = W * H
    return 4 * (n * D + 3 * n), n * D * 2 * c["iters"] * (6 * c["delta"] + 14)


def _net_work(W, H, D, layers=7, k=3, ic=3, pairwise=True):
    pad = (2 + (layers - 1) * (k - 1)) // 2
    h, w, fl, cin = H + 2 * pad, W + 2 * pad, 0, ic
    byt = 2 * 16 * h * w + 4 * W * H * (D + 2)
    for i in range(layers):
        kk = 3 if i == 0 else k
        h, w = h - (kk - 1), w - (kk - 1)
        fl += 2 * 2 * h * w * 100 * kk * kk * cin
        cin = 100
    fl += 2 * W * H * 100 * D
    if pairwise:
        fl += 2 * W * H * (64 * 9 * min(ic, 3) + 64 * 9 * 64 + 2 * 64)
    return byt, fl


def work(c):
    kind = c["kind"]
    if kind == "crf":
        b, f = _crf_work(c["W"], c["H"], c["D"], c)
    elif kind == "net":
        b, f = _net_work(c["W"], c["H"], c["D"], c["layers"], 3 if c["topology"] == "all3x3" else 2)
    elif kind == "stereo":
        W, H, D = c["W"], c["H"], c["D"]
        _, f = _crf_work(W, H, D, c)
        b = 2 * 16 * W * H + 4 * W * H * 2
        if c["match"] == "census":
            f += W * H * D * (224 // 32) * 2  # 224 bits a pixel and disparity, compared and counted 32 at a time
        else:
            ic = 1 if c["match"] == "gray" else 3
            f += _net_work(W, H, D, ic=ic)[1]
            if c["refine"] == "tv":
                f += _net_work(W, H, 3, ic=ic)[1] // 2 + 4 * 60 * W * H
    elif kind == "tv":
        n = c["W"] * c["H"]
        b, f = n * 4 * (1 + 1 + 2 + 2 + 2 + 2 + 2), n * c["iters"] * 60
    elif kind == "batch":
        b = f = 0
        for W, H, D in _shapes(c):
            b += c["per"] * (2 * 16 * W * H + 4 * W * H * 2)
            f += c["per"] * (_crf_work(W, H, D, c)[1] + _net_work(W, H, D)[1])
    else:
        W, H, D, n = c["W"], c["H"], c["D"], c["n"]
        f = n * (3 * _net_work(W, H, D)[1] + _crf_work(W, H, D, dict(iters=8, delta=3))[1])
        b = n * (2 * 16 * W * H + 4 * W * H) + 12 * 4 * 600_000
    return dict(bytes=b, flops=f)


# ------------------------------------------------------------------------------------------------ 64 bits

def _conv64(x, w, b, act):
    """A valid convolution (kernel flipped) in row bands, x (1, C, H, W) in 64 bits."""
    w = torch.from_numpy(w).cuda().double().flip(2, 3)
    b = None if b is None else torch.from_numpy(b).cuda().double()
    k, H = w.shape[2], x.shape[2] - w.shape[2] + 1
    out = torch.empty((1, w.shape[0], H, x.shape[3] - k + 1), device="cuda", dtype=torch.float64)
    for y in range(0, H, 64):
        e = min(H, y + 64)
        cols = F.unfold(x[:, :, y:e + k - 1], k)[0]
        t = w.reshape(w.shape[0], -1) @ cols
        if b is not None:
            t += b.view(-1, 1)
        out[0, :, y:e] = act(t).view(w.shape[0], e - y, -1)
    return out


def _net_exact(c, seed):
    ks, pad = _net_dims(c)
    par = _net_params(c, seed)
    feats = []
    norm = []
    for im in _net_images(c, seed):
        x = im[..., :3].double().permute(2, 0, 1)
        x = x - x.mean((1, 2), keepdim=True)
        x = (x / x.square().mean((1, 2), keepdim=True).sqrt())[None]
        norm.append(x)
        for l in range(len(ks)):
            x = _conv64(x, par[2 * l], par[2 * l + 1], torch.tanh)
        if c["unary"] == "dot":
            x = x / x.square().sum(1, keepdim=True).sqrt()
        feats.append(x[0])
    fl, fr = feats
    H, W, D = c["H"], c["W"], c["D"]
    vol = torch.zeros((H, W, D), device="cuda", dtype=torch.float64)
    for d in range(min(D, W)):
        vol[:, d:, d] = (fl[:, :, d:] * fr[:, :, :W - d]).sum(0)
    vol = 1.0 - vol if c["unary"] == "dot" else -torch.softmax(vol, 2)
    q, m = 2 * len(ks), pad - 2
    x = norm[0][:, :, m:H + 2 * pad - m, m:W + 2 * pad - m]
    x = _conv64(x, par[q], par[q + 1], torch.tanh)
    x = _conv64(x, par[q + 2], par[q + 3], torch.tanh)
    return dict(volume=vol, pairwise=_conv64(x, par[q + 4], None, torch.abs)[0])


def _tv_exact(c, seed):
    u0, qf, wx, wy = (t.double() for t in _tv_fields(c, seed))
    a, b = qf[..., 0], qf[..., 1]
    tau = sigma = 1.0 / math.sqrt(8.0)
    C, eps = 1.5, 0.01
    u = u0.clone()
    px, py, qx, qy = (torch.zeros_like(u) for _ in range(4))

    def back(v, dim):  # v - its predecessor, the first one its own
        return v - torch.cat([v.narrow(dim, 0, 1), v.narrow(dim, 0, v.shape[dim] - 1)], dim)

    def fwd(v, dim):
        return torch.cat([v.narrow(dim, 1, v.shape[dim] - 1), v.narrow(dim, v.shape[dim] - 1, 1)], dim) - v

    for _ in range(c["iters"]):
        v = u + tau * (back(px - qx, 1) + back(py - qy, 0))
        un = ((v - tau * (a - b * u0)) / (1 + tau * b)).clamp(min=u0 - 0.5, max=u0 + 0.5)
        ub, u = 2 * un - u, un
        dx, dy = fwd(ub, 1), fwd(ub, 0)
        px = torch.maximum(-wx, torch.minimum(wx, (px + sigma * dx) / (1 + sigma * eps)))
        py = torch.maximum(-wy, torch.minimum(wy, (py + sigma * dy) / (1 + sigma * eps)))

        def shrink(v, w):
            return torch.maximum(-w, torch.minimum(w, torch.sign(v) * (v.abs() - sigma * C).clamp(min=0)))

        qx, qy = shrink(qx + sigma * dx, wx), shrink(qy + sigma * dy, wy)
    return dict(u=u, u_=ub, p=torch.stack([px, py], 2), q=torch.stack([qx, qy], 2))


def _crf_exact(c, seed):
    """The bound of the solver's dual decomposition, in 64 bits (the labels are whole numbers)."""
    cost, wx, wy = (t.double() for t in _cost(seed, c["W"], c["H"], c["D"]))
    D, delta = c["D"], c["delta"]
    rho = [min(c["L1"] * (t if c["shape"] == "linear" else 1), c["L2"]) for t in range(delta + 1)]

    def minconv(v, w):  # v (chains, D), w (chains, 1): the message without its minimum, and that minimum
        g = v.amin(1, keepdim=True)
        o = torch.minimum(v, g + w * c["L2"])
        for t in range(1, min(delta, D - 1) + 1):
            s = v + w * rho[t]
            o[:, t:] = torch.minimum(o[:, t:], s[:, :-t])
            o[:, :-t] = torch.minimum(o[:, :-t], s[:, t:])
        return o - g, g

    def sweep(un, w):  # un (n, chains, D): (reduced unary, bound), un is changed
        n = un.shape[0]
        fwd = torch.zeros_like(un)
        total = 0.0
        for i in range(n):
            v = fwd[i] + un[i]
            if i < n - 1:
                fwd[i + 1], g = minconv(v, w[i])
            else:
                g = v.amin(1, keepdim=True)
            total = total + g
        back = torch.zeros_like(un[0])
        for i in range(n - 1, -1, -1):
            m = fwd[i] + un[i] + back
            un[i] -= 0.5 * (m - m.amin(1, keepdim=True))
            if i > 0:
                back, _ = minconv(un[i] + back, w[i - 1])
        return un, float(total.sum())

    phi = torch.zeros_like(cost)
    for _ in range(c["iters"]):
        un, h = sweep((cost - phi).transpose(0, 1).contiguous(), wx.t().unsqueeze(2).contiguous())
        phi = cost - un.transpose(0, 1)
        phi, v = sweep(phi.contiguous(), wy.unsqueeze(2))
    return dict(labels=None, bound=h + v)


def exact(c, seed):
    if c["kind"] == "net":
        return _net_exact(c, seed)
    if c["kind"] == "tv":
        return _tv_exact(c, seed)
    if c["kind"] == "crf":
        return _crf_exact(c, seed)
    return None
