"""The work that users of this framework have it do on one GPU, as cases that can be timed and compared.

Three kinds, all through the public entry points:
  "attention"  forward + backward through the autograd class that `create_attention_class()` returns, or the forward
               alone through `_attn_forward`, on q [B, Hq, Sq, 128] and k, v [B, Hkv, Skv, 128]. With "padded" the batch
               entries have fewer and fewer valid keys (`kv_valid_len`).
  "bias"       the same call with a `bias_func`: a text token sees only the images that stand before it in its text.
  "layer"      the Llama-3.2-Vision cross-attention layer behind `patch_cross_attention_forward`: q/k/v/o projections,
               per-head RMSNorm on q and k, K/V projected again in backward; gradients of the text states and weights.
Inputs are N(0, 0.5^2) for q, k, v, N(0, 1) for upstream gradients and states, N(0, 0.02^2) for weights.
"""
import math

import torch

import lv_xattn_b200 as lvx

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SCALE = 1.0 / math.sqrt(128.0)
IMAGE = 6404            # visual tokens of one image: 4 tiles of 1,601


def _attention(name, dtype, B, Hq, Hkv, Sq, Skv, backward, padded=False, kind="attention"):
    c = dict(kind=kind, dtype=dtype, B=B, Hq=Hq, Hkv=Hkv, Sq=Sq, Skv=Skv, backward=backward, padded=padded)
    return dict(c, name=name) if name else c


def _layer(name, hidden, Hq, Hkv, Sq, Skv):
    c = dict(kind="layer", dtype="bf16", hidden=hidden, Hq=Hq, Hkv=Hkv, Sq=Sq, Skv=Skv)
    return dict(c, name=name) if name else c


def listed():
    return [
        # generation: one new text token attends to a single image, the smallest call there is
        _attention("token_one_image", "bf16", 1, 32, 8, 1, IMAGE, False),
        # generation over a long video: one new text token, 64 frames of 4 tiles (409,856 visual tokens)
        _attention("token_long_video", "bf16", 1, 32, 8, 1, 64 * IMAGE, False),
        # scoring or prefill of two prompts of odd length over four images, the second with fewer visual tokens
        _attention("prompt_padded", "bf16", 2, 32, 8, 333, 4 * IMAGE, False, padded=True),
        # the shape of the reference's own benchmark script: 16 heads without grouping, 1,024 x 4,096, fp16
        _attention("train_fp16_mha", "fp16", 1, 16, 16, 1024, 4096, True),
        # fine-tuning on short texts: four samples of 77 tokens, one image tile each (an odd 1,601 tokens), padded
        _attention("train_short_padded", "bf16", 4, 32, 8, 77, 1601, True, padded=True),
        # the headline layer, 2,048 text x 131,072 visual tokens, on a single GPU
        _attention("train_headline", "bf16", 1, 32, 8, 2048, 131072, True),
        # the same text against the 16,384 visual tokens that each of eight GPUs holds of it
        _attention("train_rank_of_eight", "bf16", 1, 32, 8, 2048, 16384, True),
        # long-visual training, 256 text tokens, B = 2 with key padding: one of four GPUs' 262,144 of 1,048,576 keys
        _attention("train_long_visual", "bf16", 2, 32, 8, 256, 262144, True, padded=True),
        # the fp32 configuration, used for checking a model against its full-precision self
        _attention("train_fp32", "fp32", 1, 32, 8, 512, 8192, True),
        # interleaved text and images: the bias_func protocol with a text-to-image mask, one 4-tile image's worth of keys
        _attention("train_image_mask", "bf16", 1, 32, 8, 512, IMAGE, True, kind="bias"),
        # the Llama-3.2-11B-Vision layer on one image with a short prompt
        _layer("layer_one_image", 4096, 32, 8, 64, IMAGE),
        # the same layer on a long video: 1,024 text tokens, one of eight GPUs' share of 409,856 visual tokens
        _layer("layer_long_video", 4096, 32, 8, 1024, 51232),
    ]


def _log_int(rng, lo, hi):
    """An integer from lo to hi, spread over its logarithm; most of what comes out is neither even nor a power of two."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: text of 1 to 2,048 tokens, 1,000 to 409,856 visual tokens, every data type and option above."""
    what = rng.choices(["train", "forward", "fp32", "bias", "layer"], [6, 4, 2, 2, 3])[0]
    if what == "layer":
        hidden, Hq, Hkv = rng.choice([(512, 4, 2), (4096, 32, 8)])
        return _layer(None, hidden, Hq, Hkv, _log_int(rng, 16, 1024), _log_int(rng, 1601, 51232))
    Hq, Hkv = rng.choice([(32, 8), (32, 8), (16, 16), (8, 2), (4, 4)])
    B = rng.choice([1, 1, 2, 3, 4])
    # a drawn case has at most the headline's products, and an fp32 or biased one at most twice the fp32 case's
    most = 2 * 32 * 512 * 8192 if what in ("fp32", "bias") else 32 * 2048 * 131072
    Sq = _log_int(rng, 1 if what == "forward" else 16, 1024 if what in ("fp32", "bias") else 2048)
    Skv = _log_int(rng, 1000, max(1000, min(409856 if what in ("train", "forward") else 32768, most // (B * Hq * Sq))))
    dtype = "fp32" if what == "fp32" else rng.choice(["bf16", "bf16", "fp16"])
    return _attention(None, dtype, B, Hq, Hkv, Sq, Skv, what != "forward", padded=B > 1 and rng.random() < 0.6,
                      kind="bias" if what == "bias" else "attention")


def _valid(case):
    """Valid keys of each batch entry: all, then ever fewer, down to about half."""
    return [case["Skv"] - b * (case["Skv"] // (2 * case["B"])) for b in range(case["B"])]


class _Norm(torch.nn.Module):
    """RMSNorm over the head dimension, computed in fp32 as the Llama modules do."""

    def __init__(self, device):
        super().__init__()
        self.weight = torch.nn.Parameter(torch.ones(128, device=device, dtype=torch.bfloat16))
        self.variance_epsilon = 1e-5

    def forward(self, x):
        h = x.float()
        h = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + self.variance_epsilon)
        return self.weight * h.to(x.dtype)


class _CrossAttention(torch.nn.Module):
    """The members of the Llama-3.2-Vision text cross-attention module that the hook uses."""
    forward = lvx.patch_cross_attention_forward("lv_xattn")

    def __init__(self, hidden, Hq, Hkv, g, device):
        super().__init__()
        self.num_heads, self.num_key_value_heads, self.head_dim = Hq, Hkv, 128

        def linear(n_in, n_out):
            m = torch.nn.Linear(n_in, n_out, bias=False, device="meta", dtype=torch.bfloat16)
            w = torch.empty(n_out, n_in, device=device, dtype=torch.bfloat16).normal_(0, 0.02, generator=g)
            m.weight = torch.nn.Parameter(w)
            return m

        self.q_proj, self.k_proj = linear(hidden, Hq * 128), linear(hidden, Hkv * 128)
        self.v_proj, self.o_proj = linear(hidden, Hkv * 128), linear(Hq * 128, hidden)
        self.q_norm, self.k_norm = _Norm(device), _Norm(device)


def _image_bias(image_of_key, images_before):
    """0 where the key's image stands before the text token, -inf elsewhere: [1, 1, Sq, Skv]."""
    seen = image_of_key[None, :] < images_before[:, None]
    return torch.zeros(seen.shape, device=seen.device).masked_fill_(~seen, float("-inf"))[None, None]


def prepare(case, seed):
    device = torch.device("cuda")
    g = torch.Generator(device=device).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    Sq, Skv = case["Sq"], case["Skv"]

    def normal(std, *shape):
        return torch.empty(*shape, device=device, dtype=dtype).normal_(0, std, generator=g)

    if case["kind"] == "layer":
        hidden = case["hidden"]
        return dict(kind="layer", module=_CrossAttention(hidden, case["Hq"], case["Hkv"], g, device),
                    x=normal(1.0, 1, Sq, hidden).requires_grad_(), states=normal(1.0, 1, Skv, hidden),
                    grad=normal(1.0, 1, Sq, hidden))
    B, Hq, Hkv = case["B"], case["Hq"], case["Hkv"]
    train = case["backward"]
    s = dict(kind=case["kind"], valid=_valid(case) if case["padded"] else None)
    s["q"] = normal(0.5, B, Hq, Sq, 128).requires_grad_(train)
    s["k"] = normal(0.5, B, Hkv, Skv, 128).requires_grad_(train)
    s["v"] = normal(0.5, B, Hkv, Skv, 128).requires_grad_(train)
    if train:
        s["attention"] = lvx.create_attention_class("lv_xattn").apply
        s["grad"] = normal(1.0, B, Hq, Sq, 128)
    if case["kind"] == "bias":
        # four images in the keys; the text tokens see one image at the start and all four at the end
        s["image_of_key"] = torch.arange(Skv, device=device) * 4 // Skv
        s["images_before"] = torch.arange(Sq, device=device) * 4 // Sq + 1
    return s


def run(s):
    if s["kind"] == "layer":
        module = s["module"]
        lvx.set_global_cross_attention_states(s["states"])
        out, _ = module(s["x"])
        grads = torch.autograd.grad(out, [s["x"], *module.parameters()], s["grad"])
        lvx.clear_global_cross_attention_states()
        return [out.detach(), *grads]
    q, k, v = s["q"], s["k"], s["v"]
    if "attention" not in s:
        _, _, _, o, lse = lvx._attn_forward(q, k, v, False, SCALE, None, kv_valid_len=s["valid"])
        return [o, lse]
    bias = (_image_bias, [s["image_of_key"]], [s["images_before"]]) if s["kind"] == "bias" else (None, [], [])
    o = s["attention"](q, k, v, False, SCALE, *bias, s["valid"])
    return [o.detach(), *torch.autograd.grad(o, (q, k, v), s["grad"])]


def work(case):
    es = 4 if case["dtype"] == "fp32" else 2
    Sq, Skv, Hq, Hkv = case["Sq"], case["Skv"], case["Hq"], case["Hkv"]
    if case["kind"] == "layer":
        hidden = case["hidden"]
        pairs = Hq * Sq * Skv
        weights = 2 * hidden * 128 * (Hq + Hkv)
        # attention 2 + 5 products; K/V projection forward, again in backward, and its weight gradients; q and o
        # projections forward and both gradients
        flops = 7 * 2 * pairs * 128 + 3 * 2 * Skv * hidden * 2 * Hkv * 128 + 3 * 2 * Sq * hidden * 2 * Hq * 128
        return {"bytes": es * (Skv * hidden + 4 * Sq * hidden + 2 * weights), "flops": flops}
    B = case["B"]
    keys = _valid(case) if case["padded"] else [Skv] * B
    q_bytes, kv_bytes = es * Hq * Sq * 128, es * Hkv * 128
    if case["backward"]:
        # q, k, v, dO in; o, dQ, dK, dV out (gradients of padded keys are written too)
        return {"bytes": 4 * B * q_bytes + 2 * kv_bytes * (sum(keys) + B * Skv), "flops": 7 * 2 * 128 * Hq * Sq * sum(keys)}
    return {"bytes": 2 * B * q_bytes + 4 * B * Hq * Sq + 2 * kv_bytes * sum(keys), "flops": 2 * 2 * 128 * Hq * Sq * sum(keys)}


def tolerance(case):
    # about four times the error against the same computation in 64 bits, measured over the listed and a dozen drawn
    # cases: fp32 1.2e-6 (growing with the number of keys), 16-bit attention 2.9e-3 (fp16 3.6e-4, but 4e-3 where the
    # probabilities of 200,000 keys are subnormal), with a bias 1.7e-3, the layer with its projections and norms 6.0e-3
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 2e-4}
    if case["kind"] == "layer":
        return {"rel": 2.4e-2, "max": 0.12}
    if case["kind"] == "bias":
        return {"rel": 7e-3, "max": 0.04}
    return {"rel": 1.2e-2, "max": 0.1}


def _attention64(q, k, v, valid, bias, grad):
    """Attention of q [B, Hq, Sq, 128] over k, v [B, Hkv, Skv, 128] in 64 bits, a block of query rows at a time: o and
    lse [B * Hq, Sq], and with an upstream gradient dq, dk, dv."""
    B, Hq, Sq, _ = q.shape
    per_kv = Hq // k.shape[1]
    o, lse = torch.empty_like(q), q.new_empty(B, Hq, Sq)
    grads = [torch.zeros_like(t) for t in (q, k, v)] if grad is not None else []
    step = max(1, (1 << 27) // k.shape[2])
    for b in range(B):
        n = valid[b] if valid is not None else k.shape[2]
        for h in range(Hq):
            kh, vh = k[b, h // per_kv, :n], v[b, h // per_kv, :n]
            for i in range(0, Sq, step):
                rows = slice(i, min(i + step, Sq))
                scores = q[b, h, rows] @ kh.T * SCALE
                if bias is not None:
                    scores += bias[0, 0, rows, :n]
                lse[b, h, rows] = torch.logsumexp(scores, -1)
                p = scores.sub_(lse[b, h, rows, None]).exp_()
                o[b, h, rows] = p @ vh
                if grad is not None:
                    dq, dk, dv = grads
                    do = grad[b, h, rows]
                    dv[b, h // per_kv, :n] += p.T @ do
                    ds = p.mul_(do @ vh.T - (do * o[b, h, rows]).sum(-1, keepdim=True)).mul_(SCALE)
                    dq[b, h, rows] = ds @ kh
                    dk[b, h // per_kv, :n] += ds.T @ q[b, h, rows]
    return [o, lse.view(B * Hq, Sq), *grads]


def _layer64(case, s):
    Hq, Hkv = case["Hq"], case["Hkv"]
    module, eps = s["module"], s["module"].q_norm.variance_epsilon
    leaves = {"x": s["x"], **dict(module.named_parameters())}
    leaves = {name: t.detach().double().requires_grad_() for name, t in leaves.items()}

    def heads(t, weight, n):
        return (t @ weight.T).view(1, -1, n, 128).transpose(1, 2)

    def norm(t, weight):
        return weight * t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + eps)

    states = s["states"].double()
    q = norm(heads(leaves["x"], leaves["q_proj.weight"], Hq), leaves["q_norm.weight"])
    k = norm(heads(states, leaves["k_proj.weight"], Hkv), leaves["k_norm.weight"])
    v = heads(states, leaves["v_proj.weight"], Hkv)
    grad = s["grad"].double()
    d_attn = heads(grad, leaves["o_proj.weight"].detach().T, Hq)
    o, _, dq, dk, dv = _attention64(q.detach(), k.detach(), v.detach(), None, None, d_attn)
    attn = o.transpose(1, 2).reshape(1, -1, Hq * 128)
    out = attn @ leaves["o_proj.weight"].T
    return [out.detach(), *torch.autograd.grad((q, k, v, out), list(leaves.values()), (dq, dk, dv, grad))]


def exact(case, seed):
    s = prepare(case, seed)
    if s["kind"] == "layer":
        return _layer64(case, s)
    bias = _image_bias(s["image_of_key"], s["images_before"]).double() if s["kind"] == "bias" else None
    q, k, v = (s[n].detach().double() for n in "qkv")
    o, lse, *grads = _attention64(q, k, v, s["valid"], bias, s["grad"].double() if case["backward"] else None)
    return [o, *grads] if case["backward"] else [o, lse]
