"""The forward passes that users of m2_b200 run, as cases that can be timed.

Six ways into the package are covered, each through its public entry point:

  embed    M2BertEmbedder.encode: token-id lists on the host -> pooled vectors on the host
  graphed  GraphedForward over M2BertModel: fixed-shape throughput jobs, bf16
  eager    M2BertModel under torch.autocast(bfloat16), shapes that change from call to call
  float32  M2BertModel without autocast
  layer    the drop-in modules inside somebody else's encoder: mixer, then GLU MLP, bf16 autocast
  mixer    the sequence mixer alone on float32 activations

`shape` names the model: "80m" (12 layers, d_model 768, intermediate 3072) or "large" (24 layers, 1536, 6144).
Weights are the constructors' random init with filters of a trained filter's energy, token ids are uniform over the
vocabulary.
"""
import math

import torch

from m2_b200 import BertGatedLinearUnitMLP, GraphedForward, HyenaFilter, MonarchMixerSequenceMixing
from m2_b200.embed import M2BertEmbedder
from m2_b200.encoder import M2BertConfig, M2BertModel

SHAPES = {"80m": dict(layers=12, d=768, inter=3072), "large": dict(layers=24, d=1536, inter=6144)}
NBLOCKS = 4
VOCAB = 30528
DEVICE = "cuda"


def listed():
    return [
        # a search box: one short query is embedded while somebody waits for the answer
        dict(name="embed-1-query", what="embed", shape="80m", texts=1, batch=1, length=128),
        # indexing a few documents with the 2K retrieval model: ragged texts, padded to one length, a last part chunk
        dict(name="embed-20-docs", what="embed", shape="80m", texts=20, batch=8, length=2048),
        # an interactive classifier or a test: a small batch, launched call by call
        dict(name="eager-8x128", what="eager", shape="80m", batch=8, length=128),
        # batches padded to their own longest text: no length is round
        dict(name="eager-6x1531", what="eager", shape="80m", batch=6, length=1531),
        # bulk scoring of short texts, the shape that M2-BERT was pretrained at
        dict(name="graphed-256x128", what="graphed", shape="80m", batch=256, length=128),
        # bulk embedding of long documents with the 8K and the 32K models
        dict(name="graphed-32x8192", what="graphed", shape="80m", batch=32, length=8192),
        dict(name="graphed-8x32768", what="graphed", shape="80m", batch=8, length=32768),
        # the large model, at its pretraining length and at 2K
        dict(name="graphed-large-512x128", what="graphed", shape="large", batch=512, length=128),
        dict(name="graphed-large-64x2048", what="graphed", shape="large", batch=64, length=2048),
        # no autocast: checking a checkpoint, exporting reference activations
        dict(name="float32-4x512", what="float32", shape="80m", batch=4, length=512),
        # one encoder layer made of the drop-in modules, its input the float32 output of another library's LayerNorm
        dict(name="layer-16x1024", what="layer", shape="80m", batch=16, length=1024),
        # the mixer alone in float32 (8 sequences of 128 steps, the published single-layer configuration)
        dict(name="mixer-float32-8x128", what="mixer", shape="80m", batch=8, length=128),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _length(rng, lo, hi, ragged):
    """Log-uniform over [lo, hi]; where `ragged`, every other one is any number, else all are multiples of 8."""
    n = _log_int(rng, lo, hi)
    return n if ragged and rng.random() < 0.5 else min(hi, max(8, n // 8 * 8))


def draw(rng):
    what = rng.choice(["embed", "graphed", "graphed", "eager", "eager", "float32", "layer", "mixer"])
    shape = "80m"
    if what == "embed":
        length = rng.choice([128, 256, 512, 1024, 2048, 8192])
        batch = _log_int(rng, 1, max(1, min(32, 32768 // length)))
        return dict(what=what, shape=shape, texts=_log_int(rng, 1, 3 * batch), batch=batch, length=length)
    if what == "graphed":
        shape = rng.choice(["80m", "80m", "large"])
        most, longest = (262144, 32768) if shape == "80m" else (131072, 2048)
        length = _length(rng, 64, longest, False)
        tokens = _log_int(rng, max(length, 8192), most)
    elif what == "eager":
        length = _length(rng, 16, 2048, True)
        tokens = _log_int(rng, max(length, 64), 16384)
    elif what == "float32":
        length = _length(rng, 16, 1024, True)
        tokens = _log_int(rng, max(length, 64), 4096)
    elif what == "layer":
        shape = rng.choice(["80m", "large"])
        length = _length(rng, 32, 4096, True)
        tokens = _log_int(rng, max(length, 256), 32768)
    else:
        length = _length(rng, 16, 2048, True)
        tokens = _log_int(rng, max(length, 64), 8192)
    return dict(what=what, shape=shape, batch=max(1, tokens // length), length=length)


def _config(case):
    s, l_max = SHAPES[case["shape"]], max(128, 1 << (case["length"] - 1).bit_length())
    return M2BertConfig(vocab_size=VOCAB, hidden_size=s["d"], intermediate_size=s["inter"], num_hidden_layers=s["layers"],
                        max_position_embeddings=l_max, long_conv_l_max=l_max, pool_all=case["what"] == "embed")


def _settle(module, conf):
    """Divides the filters' last weights by sqrt(l_max / 128).  A filter's taps then have the same energy at every length,
    as those of a trained model do; with the constructor's init it grows with the length, the gated product behind it
    grows with it, and from 1K on a deep stack of such layers amplifies single roundings until nothing can be compared."""
    with torch.no_grad():
        for m in module.modules():
            if isinstance(m, HyenaFilter):
                for net in (m.implicit_filter, m.implicit_filter_rev):
                    net[6].weight.div_(math.sqrt(conf.long_conv_l_max / 128))
    return module.eval()


def _layer(conf):
    mixer = MonarchMixerSequenceMixing(conf.hidden_size, l_max=conf.long_conv_l_max, bidirectional=True, hyena_emb_dim=5,
                                       hyena_filter_order=128, hyena_w=10, residual_long_conv=True,
                                       hyena_kernel_lr=1e-3, hyena_lr_pos_emb=1e-5)
    return _settle(mixer, conf), BertGatedLinearUnitMLP(conf).eval()


def prepare(case, seed):
    """Model and inputs on the GPU (for `embed`: token lists on the host), the handle that such a program keeps, and one
    forward behind it, so that weights and filter tables are laid out."""
    torch.manual_seed(seed)
    what, conf = case["what"], _config(case)
    B, L = case["batch"], case["length"]
    with torch.device(DEVICE):
        if what in ("layer", "mixer"):
            mixer, mlp = _layer(conf)
            u = torch.nn.functional.layer_norm(torch.randn(B, L, conf.hidden_size), (conf.hidden_size,))
            state = dict(what=what, mixer=mixer, mlp=mlp, u=u)
            run(state)
            return state
        model = _settle(M2BertModel(conf, add_pooling_layer=what == "embed"), conf)
    if what == "embed":
        g = torch.Generator().manual_seed(seed)
        lens = torch.randint(max(1, L // 8), L + 1, (case["texts"],), generator=g).tolist()
        texts = [torch.randint(1, VOCAB, (n,), generator=g).tolist() for n in lens]
        embedder = M2BertEmbedder(model, max_len=L, batch_size=B)
        embedder.encode([[1]])
        return dict(what=what, embedder=embedder, texts=texts)
    ids = torch.randint(0, VOCAB, (B, L), device=DEVICE)
    state = dict(what=what, model=model, ids=ids)
    if what == "graphed":
        state["graphed"] = GraphedForward(model, ids.clone(), warmup=1)
    else:
        run(state)
    return state


def run(state):
    what = state["what"]
    if what == "embed":
        return state["embedder"].encode(state["texts"])
    if what == "graphed":
        return state["graphed"](state["ids"])[0]
    with torch.no_grad():
        if what == "float32":
            return state["model"](state["ids"])[0]
        if what == "mixer":
            return state["mixer"](state["u"])[0]
        with torch.autocast("cuda", dtype=torch.bfloat16):
            if what == "eager":
                return state["model"](state["ids"])[0]
            mixed, _ = state["mixer"](state["u"])
            return state["mlp"](mixed)


def work(case):
    """Multiplications and additions of the GEMMs and of the convolutions as real FFTs (one forward, one inverse of 2L
    points for each of the two filters of a channel and sequence, the filters' own transforms done ahead); bytes of the
    weights in the compute type, of the filters, and of what enters and leaves."""
    s = SHAPES[case["shape"]]
    what, L, D, inter = case["what"], case["length"], s["d"], s["inter"]
    rows = case["texts"] if what == "embed" else case["batch"]
    layers = 1 if what in ("layer", "mixer") else s["layers"]
    size = 4 if what in ("float32", "mixer") else 2
    mlp_weights = 0 if what == "mixer" else 3 * inter * D // NBLOCKS
    weights = 4 * D * D + mlp_weights
    conv = rows * D * 2 * (2 * 2.5 * 2 * L * math.log2(2 * L))
    flops = layers * (2 * rows * L * weights + conv)
    nbytes = layers * (size * weights + 2 * size * 2 * L * D)
    if what in ("layer", "mixer"):
        nbytes += 2 * 4 * rows * L * D                                     # activations in and out, float32
    else:
        nbytes += rows * L * 8 + 4 * D * (min(rows * L, VOCAB) + L)        # ids and the embedding rows they name
        nbytes += 4 * D * rows * (1 if what == "embed" else L)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    what = case["what"]
    if what == "mixer":
        return {"rel": 2e-5}
    if what == "float32":
        return {"rel": 1e-4}      # twelve layers, each of which passes on the rounding of the one before
    if what == "layer":
        return {"rel": 1e-2}
    # bf16 between all operators; each layer adds its own rounding and passes on that of the layers before it (the two
    # long-convolution families of this package, same taps, differ by 0.8 to 1.3e-2 after twelve layers, by 1.9e-2 after 24
    # layers at 2K and by 2.2e-2 after twelve at 32K)
    return {"rel": 3e-2 if case["shape"] == "large" or case["length"] > 8192 else 2e-2}
