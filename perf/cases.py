"""What the framework is timed on: training steps and evaluation passes of its own models through ``AutoDist`` ->
``scope`` -> ``create_distributed_session`` -> ``sess.run``, from the smallest step (launch-bound) to the headline one.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` builds what a user's program
holds before the call (a session over a model with random weights, one batch on the device), ``run`` is one call, ``work``
the bytes and operations one call cannot do without and ``tolerance`` how far another correct implementation at the same
precision may be off.
"""
import atexit
import gc
import math

import torch

from autodist_b200 import AutoDist
from autodist_b200 import strategy as S
from autodist_b200.autodist import _reset_default_autodist
from autodist_b200.models.bert import BertConfig, BertPretrainer
from autodist_b200.models.cnn import ImageClassifier, ResNet
from autodist_b200.models.lm1b import LM1B, LM1BConfig
from autodist_b200.models.ncf import NeuMF, NeuMFConfig
from autodist_b200.resource_spec import ResourceSpec

DEVICE = "cuda:0"

#: Parameters of the convolutional backbones (1000 classes) and multiply-adds of one forward pass on one 224 x 224 image.
CNN = {"resnet14": (9.0e6, 1.2e9), "resnet50": (25.6e6, 4.1e9), "resnet101": (44.5e6, 7.8e9), "vgg16": (138.4e6, 15.5e9),
       "densenet121": (8.0e6, 2.9e9), "inceptionv3": (24.0e6, 3.5e9)}


def _bert(name, hidden, layers, batch, seq, preds, vocab=30522, dropout=0.1, tie=False, train=True):
    case = {"kind": "bert", "hidden": hidden, "layers": layers, "batch": batch, "seq": seq, "preds": preds, "vocab": vocab,
            "dropout": dropout, "tie": tie, "train": train}
    return dict(case, name=name) if name else case


def _cnn(name, backbone, batch, image, train=True):
    case = {"kind": "cnn", "backbone": backbone, "batch": batch, "image": image, "train": train}
    return dict(case, name=name) if name else case


def _lm(name, vocab, batch, steps, state, projected, sampled):
    case = {"kind": "lm", "vocab": vocab, "batch": batch, "steps": steps, "state": state, "projected": projected, "sampled": sampled}
    return dict(case, name=name) if name else case


def _ncf(name, users, items, batch):
    case = {"kind": "ncf", "users": users, "items": items, "batch": batch}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the headline: BERT-large pre-training, 32 sequences of 128 tokens per GPU, Adam (bench.py's default)
        _bert("bert_large_s128", 1024, 24, 32, 128, 20),
        # its second phase: long sequences, 76 predictions each, where attention grows with the square of the length
        _bert("bert_large_s512", 1024, 24, 6, 512, 76),
        # the base model on an odd batch (7 sequences of 256 tokens), no dropout, output projection tied to the embeddings
        _bert("bert_base_tied", 768, 12, 7, 256, 38, dropout=0.0, tie=True),
        # evaluation of the base model: forward only, the loss is read back
        _bert("bert_base_eval", 768, 12, 32, 128, 20, train=False),
        # the smallest step: the tiny configuration of the tests, bound by latency and launches
        _bert("bert_tiny", 128, 2, 4, 128, 8, vocab=1000),
        # the second headline: ResNet-101, 64 images per GPU, SGD with momentum
        _cnn("resnet101_train", "resnet101", 64, 224),
        # a short residual network (one block per stage) on an odd batch of odd-sized images: odd feature maps, few rows per layer
        _cnn("resnet14_ragged", "resnet14", 13, 203),
        # evaluation mode, logits out (running statistics in the batch-norms)
        _cnn("resnet50_eval", "resnet50", 32, 224, train=False),
        # plain 3 x 3 convolutions with bias + ReLU and the 25088 x 4096 / 4096 x 4096 fully connected layers
        _cnn("vgg16_train", "vgg16", 32, 224),
        # many narrow layers of growing width
        _cnn("densenet121_train", "densenet121", 16, 224),
        # LM1B: one LSTM layer over 20 steps, sampled softmax, row-sparse tables of the 793471-word vocabulary, Adagrad + clip
        _lm("lm1b_train", 793471, 128, 20, 2048, 512, 8192),
        # recommendation: NeuMF on the ml-20m shape, dense embedding gradients, Adam
        _ncf("ncf_train", 138493, 26744, 16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bert", "bert", "bert", "cnn", "cnn", "cnn", "lm", "ncf"])
    if kind == "bert":
        hidden = rng.choice([128, 256, 512, 768, 1024])
        layers = _log_int(rng, 2, 24)
        seq = rng.choice([64, 128, 256, 512])
        batch = _log_int(rng, 2, min(48, 4000 // seq))
        return _bert(None, hidden, layers, batch, seq, max(1, int(0.15 * seq)), vocab=rng.choice([1000, 21128, 30522]),
                     dropout=rng.choice([0.0, 0.1, 0.1]), tie=rng.random() < 0.3, train=rng.random() < 0.8)
    if kind == "cnn":
        backbone = rng.choice(["resnet14", "resnet50", "resnet101", "vgg16", "densenet121", "inceptionv3"])
        image = rng.randint(160, 224)
        batch = _log_int(rng, 4, 16 if backbone == "densenet121" else 32 if backbone == "vgg16" else 56)
        return _cnn(None, backbone, batch, image, train=rng.random() < 0.8)
    if kind == "lm":
        state = rng.choice([512, 1024, 2048])
        return _lm(None, _log_int(rng, 10000, 793471), _log_int(rng, 8, 128), rng.randint(5, 20), state, state // 4,
                   8 * _log_int(rng, 64, 1024))
    return _ncf(None, _log_int(rng, 6000, 138493), _log_int(rng, 3700, 26744), _log_int(rng, 256, 32768))


class _Job:
    """A session with its batch; gives its buffers back when the last reference goes."""

    def __init__(self, autodist, session, fetches, feed, model, gradients):
        self.autodist, self.session, self.fetches, self.feed, self.model = autodist, session, fetches, feed, model
        # Gradients come back beside the updated weights where bf16 determines them. In a randomly initialised batch-norm network
        # of any depth it does not: two correct implementations (measured: this one and the library's) agree on the loss to 1e-3
        # and on no digit of the gradient. A BERT step's gradient mixes magnitudes in one buffer and is judged through Adam's update.
        self.gradients = gradients

    def __del__(self):
        try:
            atexit.unregister(self.autodist._shutdown)
            engine = self.session.engine
            self.session.close()
            engine.__dict__.clear()
            for p in self.model.parameters():
                p.__dict__.clear()
                p.grad, p.data = None, torch.empty(0)
            if hasattr(self.model, "materialize"):
                self.model.flat = self.model._ws = self.model.grad_ready = None
        except Exception:      # interpreter shutdown
            pass


def _bert_config(case):
    return BertConfig(vocab_size=case["vocab"], hidden_size=case["hidden"], num_hidden_layers=case["layers"],
                      num_attention_heads=case["hidden"] // 64, intermediate_size=4 * case["hidden"], max_position_embeddings=512,
                      hidden_dropout_prob=case["dropout"], attention_probs_dropout_prob=case["dropout"],
                      tie_word_embeddings=case["tie"])


def _batch(case, gen):
    """One batch on the device, with the distributions the models' own synthetic inputs have."""
    def ints(hi, *shape):
        return torch.randint(0, hi, shape, generator=gen, device=DEVICE)

    kind, n = case["kind"], case["batch"]
    if kind == "bert":
        s, p = case["seq"], case["preds"]
        ids = ints(case["vocab"], n, s)
        pos = torch.rand(n, s, generator=gen, device=DEVICE).argsort(1)[:, :p].sort(1).values
        # sequences of different lengths: the last quarter of the positions is padding for some of them
        length = s - ints(max(1, s // 4), n)
        mask = (torch.arange(s, device=DEVICE)[None] < length[:, None]).to(torch.int64)
        return {"input_ids": ids, "input_mask": mask, "segment_ids": ints(2, n, s), "mlm_positions": pos,
                "mlm_ids": torch.gather(ids, 1, pos), "mlm_weights": torch.ones(n, p, device=DEVICE), "nsp_labels": ints(2, n)}
    if kind == "cnn":
        return {"images": torch.randn(n, 3, case["image"], case["image"], generator=gen, device=DEVICE), "labels": ints(1000, n)}
    if kind == "lm":
        # Zipf(1.1) over the vocabulary by inverting the continuous distribution function
        u = torch.rand(n, case["steps"] + 1, generator=gen, device=DEVICE, dtype=torch.float64)
        v, a = case["vocab"], 1.0 - 1.1
        ids = ((u * (v ** a - 1.0) + 1.0) ** (1.0 / a)).long().clamp_(1, v) - 1
        return {"x": ids[:, :-1].contiguous(), "y": ids[:, 1:].contiguous()}
    return {"users": ints(case["users"], n), "items": ints(case["items"], n),
            "labels": (torch.arange(n, device=DEVICE) % 5 == 0).float()}


def _model(case):
    kind = case["kind"]
    if kind == "bert":
        return BertPretrainer(_bert_config(case))
    if kind == "cnn":
        if case["backbone"] == "resnet14":          # one bottleneck block per stage
            return ImageClassifier(ResNet((1, 1, 1, 1)))
        return ImageClassifier(case["backbone"], **({"image_size": case["image"]} if case["backbone"] == "vgg16" else {}))
    if kind == "lm":
        return LM1B(LM1BConfig(vocab_size=case["vocab"], emb_size=case["projected"], state_size=case["state"],
                               projected_size=case["projected"], num_sampled=case["sampled"], num_steps=case["steps"]))
    return NeuMF(NeuMFConfig(num_users=case["users"], num_items=case["items"], dense_gradient=True))


def prepare(case, seed):
    gc.collect()
    _reset_default_autodist()
    torch.manual_seed(seed)
    gen = torch.Generator(device=DEVICE).manual_seed(seed + 1)
    kind = case["kind"]
    data = _batch(case, gen)
    autodist = AutoDist(resource_spec=ResourceSpec.local(num_gpus=1), strategy_builder=S.AllReduce(chunk_size=256))
    with autodist.scope():
        with torch.device(DEVICE):          # random weights are drawn on the device
            model = _model(case)
        holders = {k: autodist.placeholder((None,) + tuple(v.shape[1:]), v.dtype, name=k) for k, v in data.items()}
        loss = model(**holders)
        if kind == "lm":
            optimizer = torch.optim.Adagrad(model.parameters(), lr=0.2, initial_accumulator_value=1.0)
            train_op = optimizer.minimize(loss, clip_global_norm=(10.0, model.dense_parameters()))
        elif kind == "cnn":
            train_op = torch.optim.SGD(model.parameters(), lr=1e-4, momentum=0.9).minimize(loss)      # start of a warm-up
        else:
            train_op = torch.optim.Adam(model.parameters(), lr=1e-4).minimize(loss)
        session = autodist.create_distributed_session()
    if kind == "cnn" and not case["train"]:
        # running statistics as training leaves them: a mean and a variance for every channel
        with torch.no_grad():
            for name, buf in model.named_buffers():
                if name.endswith("running_mean"):
                    buf.normal_(0.0, 0.05)
                elif name.endswith("running_var"):
                    buf.uniform_(0.05, 0.15)
        model.eval()
    fetches = [loss, train_op] if case.get("train", True) else [loss]
    return _Job(autodist, session, fetches, {holders[k]: v for k, v in data.items()}, model, kind in ("lm", "ncf"))


def run(job):
    if not job.model.training:
        images = next(v for v in job.feed.values() if v.dim() == 4)
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return {"logits": job.model.net(images.contiguous(memory_format=torch.channels_last))}
    out = job.session.run(job.fetches, job.feed)
    if len(out) == 1:
        return {"loss": out[0]}
    engine = job.session.engine
    result = {"loss": out[0], "weights": engine.flat.master}
    if job.gradients:
        result["grad"] = engine.flat.grad
    for name, rows in engine.sharded_rows.items():
        result[name] = rows.master
    return result


def _bert_parameters(case):
    h, v = case["hidden"], case["vocab"]
    return case["layers"] * (12 * h * h + 13 * h) + (v + 514) * h + (0 if case["tie"] else v * h) + v + 2 * h * h + 10 * h


def work(case):
    """Operations: 2 per multiply-add of every contraction, backward twice the forward. Bytes: weights (bf16 or fp32) once, and
    for training the gradient written once and master weights and optimizer state read and written once, plus the batch;
    activations are left out (a pass could keep them on the chip)."""
    kind, n = case["kind"], case["batch"]
    train = case.get("train", True)
    if kind == "bert":
        h, s, p = case["hidden"], case["seq"], case["preds"]
        params = _bert_parameters(case)
        forward = 2.0 * n * s * case["layers"] * (12 * h * h + 2 * s * h) + 2.0 * n * p * (h * h + h * case["vocab"]) + 2.0 * n * h * h
        return {"bytes": params * (30 if train else 2) + 8.0 * n * (3 * s + 3 * p), "flops": forward * (3 if train else 1)}
    if kind == "cnn":
        params, macs = CNN[case["backbone"]]
        if case["backbone"] == "vgg16":
            fc = 512 * (case["image"] // 32) ** 2 * 4096.0
            macs = (macs - 123.6e6) * (case["image"] / 224.0) ** 2 + fc + 20.9e6
            params = params - 102.8e6 + fc
        else:
            macs *= (case["image"] / 224.0) ** 2
        return {"bytes": params * (22 if train else 2) + 12.0 * n * case["image"] ** 2, "flops": 2.0 * macs * n * (3 if train else 1)}
    if kind == "lm":
        t, st, pr, k = n * case["steps"], case["state"], case["projected"], case["sampled"]
        dense = 8.0 * st * pr + 4 * st + pr * st
        rows = 2.0 * t + k                                   # looked-up rows: read as bf16, updated with their accumulator in fp32
        return {"bytes": dense * 22 + rows * pr * 20 + case["vocab"] * 20.0 + 16.0 * t,
                "flops": 6.0 * t * (8 * st * pr + st * pr + pr * k)}
    width = 64 + 128
    params = (case["users"] + case["items"]) * width + 256 * 256 + 256 * 128 + 128 * 64
    return {"bytes": params * 30.0 + 20.0 * n, "flops": 6.0 * n * (256 * 256 + 256 * 128 + 128 * 64)}


def tolerance(case):
    """About four times what was measured between this code and another computation of the same precision or better, over three
    steps: BERT against fp32 arithmetic with no dropout (loss 1.4e-3, weights 9.5e-4, largest weight 2.6e-2 of the mean square
    root), the convolutional networks against the library's bf16 kernels (loss 6.7e-3, the largest weight 0.17; evaluation:
    logits 3.8e-3, largest 1.2e-2), LM1B and NeuMF with library matrix products (gradient 1.5e-3 and 1.0e-3, largest 7.0e-2
    and 0.20)."""
    kind = case["kind"]
    if kind == "bert":
        return {"rel": 0.005, "max": 0.1}
    if kind == "cnn":
        return {"rel": 0.03, "max": 0.5} if case["train"] else {"rel": 0.015, "max": 0.05}
    return {"rel": 0.006, "max": 0.3} if kind == "lm" else {"rel": 0.004, "max": 0.8}
