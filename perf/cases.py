"""The work that users of this package have it do, as cases to be timed.

A network is Flatten -> LogicLayer(n_in, width) -> (layers - 1) x LogicLayer(width, width) -> GroupSum(classes, tau) with
random connections and standard normal gate weights.  Four uses of it, each through the package's public interface:

  train    one optimizer step on a batch of binary float features: the plain loop (forward, loss, backward, FlatAdam.step)
           or, with `captured`, a TrainStep whose step was captured in a CUDA graph and is fed a new batch;
  score    float features through the network in eval mode (validation between two epochs);
  packed   a bool matrix packed into words of `bits` bits and counted by the network in eval mode;
  pixels   uint8 pixels, thermometer-encoded and packed in one call, then counted the same way.

Inputs are synthetic: Bernoulli features, uniform pixels, uniform class labels.
"""
import math

import torch

import difflogic_b200 as D
from difflogic_b200.optim import FlatAdam
from difflogic_b200.training import TrainStep

THRESHOLDS = (63, 127, 191)   # three thermometer features per pixel


def _train(name, n_in, width, layers, classes, tau, batch, captured, grad_factor=1.0, ones=0.19):
    return {"name": name, "use": "train", "n_in": n_in, "width": width, "layers": layers, "classes": classes, "tau": tau,
            "batch": batch, "captured": captured, "grad_factor": grad_factor, "ones": ones}


def _score(name, n_in, width, layers, classes, tau, batch, ones=0.19):
    return {"name": name, "use": "score", "n_in": n_in, "width": width, "layers": layers, "classes": classes, "tau": tau,
            "batch": batch, "ones": ones}


def _packed(name, n_in, width, layers, classes, batch, bits, ones=0.19):
    return {"name": name, "use": "packed", "n_in": n_in, "width": width, "layers": layers, "classes": classes, "tau": 1.0,
            "batch": batch, "bits": bits, "ones": ones}


def _pixels(name, pixels, width, layers, classes, batch, bits):
    return {"name": name, "use": "pixels", "n_in": len(THRESHOLDS) * pixels, "width": width, "layers": layers, "classes": classes,
            "tau": 1.0, "batch": batch, "bits": bits}


def listed():
    return [
        # a small tabular set trained with the plain loop: every size odd, nothing but launches and host work
        _train("train_loop_tabular", 117, 1001, 3, 7, 10.0, 61, False, ones=0.5),
        # the plain loop at the sizes of the smallest 28 x 28 network
        _train("train_loop_784_8000", 784, 8000, 4, 10, 10.0, 100, False),
        # the last, incomplete batch of an epoch
        _train("train_loop_last_batch", 784, 16000, 5, 10, 30.0, 75, False),
        # the same network in full batches, captured: how a whole epoch is trained
        _train("train_step_784_16000", 784, 16000, 5, 10, 30.0, 128, True),
        # a wide network on thermometer-encoded images
        _train("train_step_9216_128000", 9216, 128000, 4, 10, 100.0, 256, True, ones=0.5),
        # a deep network at a large batch (the largest training work)
        _train("train_step_256_64000_deep", 256, 64000, 12, 2, 20.0, 1024, True, grad_factor=2.0, ones=0.5),
        # validation in float between two epochs
        _score("score_784_16000", 784, 16000, 5, 10, 30.0, 1000),
        # one request of a serving process, default word width
        _packed("packed_784_8000_request", 784, 8000, 4, 10, 100, 32),
        # a test set of ten thousand samples, default word width: rows are no multiple of 16 bytes
        _packed("packed_784_16000_test_set", 784, 16000, 5, 10, 10000, 32),
        # bulk inference
        _packed("packed_784_8000_bulk", 784, 8000, 4, 10, 1 << 20, 64),
        # bulk inference with a deep and wide network
        _packed("packed_256_64000_deep", 256, 64000, 12, 2, 1 << 17, 64, ones=0.5),
        # a test set of ten thousand images straight from their pixels
        _pixels("pixels_3072_128000_test_set", 3072, 128000, 4, 10, 10000, 64),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    use = rng.choice(["loop", "step", "step", "score", "packed", "packed", "pixels"])
    classes = rng.choice([2, 3, 7, 10, 10, 16, 100])
    layers = rng.randint(2, 12)
    width = _log_uniform(rng, 400, 128000)
    if rng.random() < 0.5:                       # round numbers are what people choose
        step = 1000 if width >= 4000 else 100
        width = max(step, width // step * step)
    width = max(1, width // classes) * classes
    n_in = min(_log_uniform(rng, 16, 9216), 2 * width)
    ones = rng.choice([0.19, 0.5])
    # tau grows with the classes, as it has to for the scores not to saturate the loss
    tau = float(rng.choice([t for t in (1, 10, 30, 100) if t * 4 >= math.sqrt(width / classes)]))
    if use in ("loop", "step"):
        most = min(2048, 12 * 64000 * 1024 // (layers * width))
        batch = _log_uniform(rng, 16, max(16, most))
        if rng.random() < 0.5:
            batch = max(16, batch // 16 * 16)
        c = _train("", n_in, width, layers, classes, tau, batch, use == "step", 2.0 if layers > 6 else 1.0, ones)
    elif use == "score":
        c = _score("", n_in, width, layers, classes, tau, _log_uniform(rng, 16, max(16, min(10000, 12 * 64000 * 1024 // (layers * width)))),
                   ones)
    else:
        most = min(1 << 20, 12 * 64000 * (1 << 17) // (layers * width), (1 << 30) // n_in)
        batch = _log_uniform(rng, 1, most)
        if rng.random() < 0.3:
            batch = max(64, batch // 64 * 64)
        bits = rng.choice([8, 16, 32, 32, 64, 64])
        if use == "packed":
            c = _packed("", n_in, width, layers, classes, batch, bits, ones)
        else:
            c = _pixels("", max(8, n_in // len(THRESHOLDS)), width, layers, classes, batch, bits)
    del c["name"]
    return c


def _network(case):
    n_in = case["n_in"]
    layers = [torch.nn.Flatten()]
    for i in range(case["layers"]):
        layers.append(D.LogicLayer(n_in if i == 0 else case["width"], case["width"], device="cuda",
                                   grad_factor=case.get("grad_factor", 1.0), connections="random"))
    layers.append(D.GroupSum(case["classes"], tau=case["tau"]))
    return torch.nn.Sequential(*layers)


def prepare(case, seed):
    torch.manual_seed(seed)
    state = {"case": case, "model": _network(case)}
    if case["use"] == "pixels":
        state["x"] = torch.randint(0, 256, (case["batch"], case["n_in"] // len(THRESHOLDS)), dtype=torch.uint8, device="cuda")
    else:
        ones = torch.empty((case["batch"], case["n_in"]), dtype=torch.float32 if case["use"] in ("train", "score") else torch.bool,
                           device="cuda")
        state["x"] = ones.bernoulli_(case["ones"])
    if case["use"] != "train":
        state["model"].eval()
        return state
    state["y"] = torch.randint(0, case["classes"], (case["batch"],), device="cuda")
    state["opt"] = FlatAdam(state["model"].parameters(), lr=0.01)
    if case["captured"]:
        state["step"] = TrainStep(state["model"], state["opt"], torch.nn.CrossEntropyLoss())
        state["step"].capture(state["x"], state["y"])
    else:
        state["loss_fn"] = torch.nn.CrossEntropyLoss()
    return state


def run(state):
    case, model, x = state["case"], state["model"], state["x"]
    if case["use"] == "train":
        opt = state["opt"]
        if case["captured"]:
            loss = state["step"](x, state["y"])
            return {"loss": loss, "weights": opt.flat_param, "exp_avg": opt.exp_avg, "exp_avg_sq": opt.exp_avg_sq}
        scores = model(x)
        loss = state["loss_fn"](scores, state["y"])
        opt.zero_grad()
        loss.backward()
        opt.step()
        return {"loss": loss, "scores": scores, "gradients": [p.grad for p in model.parameters()], "weights": opt.flat_param,
                "exp_avg": opt.exp_avg, "exp_avg_sq": opt.exp_avg_sq}
    with torch.no_grad():
        if case["use"] == "score":
            return model(x)
        if case["use"] == "packed":
            return model(D.PackBitsTensor(x, bit_count=case["bits"]))
        return model(D.PackBitsTensor.from_uint8_thresholds(x, THRESHOLDS, bit_count=case["bits"]))


def work(case):
    """Training: every activation is written once, read by the next layer and again by its own layer's backward pass, every
    gradient of one written and read once; weights and both moments are read and written.  Inference: the input read and the
    scores or counts written; what lies between could stay on the chip."""
    n_in, width, layers, batch, classes = (case[k] for k in ("n_in", "width", "layers", "batch", "classes"))
    gates = layers * width
    per_gate = 16 + 64                                   # two connection indices, sixteen weights
    if case["use"] == "train":
        hidden = 4 * batch * width * (layers - 1)        # the last layer's output goes straight into the class sums
        bytes_ = 4 * batch * n_in * 2 + hidden * 5 + 8 * batch + gates * (per_gate + 5 * 64)
        if not case["captured"]:
            bytes_ += gates * 2 * 64 + 4 * batch * classes   # the gradients are handed to the user
        return {"bytes": bytes_, "flops": gates * batch * (7 + 8 + 7)}
    if case["use"] == "score":
        return {"bytes": 4 * batch * (n_in + classes) + gates * per_gate, "flops": gates * batch * 7}
    source = n_in if case["use"] == "packed" else n_in // len(THRESHOLDS)
    return {"bytes": batch * (source + 4 * classes) + gates * (16 + 1), "flops": gates * (batch / 32.0)}


def tolerance(case):
    if case["use"] in ("packed", "pixels"):
        return "exact"
    if case["use"] == "score":
        return {"rel": 1e-6}   # sums of zeros and ones are exact in float; only the division by tau can round
    # Against the same steps in 64 bits: weights 2e-7, gradients and first moments up to 1e-5, second moments 1.4e-5 (the
    # rounding of 1 - 0.999 in float).  Scores of size s carry an absolute error of about 1e-7 s, which the softmax turns
    # into a relative one of the gradients: 1.7e-4, and 3.5e-4 of their squares, at s = 1600.
    return {"rel": 5e-5 + 1e-6 * case["width"] / (case["classes"] * case["tau"])}
