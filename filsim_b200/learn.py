"""Learned Broyden warm start: host side of the fs_mlp_* / fs_learn_* entry points.

The library owns the network (one per context) and runs every forward,
backward and Adam step in its own kernels; this module prepares the data,
drives training, and saves / loads parameters. There is no reference
counterpart: the reference always starts Broyden from the extrapolated guess
(Filament::initialGuess, Filament.hpp:227-237) with J0^-1 as the initial
inverse Jacobian.

Training pairs are generated by the plain solver: before a step the features
of the state are taken (fs_learn_features); after the step converges the
library writes the targets (fs_learn_targets): the update from the
extrapolated guess to the converged state and the diagonal of the Broyden
correction accumulated during the step.
"""
import ctypes

import numpy as np
import torch

from . import abi
from .abi import check, lib
from .fcm import Context, Simulation

WARM_PLAIN, WARM_LEARNED, WARM_LEARNED_DIAG = 0, 1, 2


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _np_ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


class WarmStartModel:
    """The context's MLP: features (19 per bead, 9 per link, log K_B) -> 3 x (hidden + SiLU) -> 12 nw outputs."""

    def __init__(self, ctx, nw, hidden=256, batch_capacity=4096, seed=0):
        self.ctx = ctx
        check(lib().fs_mlp_create(ctx.h, nw, hidden, batch_capacity, seed), "fs_mlp_create")
        d = np.zeros(8, dtype=np.int32)
        check(lib().fs_mlp_dims(ctx.h, _np_ptr(d)), "fs_mlp_dims")
        (self.nw, self.n_features, self.k_in, self.hidden, self.n_targets, self.k_out, self.capacity,
         self.n_params) = (int(v) for v in d)
        self.in_mean = np.zeros(self.n_features, np.float32)
        self.in_std = np.ones(self.n_features, np.float32)
        self.out_mean = np.zeros(self.n_targets, np.float32)
        self.out_std = np.ones(self.n_targets, np.float32)

    @property
    def dims(self):
        return [self.k_in, self.hidden, self.hidden, self.hidden, self.k_out]

    def set_normalization(self, in_mean, in_std, out_mean, out_std):
        self.in_mean, self.in_std, self.out_mean, self.out_std = (
            np.ascontiguousarray(a, dtype=np.float32) for a in (in_mean, in_std, out_mean, out_std))
        check(lib().fs_mlp_set_normalization(self.ctx.h, _np_ptr(self.in_mean), _np_ptr(self.in_std),
                                             _np_ptr(self.out_mean), _np_ptr(self.out_std)),
              "fs_mlp_set_normalization")

    def fit_normalization(self, feats, tgts):
        """Per-column mean and standard deviation of the training data (constant columns get 1)."""
        f = feats.double()
        t = tgts.double()

        def stats(a):
            mu = a.mean(0)
            sd = a.std(0)
            # columns with no spread (or only rounding noise) are passed through centred
            sd = torch.where(sd > 1e-12 * (1.0 + mu.abs()), sd, torch.ones_like(sd))
            return mu.cpu().numpy(), sd.cpu().numpy()

        im, isd = stats(f)
        om, osd = stats(t)
        self.set_normalization(im, isd, om, osd)

    def params(self):
        out = np.zeros(self.n_params, np.float32)
        check(lib().fs_mlp_get_params(self.ctx.h, _np_ptr(out), out.size), "fs_mlp_get_params")
        return out

    def set_params(self, flat):
        flat = np.ascontiguousarray(flat, dtype=np.float32)
        check(lib().fs_mlp_set_params(self.ctx.h, _np_ptr(flat), flat.size), "fs_mlp_set_params")

    def forward(self, feats):
        feats = feats.to(device="cuda", dtype=torch.float32).contiguous()
        out = torch.empty((feats.shape[0], self.n_targets), dtype=torch.float32, device="cuda")
        self.ctx.call("fs_mlp_forward", _ptr(feats), feats.shape[0], _ptr(out))
        return out

    def gradients(self, feats, tgts):
        feats = feats.to(device="cuda", dtype=torch.float32).contiguous()
        tgts = tgts.to(device="cuda", dtype=torch.float32).contiguous()
        g = np.empty(self.n_params, np.float32)  # written whole
        loss = ctypes.c_double()
        self.ctx.call("fs_mlp_gradients", _ptr(feats), _ptr(tgts), feats.shape[0], _np_ptr(g), g.size,
                      ctypes.byref(loss))
        return g, loss.value

    def train_step(self, feats, tgts, lr, want_loss=False):
        loss = ctypes.c_double()
        check(lib().fs_mlp_train_step(self.ctx.h, _ptr(feats), _ptr(tgts), feats.shape[0], float(lr),
                                      ctypes.byref(loss) if want_loss else None), "fs_mlp_train_step")
        return loss.value if want_loss else None

    def fit(self, feats, tgts, epochs=40, batch=None, lr=1e-3, lr_final=1e-4, seed=0, log=None):
        """Adam over shuffled mini-batches with a geometric learning-rate decay; returns
        the mean training loss of each epoch (normalised units)."""
        feats = feats.to(device="cuda", dtype=torch.float32).contiguous()
        tgts = tgts.to(device="cuda", dtype=torch.float32).contiguous()
        n = feats.shape[0]
        batch = min(batch or self.capacity, self.capacity, n)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        losses = []
        steps = epochs * max(1, n // batch)
        k = 0
        for ep in range(epochs):
            perm = torch.randperm(n, device="cuda", generator=gen)
            tot, cnt = 0.0, 0
            for b0 in range(0, n - batch + 1, batch):
                idx = perm[b0:b0 + batch]
                fb = feats[idx].contiguous()
                tb = tgts[idx].contiguous()
                rate = lr * (lr_final / lr) ** (k / max(1, steps - 1))
                last = b0 + 2 * batch > n
                loss = self.train_step(fb, tb, rate, want_loss=last)
                k += 1
                if last:
                    if not np.isfinite(loss):
                        raise FloatingPointError("warm-start training loss is not finite (epoch %d)" % ep)
                    tot += loss
                    cnt += 1
            losses.append(tot / max(1, cnt))
            if log:
                log("epoch %d loss %.4g" % (ep, losses[-1]))
        self.ctx.synchronize()
        return losses

    def save(self, path):
        np.savez(path, params=self.params(), in_mean=self.in_mean, in_std=self.in_std, out_mean=self.out_mean,
                 out_std=self.out_std, dims=np.array([self.nw, self.hidden], np.int32))

    def load(self, path):
        d = np.load(path)
        nw, hidden = (int(v) for v in d["dims"])
        if nw != self.nw or hidden != self.hidden:
            raise ValueError("saved model is for nw=%d hidden=%d" % (nw, hidden))
        self.set_params(d["params"])
        self.set_normalization(d["in_mean"], d["in_std"], d["out_mean"], d["out_std"])


def set_warm_start(ctx, mode):
    check(lib().fs_set_warm_start(ctx.h, mode), "fs_set_warm_start")


def model_rows(susp, nw):
    """Indices of the filaments of nw beads."""
    lens = np.diff(susp.fil_start)
    return np.nonzero(lens == nw)[0]


def record(sim, model, nt_start, nsteps):
    """Runs nsteps implicit steps (with the context's current start) and returns the
    (features, targets) pairs of the filaments the model serves, as CUDA tensors.
    Steps that did not converge contribute no pairs, nor do rows with a
    non-finite value."""
    ctx = sim.ctx
    nfil = sim.susp.nfil
    rows = torch.as_tensor(model_rows(sim.susp, model.nw), device="cuda")
    check(lib().fs_learn_record(ctx.h, 1), "fs_learn_record")
    feats, tgts, iters = [], [], []
    try:
        for k in range(nsteps):
            f = torch.empty((nfil, model.n_features), dtype=torch.float32, device="cuda")
            ctx.call("fs_learn_features", _ptr(f))
            it, st = sim.step_implicit(nt_start + k)
            iters.append(it)
            if st != abi.FS_OK:
                continue
            t = torch.empty((nfil, model.n_targets), dtype=torch.float32, device="cuda")
            ctx.call("fs_learn_targets", _ptr(t))
            f, t = f[rows], t[rows]
            ok = torch.isfinite(f).all(1) & torch.isfinite(t).all(1)
            feats.append(f[ok])
            tgts.append(t[ok])
    finally:
        check(lib().fs_learn_record(ctx.h, 0), "fs_learn_record")
    return torch.cat(feats), torch.cat(tgts), iters


def generate(make_case, seeds, warm_steps, record_steps, kb_range=(0.1, 10.0), precision=abi.FS_PREC_FP32,
             model=None, log=None):
    """Training data from plain-solver runs: for each seed a suspension with K_B drawn
    log-uniformly in kb_range, warm_steps steps to pass the start-up (implicit
    Euler and the linear lambda extrapolation), then record_steps recorded steps.
    make_case(seed, kap) -> (params, suspension)."""
    feats, tgts, its = [], [], []
    own = model is None
    ctx = None if own else model.ctx
    for s in seeds:
        rng = np.random.default_rng(s)
        kb = float(np.exp(rng.uniform(np.log(kb_range[0]), np.log(kb_range[1]))))
        p, susp = make_case(s, kb)
        if ctx is None:
            ctx = Context(p, max_beads=susp.np, max_filaments=susp.nfil)
            model = WarmStartModel(ctx, int(np.diff(susp.fil_start)[0]), batch_capacity=128)
        ctx.set_precision(precision)
        set_warm_start(ctx, WARM_PLAIN)
        sim = Simulation(ctx, susp)
        sim.run_steps(1, warm_steps)
        f, t, it = record(sim, model, warm_steps + 1, record_steps)
        feats.append(f)
        tgts.append(t)
        its += it
        if log:
            log("seed %d K_B %.3g: %d pairs, iters %s" % (s, kb, f.shape[0], it))
    out = torch.cat(feats), torch.cat(tgts), its
    if own:
        ctx.close()
    return out
