"""A thin boosting-round driver over ``Tree``: just enough of ``LBRegressor`` / ``LBClassifier`` to
grow an ensemble and measure rounds per second.

It restates the reference's round (legateboost/legateboost.py:254-298): gradient of the objective
at the current prediction, times the learning rate (``_get_weighted_gradient``, :189-224, hessian
floored at 1e-8), ``Tree(...).set_random_state(rs).fit(X, g, h)``, ``train_pred += tree.predict(X)``.
Objectives: squared error (objectives.py:119-147) and multi-class / binary log loss
(objectives.py:477-531).  Everything else of the estimators (callbacks, metrics registry, other base
models, update, sklearn plumbing) is outside the tree-building hot path and is not provided.
Arrays are torch CUDA tensors; under ``torch.distributed`` each rank holds a block of rows.
"""
import ctypes as C
from copy import deepcopy
from typing import List, Optional

import numpy as np
import torch

from . import library as L
from .tree import _ARRAYS, Sketch, Tree, TreeTable, _row_layout, _tensor_key


def _several_ranks() -> bool:
    import torch.distributed as dist

    return dist.is_available() and dist.is_initialized() and dist.get_world_size() > 1


def _all_sum(t: torch.Tensor) -> torch.Tensor:
    import torch.distributed as dist

    if _several_ranks():
        dist.all_reduce(t)
    return t


def _is_own(model, name: str) -> bool:
    """Whether a method is _LBBase's own, overridden neither in a subclass nor on the object."""
    return getattr(getattr(model, name), "__func__", None) is _LBBase.__dict__[name]


def _is_own_sampling(base: Tree) -> bool:
    """Whether a base model samples features as Tree does."""
    return getattr(base._sample_features, "__func__", None) is Tree._sample_features


def _is_plain(base: Tree) -> bool:
    """Whether a base model's attributes are plain values, as they are as a rule."""
    return all(type(v) in (int, float, str, bool, type(None)) for v in base.__dict__.values())


def _copy_of(base: Tree, plain: bool) -> Tree:
    """deepcopy of a base model."""
    if plain:
        tree = Tree.__new__(Tree)
        tree.__dict__.update(base.__dict__)
        return tree
    return deepcopy(base)


class _NoSeed(np.random.bit_generator.ISeedSequence):
    """For a generator that is seeded right after it is made."""

    def generate_state(self, n_words, dtype=np.uint32):
        return np.zeros(n_words, dtype=dtype)


def _random_state(seed) -> np.random.RandomState:
    """RandomState(seed).  That one first seeds its generator from the system's entropy, which takes 100 of its 140 us."""
    if type(seed) is not int:
        return np.random.RandomState(seed)
    state = np.random.RandomState(np.random.MT19937(_NoSeed()))
    state.seed(seed)
    return state


def _counts_by_comparison(num_class: int, n: int) -> bool:
    """Whether n labels are counted by comparing each with every class, which reads n x num_class values, instead of by
    bincount, which waits for the device twice more and whose atomics meet in num_class words.  Microseconds, bincount and
    comparison: 2 classes, 4M labels 529 and 168, 6 classes, 8M 492 and 454; 8 classes, 1M 186 and 149, 4M 303 and 335;
    16 classes, 500k 169 and 152, 1M 175 and 219, 4M 261 and 564.  (2^26: the comparisons' bytes)"""
    return num_class * n <= (1 << 26 if num_class <= 6 else 1 << 23) and num_class <= 16


class _SquaredError:
    code = 0  # LBK_SQUARED_ERROR

    def gradient(self, y, pred):
        return pred - y, torch.ones_like(pred)

    def transform(self, pred):
        return pred

    def init(self, y, average):
        if not average:
            return torch.zeros(y.shape[1], dtype=torch.float64, device=y.device)
        count = torch.full((1,), float(y.shape[0]), dtype=torch.float64, device=y.device)
        if not _several_ranks():
            return y.sum(dim=0) / count
        s = _all_sum(torch.cat([y.sum(dim=0), count]))
        return s[:-1] / s[-1]

    def metric(self, y, pred):
        s = _all_sum(torch.cat([((y - pred) ** 2).sum(dim=0), torch.tensor([float(y.shape[0])], dtype=torch.float64, device=y.device)]))
        return float((s[:-1] / s[-1]).mean())


class _LogLoss:
    code = 1  # LBK_LOG_LOSS

    def gradient(self, y, pred):
        if pred.shape[1] == 1:
            return pred - y, pred * (1.0 - pred)
        label = y.to(torch.int64).reshape(-1)
        h = pred * (1.0 - pred)
        g = pred.clone()
        g[torch.arange(label.numel(), device=g.device), label] -= 1.0
        return g, h

    def transform(self, pred):
        if pred.shape[1] == 1:
            return 1.0 / (1.0 + torch.exp(-pred))
        s = pred.max(dim=1, keepdim=True).values
        e = torch.exp(pred - s)
        return e / e.sum(dim=1, keepdim=True)

    def init(self, y, average):
        lo = 0.0
        if _several_ranks():
            import torch.distributed as dist

            mx = torch.tensor([float(y.max()) if y.numel() else 0.0], dtype=torch.float64, device=y.device)
            dist.all_reduce(mx, op=dist.ReduceOp.MAX)
            hi = mx.item()
        else:
            lo, hi = torch.stack(torch.aminmax(y)).tolist() if y.numel() else (0.0, 0.0)
        num_class = int(hi) + 1
        n_targets = num_class if num_class > 2 else 1
        if not average:
            return torch.zeros(n_targets, dtype=torch.float64, device=y.device)
        labels = y.reshape(-1).to(torch.int64)
        if _several_ranks() or lo <= -1.0 or not _counts_by_comparison(num_class, y.numel()):
            counts = _all_sum(torch.bincount(labels, minlength=num_class).to(torch.float64))
        else:  # (bincount waits for the device twice more; it refuses negative labels)
            counts = (labels[:, None] == torch.arange(num_class, device=y.device)).sum(dim=0, dtype=torch.float64)
        prob = counts / counts.sum()
        if n_targets == 1:
            return -torch.log(1.0 / prob[1:2] - 1.0)
        return torch.log(prob)

    def metric(self, y, pred):
        eps = torch.finfo(pred.dtype).eps
        p = pred.clamp(eps, 1 - eps)
        if p.shape[1] == 1:
            yy = y.reshape(-1)
            p = p.reshape(-1)
            ll = -(yy * torch.log(p) + (1 - yy) * torch.log(1 - p))
        else:
            label = y.to(torch.int64).reshape(-1)
            ll = -torch.log(p[torch.arange(label.numel(), device=p.device), label])
        s = _all_sum(torch.stack([ll.sum(), torch.tensor(float(ll.numel()), dtype=torch.float64, device=p.device)]))
        return float(s[0] / s[1])


class _LBBase:
    _objective = None

    def __init__(self, n_estimators: int = 100, learning_rate: float = 0.1, init: Optional[str] = "average",
                 base_models=(Tree(max_depth=6),), random_state=None, verbose: int = 0, fixed_sketch: bool = False):
        # fixed_sketch (an extension, off by default): the first tree of every base model saves its
        # split proposals and binned matrix, the later ones reuse them instead of sampling and
        # binning X again; the trees then differ from the reference's, which re-samples per tree
        self.fixed_sketch = fixed_sketch
        self.n_estimators = n_estimators
        self.learning_rate = learning_rate
        self.init = init
        self.base_models = base_models
        self.random_state = random_state
        self.verbose = verbose

    def _check(self, X, y):
        if not (torch.is_tensor(X) and X.is_cuda):
            raise ValueError("X must be a CUDA tensor (there is no CPU path)")
        if X.dtype not in (torch.float32, torch.float64):
            X = X.to(torch.float32)  # integer X -> float32 (reference: input_validation.py:73-75)
        y = torch.as_tensor(y, device=X.device).to(torch.float64)  # y -> float64 (:85)
        if y.dim() == 1:
            y = y[:, None]
        if y.shape[0] != X.shape[0]:
            raise ValueError("Number of labels does not match number of samples.")
        return X, y

    def _weighted_gradient(self, y, raw_pred):
        """g * learning_rate and h floored at 1e-8 at the current raw prediction, in one pass over the
        rows (`lbk_gradient`; reference: `_get_weighted_gradient`, legateboost.py:189-224)."""
        code = getattr(self._obj, "code", None)
        if code is None:  # an objective the library has no kernel for
            g, h = self._obj.gradient(y, self._obj.transform(raw_pred))
            return g * self.learning_rate, torch.clamp(h, min=1e-8)
        raw_pred = raw_pred.contiguous()
        y = y.contiguous()
        g = torch.empty_like(raw_pred)
        h = torch.empty_like(raw_pred)
        ctx = L.context(raw_pred.device.index)
        with torch.cuda.device(raw_pred.device):
            ctx.check(ctx.lib.lbk_gradient(ctx.handle, code, raw_pred.data_ptr(), y.data_ptr(), raw_pred.shape[0],
                                           raw_pred.shape[1], float(self.learning_rate), g.data_ptr(), h.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream))
        return g, h

    def fit(self, X, y):
        X, y = self._check(X, y)
        if not isinstance(self.base_models, tuple) or len(self.base_models) == 0:
            raise ValueError("base_models should be a tuple")
        self.n_features_in_ = X.shape[1]
        self.models_: List[Tree] = []
        rs = self.random_state
        self.random_state_ = rs if isinstance(rs, np.random.RandomState) else _random_state(rs)
        self._obj = self._objective()
        self.model_init_ = self._obj.init(y, self.init == "average")
        self.train_metric_: List[float] = []
        train_pred = self.model_init_.expand(X.shape[0], -1).clone(memory_format=torch.contiguous_format)
        layout = _row_layout(X.shape[0])  # this rank's block of rows: the same for every tree
        if self._rounds_in_library():
            try:
                self._fit_rounds(X, y, train_pred, layout)
            except BaseException:
                # the rounds before the one that failed are queued and read the caller's tensors
                torch.cuda.current_stream(X.device).synchronize()
                raise
            self._train_pred = train_pred
            return self
        sketches = {}
        for i in range(self.n_estimators):
            g, h = self._weighted_gradient(y, train_pred)
            tree = deepcopy(self.base_models[i % len(self.base_models)]).set_random_state(self.random_state_)
            tree.row_layout = layout
            if self.fixed_sketch:
                tree.sketch = sketches.setdefault(i % len(self.base_models), Sketch())
            tree.fit(X, g, h)
            tree.sketch = None  # the buffer belongs to this fit, not to the tree
            self.models_.append(tree)
            train_pred += tree.predict(X)
            if self.verbose:
                m = self._obj.metric(y, self._obj.transform(train_pred))
                self.train_metric_.append(m)
                print("[%d] train: %.6f" % (i, m))
        self._train_pred = train_pred
        return self

    def _rounds_in_library(self) -> bool:
        """Whether a round is one `lbk_boost_round` call: plain trees, an objective the library knows, gradients
        that nobody overrides (sample weights, say), nothing to report per round."""
        return (not self.verbose and self.n_estimators > 0 and type(self._obj) in (_SquaredError, _LogLoss)
                and _is_own(self, "_weighted_gradient")
                and all(type(b) is Tree and not callable(b.feature_fraction) and b.max_depth >= 0 for b in self.base_models))

    def _fit_rounds(self, X, y, train_pred, layout):
        """The rounds of fit(), one library call each, queued without waiting for the device.  What the host
        decides - seeds and feature samples, in the order in which Tree.fit draws them - is drawn before
        the first round; the trees of up to 64 rounds share one allocation per array."""
        N, F = X.shape
        K = train_pred.shape[1]
        dev, rs = X.device, self.random_state_
        bases = [self.base_models[i % len(self.base_models)] for i in range(self.n_estimators)]
        masks = None
        if type(rs) is np.random.RandomState and all(b.feature_fraction >= 1.0 and _is_own_sampling(b) for b in self.base_models):
            seeds = rs.randint(0, 2**31, size=self.n_estimators).tolist()  # (the same draws as one by one)
        else:
            seeds, masks = [], np.ones((self.n_estimators, F), dtype=np.uint8)
            for i, b in enumerate(bases):
                seeds.append(int(rs.randint(0, 2**31)))
                mask = b._sample_features(rs, F)
                if mask is not None:
                    masks[i] = mask
            masks = None if masks.all() else torch.from_numpy(masks).to(dev)
        if X.stride(1) != 1 and N > 0:
            X = X.contiguous()
        y = y.contiguous()
        ctx = L.init_distributed(dev.index)
        lib, handle, stream = ctx.lib, ctx.handle, torch.cuda.current_stream(dev).cuda_stream
        r = L.BoostRoundArgs()
        a = r.tree
        a.X, a.x_dtype, a.ldx = X.data_ptr(), L.LBK_F32 if X.dtype == torch.float32 else L.LBK_F64, X.stride(0) if N > 0 else F
        a.row_offset, a.dataset_rows = layout
        a.n_local_rows, a.n_features, a.n_outputs = N, F, K
        a.stream = stream
        r.objective, r.y, r.pred, r.learning_rate = self._obj.code, y.data_ptr(), train_pred.data_ptr(), float(self.learning_rate)
        ref, sketches, made = C.byref(r), {}, []
        n_bases = len(self.base_models)
        at = 0
        while at < self.n_estimators:
            run = list(range(at, min(at + 64, self.n_estimators)))
            at += len(run)
            zeroed = torch.zeros((len(run),), dtype=torch.int32, device=dev)
            of_base = {}
            for b in range(min(n_bases, len(run))):
                first = run[b]
                M, n = 2 ** (bases[first].max_depth + 1) - 1, (len(run) - b + n_bases - 1) // n_bases
                f64 = dict(dtype=torch.float64, device=dev)
                arrays = {
                    "leaf_value": torch.empty((n, M, K), **f64), "feature": torch.empty((n, M), dtype=torch.int32, device=dev),
                    "split_value": torch.empty((n, M), **f64), "gain": torch.empty((n, M), **f64),
                    "hessian": torch.empty((n, M, K), **f64),
                }
                of_base[first % n_bases] = (arrays, [(t.data_ptr(), t.stride(0) * t.element_size()) for t in arrays.values()], M)
            for j, i in enumerate(run):
                base = bases[i]
                _, where, M = of_base[i % n_bases]
                q = j // n_bases  # which tree of its base model's this is
                a.leaf_value, a.feature, a.split_value, a.gain, a.hessian = [p + q * step for p, step in where]
                a.feature_set = None if masks is None else masks.data_ptr() + i * F
                r.zeroed = zeroed.data_ptr() + 4 * j
                a.max_depth, a.max_nodes = base.max_depth, M
                a.split_samples, a.seed = base.split_samples, seeds[i]
                a.l1_regularization, a.l2_regularization = base.l1_regularization, base.l2_regularization
                a.min_split_gain = base.min_split_gain
                sketch = None
                if self.fixed_sketch:
                    sketch = sketches.setdefault(i % n_bases, Sketch())
                    a.sketch_mode = sketch.mode_for(X, base.split_samples, ctx)
                    a.sketch = sketch.buffer.data_ptr()
                ctx.check(lib.lbk_boost_round(handle, ref))
                if sketch is not None:
                    sketch.key = (_tensor_key(X), base.split_samples)
            made.append((run, of_base, zeroed))
        # (the trees' objects are made while the rounds run)
        models, plain = [], [_is_plain(b) for b in self.base_models]
        for run, of_base, _ in made:
            parts = {b: {name: t.unbind(0) for name, t in arrays.items()} for b, (arrays, _, _) in of_base.items()}
            for j, i in enumerate(run):
                tree = _copy_of(bases[i], plain[i % n_bases])
                tree.__dict__.update({name: p[j // n_bases] for name, p in parts[i % n_bases].items()},
                                     random_state=rs, row_layout=layout, sketch=None, _fit_rows=None)
                models.append(tree)
        ctx.check(lib.lbk_synchronize(handle, stream))
        self.models_ = models

    def predict_raw(self, X):
        return self._predict(X, L.RAW)

    def _predict(self, X, transform):
        """Initial prediction plus the trees' sums, and what `transform` makes of them, in one call.  The
        table of the trees' addresses is kept as long as models_ holds the same tensors."""
        if X.shape[1] != self.n_features_in_:
            raise ValueError("X.shape[1] = {} should be equal to {}".format(X.shape[1], self.n_features_in_))
        assert X.is_cuda, "X must be a CUDA tensor (no CPU fallback)"
        init = self.model_init_
        if init.dtype != torch.float64 or not init.is_contiguous() or init.device != X.device:
            init = init.to(device=X.device, dtype=torch.float64).contiguous()
        if not self.models_:
            raw = init.repeat(X.shape[0], 1)
            return raw if transform == L.RAW else self._probabilities(raw)
        table = self.__dict__.get("_table")
        if table is None or not table.matches(self.models_):
            assert all(isinstance(m, Tree) for m in self.models_)
            table = TreeTable(list(map(_ARRAYS, self.models_)))
            self._table = table if table.reusable else None
        if table.n_outputs != init.shape[0]:  # (trees of the user's own with one column for all outputs)
            raw = init.repeat(X.shape[0], 1)
            raw += table.predict(X, table.n_outputs)
            return raw if transform == L.RAW else self._probabilities(raw)
        return table.predict(X, init.shape[0], init=init, transform=transform)

    def __getstate__(self):
        state = dict(self.__dict__)
        state.pop("_table", None)  # addresses of this process
        return state

    def __iter__(self):
        return iter(self.models_)

    def __getitem__(self, i):
        return self.models_[i]

    def __len__(self):
        return len(self.models_)


class LBRegressor(_LBBase):
    """Gradient-boosted regression with the squared-error objective."""

    _objective = _SquaredError

    def predict(self, X):
        pred = self._obj.transform(self.predict_raw(X))
        return pred.squeeze(1) if pred.shape[1] == 1 else pred


class LBClassifier(_LBBase):
    """Gradient-boosted classification with the log-loss objective."""

    _objective = _LogLoss

    def _probabilities(self, raw):
        pred = self._obj.transform(raw)
        if pred.shape[1] == 1:
            pred = torch.cat([1.0 - pred, pred], dim=1)
        return pred

    def predict_proba(self, X):
        if type(self._obj) is not _LogLoss or not _is_own(self, "predict_raw"):
            return self._probabilities(self.predict_raw(X))
        return self._predict(X, L.LOGISTIC if self.model_init_.shape[0] == 1 else L.SOFTMAX)

    def predict(self, X):
        return self.predict_proba(X).argmax(dim=1)
