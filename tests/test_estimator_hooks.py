"""Methods of the estimators that a subclass may override are called, on the CPU: whole rounds and whole predictions in
the library are for the methods of this package only."""
import numpy as np
import torch

import legateboost_b200 as lb
from legateboost_b200 import estimator as E


def test_overridden_gradients_keep_the_rounds_in_python():
    class Weighted(lb.LBRegressor):
        def _weighted_gradient(self, y, raw_pred):
            g, h = super()._weighted_gradient(y, raw_pred)
            return 2 * g, 2 * h

    plain, weighted, patched = lb.LBRegressor(), Weighted(), lb.LBRegressor()
    patched._weighted_gradient = lambda y, raw_pred: (raw_pred - y, torch.ones_like(y))
    for m in (plain, weighted, patched):
        m._obj = m._objective()
    assert plain._rounds_in_library()
    assert not weighted._rounds_in_library() and not patched._rounds_in_library()


def test_overridden_raw_predictions_reach_the_probabilities():
    class Shifted(lb.LBClassifier):
        def predict_raw(self, X):
            return torch.full((X.shape[0], self.model_init_.shape[0]), 2.0, dtype=torch.float64)

    X = torch.zeros((3, 4))
    for K in (1, 3):
        m = Shifted()
        m._obj, m.models_, m.n_features_in_, m.model_init_ = E._LogLoss(), [], 4, torch.zeros(K, dtype=torch.float64)
        p = m.predict_proba(X).numpy()
        want = [1 - 1 / (1 + np.exp(-2.0)), 1 / (1 + np.exp(-2.0))] if K == 1 else [1 / 3] * 3
        assert np.allclose(p, [want] * 3, rtol=1e-14)
