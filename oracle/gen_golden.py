"""Generate tests/golden/stop_rule_golden.json from the REFERENCE ITSELF.

Run in the build container (``python oracle/gen_golden.py``): it imports the reference's own
src/algorithms/dp_solver.py and src/theory/optimal_stopping.py by file path, evaluates them
on seeded inputs and on the documented example (docs/guides/GETTING_STARTED.md:61-65), and
stores inputs + outputs as C99 hex floats so the comparison is bit-exact.  Also drives the
reference's UNMODIFIED src/serving/pipeline.py through stub stage/predictor modules
and records the resulting RequestResult fields.
"""
from __future__ import annotations

import json
import os
import random
import sys
import types

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from oracle import ref_loader  # noqa: E402

OUT = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden",
                   "stop_rule_golden.json")


def hx(x):
    return float(x).hex()


def main():
    dp = ref_loader.dp_solver()
    th = ref_loader.optimal_stopping()
    rng = random.Random(7)
    gold = {"source": "generated by oracle/gen_golden.py from /root/reference "
                      "src/algorithms/dp_solver.py and src/theory/optimal_stopping.py",
            "stopping_rule": [], "bayesian": [], "expected_cost": [], "policy": [], "pipeline": []}

    fixed = [
        ([0.3, 0.5, 0.7, 0.9], [1.0, 1.6, 4.2, 8.8], 1.0),   # GETTING_STARTED.md:61-65
        ([0.3, 0.5, 0.7, 0.9], [1.0, 1.6, 4.2, 8.8], 10.0),
        ([0.9, 0.95, 1.0], [1.0, 4.5, 10.0], 1.0),
        ([0.5, 0.5, 1.0], [1.0, 4.5, 10.0], 20.0),
        ([0.2, 1.0, 1.0], [1.0, 4.5, 10.0], 8.0),
        ([0.6, 1.0], [1.0, 4.5], 5.0),
        ([0.6, 1.0], [1.0, 4.5], 12.0),
        ([1.0], [1.0], 5.0),
        ([0.0, 0.0, 0.0, 0.0], [1.0, 2.0, 4.5, 10.0], 3.0),
        ([1.0, 1.0, 1.0, 1.0], [1.0, 2.0, 4.5, 10.0], 3.0),
    ]
    cases = [(p, C, lam, False, 1.0, 1.0) for p, C, lam in fixed]
    cost_sets = [[1.0, 4.5, 10.0], [1.0, 2.0, 4.5, 10.0], [1.0, 1.6, 4.2, 8.8], [1.0, 4.5]]
    lams = [0.1, 0.5, 1.0, 2.0, 5.0, 10.0, 20.0, 100.0]
    for _ in range(600):
        C = rng.choice(cost_sets)
        L = len(C)
        p = [rng.random() for _ in range(L)]
        if rng.random() < 0.5:
            p[-1] = 1.0
        if rng.random() < 0.2:
            C = [c * rng.uniform(0.5, 2.0) for c in C]
        lam = rng.choice(lams) if rng.random() < 0.7 else rng.uniform(0.0, 50.0)
        ra = rng.random() < 0.3
        a, b = (rng.choice([0.5, 1.0, 2.0, 5.0]), rng.choice([0.5, 1.0, 2.0, 5.0])) if ra else (1.0, 1.0)
        cases.append((p, C, lam, ra, a, b))
    for p, C, lam, ra, a, b in cases:
        k, J = dp.optimal_stopping_rule(list(p), list(C), lam, risk_adjustment=ra, alpha=a, beta=b)
        gold["stopping_rule"].append({"p": [hx(x) for x in p], "C": [hx(x) for x in C], "lam": hx(lam),
                                      "risk_adjustment": ra, "alpha": hx(a), "beta": hx(b),
                                      "k_star": int(k), "J": [hx(x) for x in J]})
    for ph, n in [(0.8, 100), (0.5, 100), (0.0, 100), (1.0, 100), (0.37, 250)] + \
                 [(rng.random(), rng.choice([1, 10, 100, 1000, 12345])) for _ in range(100)]:
        for a, b in [(1.0, 1.0), (2.0, 5.0), (0.5, 0.5)]:
            gold["bayesian"].append({"p_hat": hx(ph), "n_obs": n, "alpha": hx(a), "beta": hx(b),
                                     "out": hx(dp.bayesian_adjustment(ph, n, a, b))})
    for _ in range(100):
        C = rng.choice(cost_sets)
        p = [rng.random() for _ in C]
        lam = rng.choice(lams)
        s = rng.randrange(len(C))
        gold["expected_cost"].append({"p": [hx(x) for x in p], "C": [hx(x) for x in C], "lam": hx(lam),
                                      "stage": s, "out": hx(dp.compute_expected_cost(p, C, lam, s))})
    gold["expected_cost"].append({"p": [hx(0.9), hx(0.8)], "C": [hx(1), hx(1.6)], "lam": hx(1.0), "stage": 1,
                                  "out": hx(dp.compute_expected_cost([0.9, 0.8], [1, 1.6], 1.0, 1))})
    for lam in [1.0, 0.1, 0.01, 0.5, 2.0]:
        for q, c in [(None, None), ([0.5, 0.7, 0.9], [1.0, 4.5, 10.0]), ([0.2, 0.4, 0.6, 0.95], [1.0, 1.6, 4.2, 8.8])]:
            n = 4 if q is None else len(q)
            params = th.TheoreticalParameters(n_stages=n, quality_bounds=None if q is None else list(q),
                                              cost_ratios=None if c is None else list(c), lambda_param=lam)
            theory = th.OptimalStoppingTheory(params)
            pol = theory.derive_optimal_policy()
            gold["policy"].append({"quality_bounds": [hx(x) for x in theory.params.quality_bounds],
                                   "cost_ratios": [hx(x) for x in theory.params.cost_ratios], "lam": hx(lam),
                                   "thresholds": {str(s): hx(v) for s, v in pol.items()}})

    # --- the unmodified reference pipeline driven through stubs -------------------------------------
    import numpy as np
    stage_mod = types.ModuleType("refsrc.models.stage")
    pred_mod = types.ModuleType("refsrc.models.predictor")

    class Stage:
        def __init__(self, name, cost):
            self.name, self.cost_per_token = name, cost

        def generate(self, prompts, max_tokens=512, temperature=0.7, top_p=0.9, return_logprobs=True):
            return ([f"{self.name}-says: " + p[:16] for p in prompts],
                    [np.full((3, 5), -1.0)], {"generation_time_ms": 1.0})

    class StageManager:
        def __init__(self):
            self.stages = {n: Stage(n, c) for n, c in zip(["8b", "13b", "34b", "70b"], [1.0, 1.6, 4.2, 8.8])}

        def get_stage(self, name):
            return self.stages[name]

    class QualityPredictor:
        def __init__(self, seq):
            self.seq, self.i = seq, 0

        def predict(self, prompt, draft_output, draft_logprobs, stage_id, feature_extractor=None):
            v = self.seq[self.i % len(self.seq)]
            self.i += 1
            return v

    class FeatureExtractor:
        pass

    stage_mod.Stage, stage_mod.StageManager = Stage, StageManager
    pred_mod.QualityPredictor, pred_mod.FeatureExtractor = QualityPredictor, FeatureExtractor
    pm = ref_loader.pipeline_module(stage_mod, pred_mod)
    for lam, preds, ra in [(1.0, [0.3], True), (10.0, [0.05, 0.5, 0.9], True), (100.0, [0.01], False),
                           (0.1, [0.99], True)]:
        cfg = pm.PipelineConfig(lambda_value=lam, risk_adjustment=ra, enable_caching=False)
        pipe = pm.AdaptiveSpeculativePipeline(StageManager(), QualityPredictor(preds), FeatureExtractor(), cfg)
        res = pipe.process_request("What is the capital of France?", max_tokens=8, temperature=0.7,
                                   request_id="golden")
        pipe.shutdown()
        gold["pipeline"].append({"lam": hx(lam), "risk_adjustment": ra, "predictions": [hx(x) for x in preds],
                                 "output": res.output, "stopped_at_stage": res.stopped_at_stage,
                                 "stage_probabilities": [hx(x) for x in res.stage_probabilities],
                                 "stage_costs": [hx(x) for x in res.stage_costs],
                                 "cache_hits": res.cache_hits, "total_tokens": res.total_tokens})
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    with open(OUT, "w") as f:
        json.dump(gold, f, indent=0, sort_keys=True)
    print("wrote", OUT, {k: len(v) for k, v in gold.items() if isinstance(v, list)})


if __name__ == "__main__":
    main()
