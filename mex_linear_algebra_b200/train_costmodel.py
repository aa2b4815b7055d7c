"""Train the cost model on a timing database and report its regret.

    python -m mex_linear_algebra_b200.train_costmodel --train train.json --eval eval.json \
        --steps 16000 --lr 5e-3 --seeds 5 --out mex_linear_algebra_b200/costmodel.json

(and the same, 20000 steps, with a database of wide requests for costmodel_wide.json).

Training runs on the GPU in the library's own kernels.  The report compares,
on the evaluation records (every variant timed), the total time of the
model's choices with the exhaustive best (regret) and with the fixed rule.
"""
import argparse
import json

from . import costmodel


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--train", required=True)
    ap.add_argument("--eval", required=True)
    ap.add_argument("--out", default=costmodel.DEFAULT_MODEL)
    ap.add_argument("--steps", type=int, default=4000)
    ap.add_argument("--lr", type=float, default=3e-3)
    ap.add_argument("--seeds", type=int, default=1,
                    help="train from so many starts, keep the one with the least regret on the training records")
    a = ap.parse_args()
    train = json.load(open(a.train))
    ev = json.load(open(a.eval))
    runs = []
    for seed in range(a.seeds):
        p, loss = costmodel.train(train, steps=a.steps, lr=a.lr, seed=seed)
        rep = costmodel.evaluate(p, train)
        runs.append((rep["regret"] + rep["mean_request_regret"], seed, p, loss, rep))
    _, seed, params, loss, rep_train = min(runs, key=lambda r: r[0])
    rep_eval = costmodel.evaluate(params, ev)
    costmodel.save(params, a.out, meta={"train_records": len(train), "eval_records": len(ev), "seed": seed,
                                        "final_loss": loss, "eval": rep_eval, "train": rep_train})
    print(json.dumps({"final_loss": loss, "train": rep_train, "eval": rep_eval}, indent=1))


if __name__ == "__main__":
    main()
