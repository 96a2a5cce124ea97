"""FP64 runs of unlike structures and one batch of them, as checked_run.py does
it for single FP32 runs: one JSON line with counts, flights and (for a
bounds-checked build) ptg_check_report.  Used by tests/test_gpu_checked.py."""
import json

import numpy as np
from checked_run import A, cases, synth


def _checksum(counts):
    return int(np.sum(counts.ravel() * np.arange(1, counts.size + 1, dtype=np.uint64)))


def main():
    out = {}
    spec = synth.spectrum(8, seed=1, mfp_lo=2e-9, mfp_hi=2e-6)
    models = cases()
    for name, m in models.items():
        gb = A.GeomBuf(m)
        with A.Handle(gb.view, spec) as h:
            k = h.kappa(A.make_run(kind_mfp=A.MFP_PER_MODE, nangle=7, np_=100, seed=5, precision=A.PREC_FP64),
                        want_counts=True)
            out[name] = [_checksum(k["counts"]), int(h.stats()["flights"])]
    bufs = [A.GeomBuf(m) for m in models.values()]
    n = len(bufs)
    run = A.make_run(kind_mfp=A.MFP_PER_MODE, nangle=7, np_=1)
    with A.Batch([b.view for b in bufs], [50 + 17 * i for i in range(n)], list(range(n)), [0] * n, spec, run) as bt:
        r = bt.run(want_counts=True)
        a = bt.adjoint()
        out["batch"] = [_checksum(r["counts"]), int(r["flights"]), int(a["replayed"]), int(a["mismatched"])]
    try:
        out["check"] = A.check_report()
    except A.PtgError as e:
        out["check"] = {"status": e.status}
    print(json.dumps(out))


if __name__ == "__main__":
    main()
