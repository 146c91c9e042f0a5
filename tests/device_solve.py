"""pt_poisson_solve_batch on images in device memory, for tests: what a caller with
resident images does (the call captures its work into a graph or replays it)."""
import ctypes as C

import numpy as np


def solve_batch(ctx, problems, want_history=False):
    """problems: dicts as Context.solve_batch takes; returns its (out, per-channel reports) pairs."""
    import torch
    from paintop_b200 import _lib
    n = len(problems)
    arr, outs, keep = (_lib.PtProblem * n)(), (C.c_void_p * n)(), []
    reps = [(_lib.PtReport * (p["channels"] + 1))() for p in problems]
    hists = [torch.zeros(max(p["channels"] * p["max_iterations"], 1), dtype=torch.float64, device="cuda") for p in problems]
    for i, p in enumerate(problems):
        bufs = [torch.from_numpy(np.ascontiguousarray(p[k], dtype=np.float32)).cuda() for k in ("source", "target", "mask")]
        out = torch.empty(p["width"] * p["height"] * p["channels"], device="cuda")
        keep.append((bufs, out))
        arr[i] = ctx.make_problem(*(b.data_ptr() for b in bufs), p["width"], p["height"], p["channels"], p.get("lam", 0.0),
                                  p["max_iterations"], p["tolerance"], p.get("omega", 1.8),
                                  p.get("flags", 0) | _lib.PT_FLAG_DEVICE_POINTERS)
        outs[i] = out.data_ptr()
    torch.cuda.current_stream().synchronize()  # (not the device: another thread may be capturing a graph)
    st = _lib.lib().pt_poisson_solve_batch(
        ctx.h, arr, n, outs, (C.POINTER(_lib.PtReport) * n)(*(C.cast(r, C.POINTER(_lib.PtReport)) for r in reps)),
        (C.c_void_p * n)(*(h.data_ptr() for h in hists)) if want_history else None)
    if st != _lib.PT_OK:
        raise _lib.CudaError(st, ctx.last_error())
    got = []
    for p, (_, out), rep, hist in zip(problems, keep, reps, hists):
        h = hist.cpu().numpy()
        per = []
        for c in range(p["channels"]):
            at = c * p["max_iterations"]
            per.append(rep[c].as_dict(h[at:at + rep[c].history_len].tolist() if want_history else None))
        got.append((out.cpu().numpy(), per))
    return got
