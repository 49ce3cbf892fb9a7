"""CELO2_CUDA and ELO_CELO2_CUDA on the B200 kernels.

Drop-in for the reference classes of the same names
(pylo/optim/CELO2_cuda.py:54-341, pylo/optim/ELO_CELO2_cuda.py:39-298): same
constructor arguments, param-group keys, per-parameter state keys and shapes
(``mom (3,)+shape``, ``rms shape``, ``fac_r``, ``fac_c``; for the independent
AdamW branch ``exp_avg``, ``exp_avg_sq``, ``adam_step``), hence the same
``state_dict`` / resume format.

What differs is where the work runs.  The reference does the accumulator
updates with ~10 torch ops per tensor and then calls a two-kernel extension per
tensor.  Here every tensor of a param group goes through one multi-tensor
launch per phase: row/column sums of g^2, factor update, fused EMA + feature
moments, normaliser folding, network + raw step; then Newton-Schulz, one native call
per up to eight stacks of equally shaped matrices, and one fused kernel pair
for the final normalise-and-apply.
The global-norm clip factor is computed and consumed on the device, so the step
has no host synchronisation.
"""

from __future__ import annotations

import ctypes as C
from typing import Optional

import numpy as np
import torch
from torch.optim import Optimizer

from .. import _lib as L
from ..models.CELO2_MLP import CELO2MLP
from ..plan import (GradNorm, LoPlan, LoTensor, current_stream_ptr, fp32_gradient, grad_pointers, one_minus, tile_elems,
                    with_gradients)
from ._common import (FlatWeights, ItemPlan, factored_dims_argsort, group_floats, newton_schulz, newton_schulz_bounded,
                      newton_schulz_group_buffers, newton_schulz_native, newton_schulz_tc, optimizer_step, require_cuda_param)

_IN, _HID = 30, 8
_KEPT_FLOATS = 4 << 20  # elements up to which a plan keeps Newton-Schulz results and workspaces between steps


class _Celo2Family(Optimizer):
    _shared_adam = False
    _name = "CELO2_CUDA"

    def _setup(self, params, defaults, initial_momentum_decays, initial_rms_decays, initial_adafactor_decays,
               ns_coeffs, ns_iters, ns_eps, ff_hidden_size, ff_hidden_layers, hf_key, checkpoint_path, network):
        if not torch.cuda.is_available():
            raise RuntimeError(f"{self._name} requires a CUDA device.")
        self.device = torch.device("cuda")
        Optimizer.__init__(self, params, defaults)
        dev = self.device
        clamp = lambda xs: torch.clamp(torch.tensor(xs, dtype=torch.float32, device=dev), 0.0, 1.0)
        self.beta_m, self.beta_rms, self.beta_fac = clamp(initial_momentum_decays), clamp(initial_rms_decays), clamp(initial_adafactor_decays)
        self.n_mom, self.n_rms, self.n_fac = (int(b.shape[-1]) for b in (self.beta_m, self.beta_rms, self.beta_fac))
        if self.n_mom != 3 or self.n_fac != 3:
            raise ValueError(f"{self._name} kernels are built for 3 momentum and 3 adafactor decays")
        self.ns_coeffs = tuple(float(c) for c in ns_coeffs)
        self.ns_iters, self.ns_eps = ns_iters, ns_eps
        # weights: explicit network > local checkpoint > hub > random init (CELO2_cuda.py:141-155)
        if network is not None:
            self.network = network
        elif checkpoint_path is not None:
            self.network = CELO2MLP(hidden_size=ff_hidden_size, hidden_layers=ff_hidden_layers)
            self.network.load_state_dict(torch.load(checkpoint_path, map_location="cpu"))
        elif hf_key is not None:
            self.network = CELO2MLP.from_pretrained(hf_key)
        else:
            self.network = CELO2MLP(hidden_size=ff_hidden_size, hidden_layers=ff_hidden_layers)
        self.network = self.network.to(dev)
        if sum(self.network.feature_dims) != _IN:
            raise ValueError(f"{self._name} kernel expects feature_dims summing to {_IN}, got {sum(self.network.feature_dims)}.")
        if self.network.hidden_size != _HID or len(self.network.dense_w) != 2:
            raise ValueError(f"{self._name} kernel only supports ff_hidden_size=8, ff_hidden_layers=2.")
        self.w_in, self.b_in, self.w_h, self.b_h, self.w_out, self.b_out = (
            t.to(dev) for t in self.network.flat_weights())
        self._weights = FlatWeights((self.w_in, self.b_in, self.w_h, self.b_h, self.w_out, self.b_out), dev)   # the apply sweep's launch carries them
        self._plans = {}
        self._gnorm = None
        # "3xtf32" (default): the Newton-Schulz products on the tensor cores (this library's kernels, operands split
        # into a high and a low part of eleven bits each, as accurate as fp32 products); "fp32": torch.matmul, the
        # reference's arithmetic
        self.ns_precision = "3xtf32"
        #: Newton-Schulz launches of this library since construction (for the benchmark's launch count)
        self.extra_launches = 0
        self.process_group = None   # set (or set _sharded) when the tensors of the model are split over ranks
        self._sharded = False
        self.after_group = None     # optional callable(group index), called once a param group's kernels are enqueued
        self.before_group = None    # optional callable(group index), called before a param group's first kernel
        # fp32 values of 1 - beta, read back once (the reference evaluates them on the device every step)
        self._w_m, self._w_f = one_minus(self.beta_m), one_minus(self.beta_fac)
        self._w_v = float(1 - self.beta_rms[-1])
        self._prm = None   # the launch constants, made once
        self._b1_shared, self._b2_shared = float(self.beta_m[0]), float(self.beta_rms[-1])

    @property
    def _w_flat(self):
        return self._weights.flat

    # ------------------------------------------------------------------ state
    def _init_lo_state(self, state, p):
        shape = tuple(p.shape)
        dev = p.device
        state["mom"] = torch.zeros((self.n_mom,) + shape, device=dev)
        state["rms"] = torch.zeros(shape, device=dev)
        fd = factored_dims_argsort(shape)
        if fd is not None:
            dc, dr = fd
            r_shape, c_shape = list(shape), list(shape)
            r_shape[dr], c_shape[dc] = 1, 1
            state["fac_r"] = torch.zeros([self.n_fac] + r_shape, device=dev)
            state["fac_c"] = torch.zeros([self.n_fac] + c_shape, device=dev)

    def load_state_dict(self, state_dict):
        super().load_state_dict(state_dict)
        self._plans = {}

    def add_param_group(self, param_group):
        super().add_param_group(param_group)
        self._plans = {}

    # ------------------------------------------------------------------ planning
    def _build_group_plan(self, gi, group, plist):
        lo, adam = [], []
        for p in plist:
            require_cuda_param(p, self._name)
            st = self.state[p]
            is_1d = p.dim() <= 1 or group["is_embedding"]
            to_adam = group["use_adamw_for_1d"] and is_1d
            if self._shared_adam:
                if len(st) == 0:
                    self._init_lo_state(st, p)
            elif to_adam:
                if "exp_avg" not in st:
                    st["exp_avg"] = torch.zeros_like(p)
                    st["exp_avg_sq"] = torch.zeros_like(p)
                    st["adam_step"] = 0
            else:
                if p.dim() < 2:
                    raise ValueError(f"{self._name}: tensors with fewer than 2 dims need use_adamw_for_1d=True")
                if "mom" not in st:
                    self._init_lo_state(st, p)
            (adam if to_adam else lo).append(p)
        in_lo = [not (group["use_adamw_for_1d"] and (p.dim() <= 1 or group["is_embedding"])) for p in plist]
        plan = {"lo_params": lo, "adam_params": adam, "lo": None, "adam": None, "post": None, "in_lo": in_lo,
                "post_key": None, "adam_key": None}
        if lo:
            # raw-step buffers of equally shaped tensors are slices of one stacked tensor, so that
            # Newton-Schulz runs once per shape as a batched product instead of once per tensor
            by_shape = {}
            for ti, p in enumerate(lo):
                by_shape.setdefault(tuple(p.shape), []).append(ti)
            parts, out_of = [], {}
            for shape, members in by_shape.items():
                stacked = torch.empty((len(members),) + shape, dtype=torch.float32, device=self.device)
                # parts of at most ~64 M elements keep Newton-Schulz's temporaries small
                per = max(1, (64 << 20) // stacked[0].numel())
                parts += [(stacked[c0:c0 + per], members[c0:c0 + per]) for c0 in range(0, len(members), per)]
                for j, ti in enumerate(members):
                    out_of[ti] = stacked[j]
            # what goes into one native Newton-Schulz call: up to eight parts, up to ~96 M elements
            groups = []
            for part in parts:
                if not groups or len(groups[-1]["parts"]) == 8 or groups[-1]["floats"] + part[0].numel() > (96 << 20):
                    groups.append({"parts": [], "floats": 0, "kept": None})
                groups[-1]["parts"].append(part)
                groups[-1]["floats"] += part[0].numel()
            plan["ns_groups"] = groups
            tensors = []
            for ti, p in enumerate(lo):
                st = self.state[p]
                fd = factored_dims_argsort(tuple(p.shape))
                if fd is None:
                    raise ValueError(f"{self._name}: tensors with fewer than 2 dims need use_adamw_for_1d=True")
                tensors.append(LoTensor(
                    p=p.data, m=st["mom"], v=st["rms"], fac_r=st["fac_r"], fac_c=st["fac_c"], fdims=fd,
                    rcm_axis=fd[0] + 1, out=out_of[ti], w=self._w_flat, slice_last2=True))
            plan["lo"] = LoPlan(L.FAM_CELO2, tensors, self.device)
            # the tail works on matrices: the last two axes of every tensor
            post_sizes, post_owner = [], []
            for ti, p in enumerate(lo):
                mat = p.shape[-1] * p.shape[-2]
                for k in range(p.numel() // mat):
                    post_sizes.append(mat)
                    post_owner.append((ti, k * mat))
            post = ItemPlan(L.POST_DTYPE, post_sizes, self.device, tile_elems(sum(post_sizes), 1024, 4 * L.SM_COUNT))
            post.owner = post_owner
            post.owner_t = np.array([t for t, _ in post_owner], dtype=np.int64)
            post.owner_off = np.array([4 * o for _, o in post_owner], dtype=np.uint64)
            post.part = torch.zeros(max(post.n_tiles, 1), dtype=torch.float32, device=self.device)
            post.items["part"] = post.part.data_ptr() + 4 * post.items["tile0"].astype(np.uint64)
            plan["post"] = post
            base_p = np.array([p.data_ptr() for p in lo], dtype=np.uint64)
            post.items["p"][:] = base_p[post.owner_t] + post.owner_off
        if adam:
            sizes = [p.numel() for p in adam]
            plan["adam"] = ItemPlan(L.ADAM_DTYPE, sizes, self.device, tile_elems(sum(sizes), 1024, 4 * L.SM_COUNT))
            it = plan["adam"].items
            keys = ("mom", "rms") if self._shared_adam else ("exp_avg", "exp_avg_sq")
            plan["adam_states"] = [self.state[p] for p in adam]
            it["p"][:] = [p.data_ptr() for p in adam]
            it["m"][:] = [st[keys[0]].data_ptr() for st in plan["adam_states"]]
            it["v"][:] = [st[keys[1]].data_ptr() for st in plan["adam_states"]]
        return plan

    def _build_squares(self, plan):
        """Where the packed sweep takes every matrix, its items' sums of squares of the raw steps stand in for a launch that reads
        the steps again: (their buffer, first item and items of every matrix, what the table says otherwise); else None."""
        lo, items = plan["lo"], plan["post"].items
        if lo.sliced or lo.n_tiles_slow or lo.n_rtiles:
            return None
        owner = lo.ctiles.host["tensor"]   # ascending: the units in their order
        units = np.arange(len(plan["lo_params"]))
        first = np.searchsorted(owner, units)
        count = np.searchsorted(owner, units, side="right") - first
        buffer = torch.zeros(max(len(owner), 1), dtype=torch.float32, device=self.device)
        return (buffer, buffer.data_ptr() + 4 * first.astype(np.uint64), count.astype(np.int32),
                items["part"].copy(), items["n_tiles"].copy())

    def _params_struct(self, group, gnorm_ptr):
        prm = self._prm
        if prm is None:
            prm = self._prm = L.StepParams()
            prm.family = L.FAM_CELO2
            for k in range(3):
                prm.w_m[k], prm.w_f[k] = self._w_m[k], self._w_f[k]
            prm.w_v = self._w_v
            prm.eps_feat, prm.eps_norm = 1e-8, 1e-9
        prm.w_host = self._weights.host()
        prm.clip_val, prm.gnorm_sq = float(group["grad_clip_val"]), gnorm_ptr
        return prm

    def check_status(self):
        """Synchronise and raise if a kernel reported a wait that ran out (its output is incomplete)."""
        for _, plan in self._plans.values():
            if plan["lo"] is not None:
                plan["lo"].check_status()

    def clear_status(self):
        """Acknowledge a reported timeout: the next steps write parameters again."""
        for _, plan in self._plans.values():
            if plan["lo"] is not None:
                plan["lo"].clear_status()

    # ------------------------------------------------------------------ step
    @optimizer_step
    def step(self, loss=None):
        for _, plan in self._plans.values():
            if plan["lo"] is not None:
                plan["lo"].poll_status()
        stream = current_stream_ptr()
        gnorm_ptr = None
        if any(g["clip_grad"] for g in self.param_groups):
            all_p, all_g = with_gradients([p for g in self.param_groups for p in g["params"]])
            sig = [p.numel() for p in all_p]
            if self._gnorm is None or self._gnorm[0] != sig:
                self._gnorm = (sig, GradNorm(sig, self.device))
            total = self._gnorm[1].run(all_g, stream)
            if self.process_group is not None or (torch.distributed.is_initialized() and self._sharded):
                torch.distributed.all_reduce(total, group=self.process_group)  # each rank holds its own tensors' share
            gnorm_ptr = total.data_ptr()

        for gi, group in enumerate(self.param_groups):
            if self._shared_adam:
                # every group advances on every step, with or without gradients (ELO_CELO2_cuda.py:215-216)
                group["step"] = group.get("step", 0) + 1
            plist, grads = with_gradients(group["params"])
            if not plist:
                # a sharded step hangs collectives on this hook: every rank must reach it for every group, in order,
                # also a rank that owns nothing of the group
                if self.after_group is not None:
                    self.after_group(gi)
                continue
            sig = [p.data_ptr() for p in plist] + [bool(group["is_embedding"]), bool(group["use_adamw_for_1d"])]
            cached = self._plans.get(gi)
            if cached is None or cached[0] != sig:
                cached = (sig, self._build_group_plan(gi, group, plist))
                self._plans[gi] = cached
            plan = cached[1]
            if self.before_group is not None:
                self.before_group(gi)
            prm = self._params_struct(group, gnorm_ptr)
            clip_norm = float(group["clip_norm"]) if group["clip_grad"] else 0.0
            lr, wd = group_floats(group, "lr", "weight_decay")
            tail = ()   # what the matrices' last launch still has to do, where it waits for AdamW's
            if plan["lo"] is not None:
                tail = self._lo_step(group, plan, [g for g, lo in zip(grads, plan["in_lo"]) if lo], prm, clip_norm, lr, wd, stream)
            if plan["adam"] is not None:
                self._adam_step(group, plan, [g for g, lo in zip(grads, plan["in_lo"]) if not lo], prm, clip_norm, lr, stream, tail)
            if self.after_group is not None:
                self.after_group(gi)
        return loss


    def _lo_step(self, group, plan, grads, prm, clip_norm, lr, wd, stream):
        lo: LoPlan = plan["lo"]
        exp_mult, rmsmult = group_floats(group, "exp_mult", "rmsmult")
        lo.set_hyper(lr=lr, wd=wd, clip_norm=clip_norm, exp_mult=exp_mult)
        lo.refresh(grads)
        squares = None
        if not group["orthogonalize"]:   # steps that are orthogonalised have other squares: their groups need none of it
            if "squares" not in plan:
                plan["squares"] = self._build_squares(plan)
            squares = plan["squares"]
        prm.step_squares = squares[0].data_ptr() if squares else None
        lo.run(prm, stream)
        prm.step_squares = None
        post: ItemPlan = plan["post"]
        keep = [t.out for t in lo.tensors]
        if group["orthogonalize"]:
            keep, steps = self._orthogonalise(plan, stream)
        else:
            steps = [k.data_ptr() for k in keep]
        key = (steps, lr, wd, rmsmult, squares is not None)
        if key != plan["post_key"]:
            it = post.items
            it["step"][:] = np.array(steps, dtype=np.uint64)[post.owner_t] + post.owner_off
            it["lr"][:], it["wd"][:], it["rmsmult"][:] = lr, wd, rmsmult
            if plan.get("squares"):
                it["part"][:], it["n_tiles"][:] = plan["squares"][1:3] if squares else plan["squares"][3:5]
            post.upload()
            plan["post_key"] = key
        if not squares:
            L.check(L.lib.pylo_b200_celo2_post_sums(post.table.ptr, post.tiles.ptr, post.n_tiles, stream), "celo2_post_sums")
        self._keep = keep
        tail = (post.table.ptr, post.tiles.ptr, post.n_tiles, lo.step_plan.status, lo.step_plan.host_status)
        if plan["adam"] is not None and post.n_tiles + plan["adam"].n_tiles <= L.TAIL_ONE_LAUNCH:
            return tail
        L.check(L.lib.pylo_b200_celo2_post_apply(*tail, stream), "celo2_post_apply")
        return ()

    def _orthogonalise(self, plan, stream):
        """Newton-Schulz over the plan's stacks of raw steps: (the results to keep alive, address of every tensor's)."""
        keep, steps = [], [0] * len(plan["lo_params"])
        status = plan["lo"].status   # the products OR 4 in if one of their bounded waits ran out
        native = self.ns_precision == "3xtf32" and newton_schulz_bounded(self.ns_coeffs, self.ns_iters)
        for group in plan["ns_groups"]:
            results = group["kept"]
            if native:
                if results is None:
                    results = newton_schulz_group_buffers([part for part, _ in group["parts"]], self.ns_iters)
                    if group["floats"] <= _KEPT_FLOATS:
                        # small models: results and workspaces stay with the plan; large ones take them from the allocator
                        # on every step, so that the training step can have the memory in between
                        group["kept"] = results
                launches = newton_schulz_native([part for part, _ in group["parts"]], [r for r, _ in results], [w for _, w in results],
                                                self.ns_coeffs, self.ns_iters, self.ns_eps, status, stream)
                outs = [r for r, _ in results]
            else:
                args = (self.ns_coeffs, self.ns_iters, self.ns_eps)
                outs = [(newton_schulz_tc(part, *args, status, stream) if self.ns_precision == "3xtf32"
                         else newton_schulz(part, *args)).contiguous() for part, _ in group["parts"]]
                launches = 3 * self.ns_iters
            if self.ns_precision == "3xtf32":
                self.extra_launches += launches
            keep += outs
            for res, (part, members) in zip(outs, group["parts"]):
                at, n = res.data_ptr(), 4 * part[0].numel()
                for j, ti in enumerate(members):
                    steps[ti] = at + n * j
        return keep, steps

    def _adam_step(self, group, plan, grads, prm, clip_norm, lr, stream, tail=()):
        adam: ItemPlan = plan["adam"]
        it = adam.items
        ptrs = grad_pointers(grads)
        copies = []
        if ptrs is None:   # a gradient that is not contiguous fp32 is copied, which gives it a new address on every step
            copies = [fp32_gradient(g) for g in grads]
            ptrs = [g.data_ptr() for g in copies]
        if self._shared_adam:
            b1, b2, eps = self._b1_shared, self._b2_shared, 1e-8
            ts = [group["step"]]
        else:
            b1, b2, eps = self.adam_beta1, self.adam_beta2, self.adam_eps
            for st in plan["adam_states"]:
                st["adam_step"] += 1
            ts = [st["adam_step"] for st in plan["adam_states"]]
        same = min(ts) == max(ts)   # one step count: the bias corrections go with the launch, not through the table
        adam_lr_mult, adam_wd = group_floats(group, "adam_lr_mult", "adam_weight_decay")
        key = (ptrs, adam_lr_mult * lr, adam_wd, clip_norm)
        if key != plan["adam_key"] or not same:
            it["g"][:] = ptrs
            it["lr"][:], it["wd"][:], it["clip_norm"][:] = key[1:]
            it["bc1"][:], it["bc2"][:] = [1.0 - b1 ** t for t in ts], [1.0 - b2 ** t for t in ts]
            adam.upload()
            plan["adam_key"] = key
        bc1, bc2 = (1.0 - b1 ** ts[0], 1.0 - b2 ** ts[0]) if same else (0.0, 0.0)
        launch = L.lib.pylo_b200_celo2_tail if tail else L.lib.pylo_b200_adamw
        L.check(launch(*tail, adam.table.ptr, adam.tiles.ptr, adam.n_tiles, int(not self._shared_adam),
                       b1, 1 - b1, b2, 1 - b2, eps, bc1, bc2, C.byref(prm), stream), "adamw")
        self._keepg = copies


class CELO2_CUDA(_Celo2Family):
    """CELO2 learned optimizer; 1-D / embedding tensors take an AdamW step with their own moments."""

    _shared_adam = False
    _name = "CELO2_CUDA"

    def __init__(self, params, lr=1e-3, weight_decay=0.0, adam_lr_mult=1.0, adam_weight_decay=None,
                 adam_betas=(0.9, 0.95), adam_eps=1e-8, use_adamw_for_1d=True, orthogonalize=True, clip_grad=False,
                 clip_norm=1.0, ff_hidden_size=8, ff_hidden_layers=2, initial_momentum_decays=(0.9, 0.99, 0.999),
                 initial_rms_decays=(0.95,), initial_adafactor_decays=(0.9, 0.99, 0.999), exp_mult=0.0, rmsmult=1.0,
                 param_scale_mult=False, ns_coeffs=(3.4445, -4.7750, 2.0315), ns_iters=5, ns_eps=1e-8,
                 grad_clip_val=1000.0, hf_key: Optional[str] = "DiamondXL/celo2",
                 checkpoint_path: Optional[str] = None, network: Optional[CELO2MLP] = None, ns_precision: str = "3xtf32"):
        defaults = dict(
            lr=lr, weight_decay=weight_decay, adam_lr_mult=adam_lr_mult,
            adam_weight_decay=(adam_weight_decay if adam_weight_decay is not None else weight_decay),
            use_adamw_for_1d=use_adamw_for_1d, orthogonalize=orthogonalize, clip_grad=clip_grad, clip_norm=clip_norm,
            exp_mult=exp_mult, rmsmult=rmsmult, param_scale_mult=param_scale_mult, grad_clip_val=grad_clip_val,
            is_embedding=False)
        self.adam_beta1, self.adam_beta2 = (float(b) for b in adam_betas)
        self.adam_eps = adam_eps
        self._setup(params, defaults, initial_momentum_decays, initial_rms_decays, initial_adafactor_decays,
                    ns_coeffs, ns_iters, ns_eps, ff_hidden_size, ff_hidden_layers, hf_key, checkpoint_path, network)
        if ns_precision not in ("fp32", "3xtf32"):
            raise ValueError("ns_precision must be 'fp32' or '3xtf32'")
        self.ns_precision = ns_precision


class ELO_CELO2_CUDA(_Celo2Family):
    """ELO-CELO2: CELO2 forward with ELO defaults; the AdamW branch reuses mom[0] / rms of every tensor."""

    _shared_adam = True
    _name = "ELO_CELO2_CUDA"

    def __init__(self, params, lr=1e-3, weight_decay=0.1, clip_grad=True, clip_norm=1.0, adam_lr_mult=20.0,
                 adam_weight_decay=None, use_adamw_for_1d=True, orthogonalize=True, ff_hidden_size=8,
                 ff_hidden_layers=2, initial_momentum_decays=(0.9, 0.99, 0.999), initial_rms_decays=(0.95,),
                 initial_adafactor_decays=(0.9, 0.99, 0.999), exp_mult=0.0, rmsmult=1.0, param_scale_mult=False,
                 ns_coeffs=(3.4445, -4.7750, 2.0315), ns_iters=5, ns_eps=1e-8, grad_clip_val=1000.0,
                 hf_key: Optional[str] = "DiamondXL/elo-celo2", checkpoint_path: Optional[str] = None,
                 network: Optional[CELO2MLP] = None, ns_precision: str = "3xtf32"):
        defaults = dict(
            lr=lr, weight_decay=weight_decay, adam_lr_mult=adam_lr_mult,
            adam_weight_decay=(adam_weight_decay if adam_weight_decay is not None else weight_decay),
            use_adamw_for_1d=use_adamw_for_1d, orthogonalize=orthogonalize, clip_grad=clip_grad, clip_norm=clip_norm,
            exp_mult=exp_mult, rmsmult=rmsmult, param_scale_mult=param_scale_mult, grad_clip_val=grad_clip_val,
            is_embedding=False)
        self._setup(params, defaults, initial_momentum_decays, initial_rms_decays, initial_adafactor_decays,
                    ns_coeffs, ns_iters, ns_eps, ff_hidden_size, ff_hidden_layers, hf_key, checkpoint_path, network)
        if ns_precision not in ("fp32", "3xtf32"):
            raise ValueError("ns_precision must be 'fp32' or '3xtf32'")
        self.ns_precision = ns_precision
