"""Tensor-core field MLP (nsvf_mlp_forward_bf16) for the StandInField weights.

TensorCoreMLP(field) snapshots the field's weights as bf16 (row-major
[out, in]) and biases as FP32 on the field's device; calling it on an FP32
embedding [N, 32] returns [N, 4] = (sigma, r, g, b) in FP32.

It also keeps the FP32 weights transposed for nsvf_field_exact_dev, the
double-float re-evaluation of samples far outside their voxel.

enable_fp8(calibration_emb) adds the FP8 option of the fused sample kernel
(nsvf_field_samples_fp8): the three 128x128 hidden layers in E4M3 with
per-layer scales, the input layer and the (sigma, rgb) head in BF16.
"""
import ctypes
import math

import torch

from . import ext
from ._lib import LIB, check


class TensorCoreMLP:
    def __init__(self, field):
        dims = [(lin.out_features, lin.in_features) for lin in field.layers]
        if dims != [(128, 32), (128, 128), (128, 128), (128, 128), (4, 128)]:
            raise ValueError("tensor-core MLP supports the 32-128x4-4 field, got %s" % dims)
        self.w = [lin.weight.detach().to(torch.bfloat16).contiguous() for lin in field.layers]
        self.b = [lin.bias.detach().float().contiguous() for lin in field.layers]
        self.device = self.w[0].device
        self._wp = (ctypes.c_void_p * 5)(*[t.data_ptr() for t in self.w])
        self._bp = (ctypes.c_void_p * 5)(*[t.data_ptr() for t in self.b])
        # biases of the BF16 kernels: the field's, until calibrate_bias
        # corrects them for the BF16 rounding of the weights
        self.b_tc = [t.clone() for t in self.b]
        self._bp_tc = (ctypes.c_void_p * 5)(*[t.data_ptr() for t in self.b_tc])
        self.w32 = [lin.weight.detach().float().contiguous() for lin in field.layers]
        # transposed FP32 copies ([in, out]) for the compensated pass over
        # samples far outside their voxel (nsvf_field_exact_dev)
        self.wt32 = [w.t().contiguous() for w in self.w32]
        self._wtp = (ctypes.c_void_p * 5)(*[t.data_ptr() for t in self.wt32])
        # the same copies as [out, in], for pruning's FP32 stage
        self.wc32 = [t.t().contiguous() for t in self.wt32]
        self._wcp = (ctypes.c_void_p * 5)(*[t.data_ptr() for t in self.wc32])
        self.fp8 = None

    E4M3_MAX = 448.0

    @torch.no_grad()
    def calibrate_bias(self, calibration_emb):
        """Bias correction for the BF16 kernels: rounding the weights to bf16
        shifts each layer's output by (bf16(W) - W) x, an error that is the
        same for neighbouring samples and so adds up along a ray. Layer by
        layer, through the BF16 network on `calibration_emb` [N, 32] (FP32
        embeddings of points inside the scene's voxels), the mean of that
        shift over the calibration inputs is subtracted from the layer's bias
        (in float64, stored in FP32). The FP32 and double-float passes keep the
        field's own biases."""
        x = calibration_emb.float().to(torch.bfloat16).float()
        for l in range(5):
            W32 = self.w32[l].double()
            dW = self.w[l].double() - W32
            shift = dW @ x.double().mean(0)
            self.b_tc[l].copy_((self.b[l].double() - shift).float())
            x = x @ self.w[l].float().t() + self.b_tc[l]
            if l < 4:
                x = torch.relu(x).to(torch.bfloat16).float()
        return self

    def enable_fp8(self, calibration_emb):
        """Per-layer scales for E4M3 hidden layers. Weights: w_scale[l] =
        448 / max|W_l|. Activations: a_scale[l] = 448 / (max of the FP32
        activation entering layer l on `calibration_emb` [N, 32]); larger
        values saturate to 448 at run time."""
        x = calibration_emb.float()
        amax = []
        with torch.no_grad():
            for i in range(3):
                x = torch.relu(x @ self.w32[i].t() + self.b[i])
                amax.append(float(x.abs().max()))
        w_scale = [self.E4M3_MAX / max(float(self.w32[l].abs().max()), 1e-30) for l in (1, 2, 3)]
        a_scale = [self.E4M3_MAX / max(a, 1e-30) for a in amax]
        w8 = [(self.w32[l] * s).clamp(-self.E4M3_MAX, self.E4M3_MAX).to(torch.float8_e4m3fn)
              .contiguous() for l, s in zip((1, 2, 3), w_scale)]
        ptrs = [self.w[0].data_ptr()] + [t.data_ptr() for t in w8] + [self.w[4].data_ptr()]
        self.fp8 = {"w8": w8, "w_scale": w_scale, "a_scale": a_scale,
                    "wp": (ctypes.c_void_p * 5)(*ptrs),
                    "scales": (ctypes.c_float * 6)(*(w_scale + a_scale))}
        return self

    def __call__(self, emb, out=None):
        emb = emb.float().contiguous()
        n = emb.shape[0]
        if out is None:
            out = torch.empty(n, 4, dtype=torch.float32, device=emb.device)
        with ext._timed("mlp_forward_bf16", emb.device):
            check(LIB.nsvf_mlp_forward_bf16(n, emb.data_ptr(), self._wp, self._bp_tc, out.data_ptr(),
                                            ext.error_word(emb.device).data_ptr(),
                                            ext.ctypes_stream(emb.device)), "mlp_forward_bf16")
        return out

    def field_samples(self, voxel, xyz_dist, centers, feats, values, voxel_size, out=None):
        """Fused interpolation + MLP on compacted samples: voxel [n] int32,
        xyz_dist [n, 4], centers [V, 3], feats [V, 8] int32, values [Kc, 32]
        -> [n, 4] (sigma, r, g, b)."""
        n = voxel.numel()
        dev = voxel.device
        if out is None:
            out = torch.empty(n, 4, dtype=torch.float32, device=dev)
        with ext._timed("field_samples_bf16", dev):
            check(LIB.nsvf_field_samples_bf16(
                n, voxel.data_ptr(), xyz_dist.data_ptr(), centers.size(0), values.size(0),
                float(voxel_size), centers.data_ptr(), feats.data_ptr(), values.data_ptr(),
                self._wp, self._bp_tc, out.data_ptr(), ext.error_word(dev).data_ptr(),
                ext.ctypes_stream(dev)), "field_samples_bf16")
        return out

    def field_samples_fp8(self, voxel, xyz_dist, centers, feats, values, voxel_size, out=None):
        """field_samples with E4M3 hidden layers (enable_fp8 first)."""
        if self.fp8 is None:
            raise RuntimeError("TensorCoreMLP.enable_fp8 has not been called")
        n = voxel.numel()
        dev = voxel.device
        if out is None:
            out = torch.empty(n, 4, dtype=torch.float32, device=dev)
        with ext._timed("field_samples_fp8", dev):
            check(LIB.nsvf_field_samples_fp8(
                n, voxel.data_ptr(), xyz_dist.data_ptr(), centers.size(0), values.size(0),
                float(voxel_size), centers.data_ptr(), feats.data_ptr(), values.data_ptr(),
                self.fp8["wp"], self._bp, self.fp8["scales"], out.data_ptr(),
                ext.error_word(dev).data_ptr(), ext.ctypes_stream(dev)), "field_samples_fp8")
        return out

    def prune_scores(self, centers, feats, values, voxel_size, bits=8, rule=1, step=0.0):
        """Per-voxel pruning score over bits^3 points (see nsvf_prune_scores_bf16):
        rule 0 -> min exp(-relu sigma), rule 1 -> max 1 - exp(-relu(sigma) step)."""
        V = centers.size(0)
        dev = centers.device
        init = 0x7F800000 if rule == 0 else 0
        score = torch.full((V,), init, dtype=torch.int32, device=dev)
        with ext._timed("prune_scores_bf16", dev):
            check(LIB.nsvf_prune_scores_bf16(
                V, int(bits), int(rule), float(step), values.size(0), float(voxel_size),
                centers.data_ptr(), feats.data_ptr(), values.data_ptr(), self._wp, self._bp,
                score.data_ptr(), ext.error_word(dev).data_ptr(), ext.ctypes_stream(dev)),
                "prune_scores_bf16")
        return score.view(torch.float32)

    # Screen band of the exact pruning pass, in units of M = sum_j |W4[0][j]| h_j:
    # the BF16 error of sigma measured on the workloads' fields stays below
    # 0.005 M (c2 pruning field, 768k points), so 0.02 leaves a factor 4.
    PRUNE_BAND = 0.02

    # The FP32 pass's band is PRUNE_BAND / 64 (nsvf_prune_fp32_dev), 3.1e-4 M:
    # FP32's error of sigma is at most 3.4e-7 M and BF16's 6.5e-3 M (twelve shell
    # and ball fields of 24,000 to 4 M points), so where the screen's band holds,
    # this one does. Up to FP32_FROM points go to double-float at once: these
    # take less than the launches and buffers before them.
    FP32_BAND = 64.0
    FP32_FROM = 512

    def prune_mask(self, centers, feats, values, voxel_size, th=0.5, bits=8, rule=1, step=0.0,
                   band=PRUNE_BAND, scores=True):
        """Exact pruning mask [V] (bool) for 0 < th < 1: rule 0 (the
        reference's, fairnr/modules/encoder.py:609-610) keeps voxels with
        1 - min exp(-relu sigma) > th, rule 1 those with max 1 - exp(-relu(sigma)
        step) >= th, sigma at bits^3 offset_points positions per voxel. The
        tensor-core pass screens every point in BF16 and decides all but the
        points within `band` M of the threshold. Those of voxels not kept yet
        are evaluated in FP32 with a band of `band` / FP32_BAND, and what that
        leaves in double-float (nsvf_prune_screen_bf16, nsvf_prune_fp32_dev,
        nsvf_prune_exact_dev). Also returns the BF16 scores (as prune_scores)
        and the number of points that the BF16 pass left undecided. With
        scores=False (the second result is then None) the BF16 pass first
        takes a few points of every voxel and then all points of the voxels
        that those do not keep; the number is then of the points it left
        undecided there, each counted once."""
        if not 0.0 < th < 1.0:
            raise ValueError("pruning threshold must lie in (0, 1), got %r" % (th,))
        if rule == 1 and not step > 0.0:
            raise ValueError("rule 1 needs a positive step")
        T = -math.log1p(-th) / (step if rule == 1 else 1.0)
        V = centers.size(0)
        dev = centers.device
        init = 0x7F800000 if rule == 0 else 0
        score = torch.empty(V, dtype=torch.int32, device=dev) if scores else None
        keep = torch.empty(V, dtype=torch.uint8, device=dev)
        n_list = torch.empty(1, dtype=torch.int64, device=dev)
        err = ext.error_word(dev)
        stream = ext.ctypes_stream(dev)
        # room for 3 % of the points (1.65 % of the c2 pass are undecided): a
        # second screen pass (7.5 ms there) costs more than the list
        cap = max(65536, V * bits ** 3 // 32)
        # The points of the first pass, per axis: at most 1.6 % of them (on
        # the c2 pass the corners keep 66 % of the voxels that are kept, and
        # 4 points per axis 87 %)
        sub = 4 if bits >= 12 else 2
        live = torch.empty(V, dtype=torch.int32, device=dev) if not scores else None
        n_live = torch.zeros(1, dtype=torch.int64, device=dev) if not scores else None
        common = (values.size(0), float(voxel_size), centers.data_ptr(), feats.data_ptr(),
                  values.data_ptr(), self._wp, self._bp)
        for _ in range(3):
            lst = torch.empty(cap, dtype=torch.int64, device=dev)
            keep.zero_()
            n_list.zero_()
            with ext._timed("prune_screen_bf16", dev):
                if scores:
                    score.fill_(init)
                    check(LIB.nsvf_prune_screen_bf16(
                        V, int(bits), int(rule), float(step), float(T), float(band), *common,
                        score.data_ptr(), keep.data_ptr(), lst.data_ptr(), n_list.data_ptr(), cap,
                        None, stream), "prune_screen_bf16")
                else:
                    for g, lv, nl in ((sub, None, None), (bits, live, n_live)):
                        if lv is None and bits < 4:
                            continue
                        # the first pass lists nothing (the second one goes
                        # over its points again) and counts into n_live, which
                        # the second one sets anew
                        out = (lv.data_ptr(), nl.data_ptr(), lst.data_ptr(), n_list.data_ptr(),
                               cap) if lv is not None else (None, None, None, n_live.data_ptr(), 0)
                        check(LIB.nsvf_prune_screen_live_bf16(
                            V, int(bits), int(g), int(rule), float(T), float(band), *common,
                            keep.data_ptr(), *out, None, stream), "prune_screen_live_bf16")
            n = int(n_list.item())
            if n <= cap:
                break
            cap = n + n // 4
        # double-float costs about 60 times FP32 a point (131 against 2.2 us per
        # thousand), so FP32 decides what it can first: the c2 pass's 23.0 ms
        # of double-float become 0.39 ms of FP32 and 0.07 ms
        if n > self.FP32_FROM and band > 0.0 and 1e-30 < T < 1e30:
            # (the weights of the double-float pass)
            packed = torch.empty(int(LIB.nsvf_field_train_packed_floats()), dtype=torch.float32,
                                 device=dev)
            check(LIB.nsvf_field_train_pack(self._wcp, self._bp, packed.data_ptr(), stream),
                  "field_train_pack")
            live = torch.empty(cap, dtype=torch.int64, device=dev)
            n_live = torch.zeros(1, dtype=torch.int64, device=dev)
            n_listed, n_list = n_list, torch.zeros(1, dtype=torch.int64, device=dev)
            with ext._timed("prune_fp32", dev):
                check(LIB.nsvf_prune_fp32_dev(
                    V, int(bits), float(T), float(band) / self.FP32_BAND, values.size(0),
                    float(voxel_size), centers.data_ptr(), feats.data_ptr(), values.data_ptr(),
                    packed.data_ptr(), lst.data_ptr(), n_listed.data_ptr(), cap,
                    keep.data_ptr(), live.data_ptr(), n_live.data_ptr(), lst.data_ptr(),
                    n_list.data_ptr(), stream), "prune_fp32_dev")
        with ext._timed("prune_exact", dev):
            check(LIB.nsvf_prune_exact_dev(
                V, int(bits), int(rule), float(T), values.size(0), float(voxel_size),
                centers.data_ptr(), feats.data_ptr(), values.data_ptr(), self._wtp, self._bp,
                lst.data_ptr(), n_list.data_ptr(), cap, keep.data_ptr(), err.data_ptr(),
                ext.ctypes_stream(dev)), "prune_exact_dev")
        return keep.bool(), score.view(torch.float32) if scores else None, n

    def reference_bf16(self, emb):
        """torch emulation of the kernel's rounding: bf16 operands, FP32 sums
        (with the BF16 kernels' biases, b_tc)."""
        x = emb.float().to(torch.bfloat16).float()
        for i, (W, b) in enumerate(zip(self.w, self.b_tc)):
            x = x @ W.float().t() + b
            if i < 4:
                x = torch.relu(x).to(torch.bfloat16).float()
        return x

    def reference_fp8(self, emb):
        """torch emulation of the FP8 kernel: bf16 input layer; the
        accumulator of layer l starts at bias / dq (dq = 1 / (a_scale *
        w_scale) of the layer, 1 for layer 0; float32 scalars as the library
        computes them); for layers 0-2 the output relu(acc * dq * qs) (qs =
        a_scale of the next layer) rounded to saturating E4M3, E4M3 weights;
        layer 3 relu(acc * dq) in bf16; bf16 head."""
        import numpy as np
        f = self.fp8
        f32 = np.float32
        e4 = torch.float8_e4m3fn
        ws = [f32(x) for x in f["w_scale"]]
        as_ = [f32(x) for x in f["a_scale"]]
        dq = [f32(1.0)] + [f32(f32(1.0) / f32(ws[l - 1] * as_[l - 1])) for l in (1, 2, 3)]
        qs = as_ + [f32(1.0)]
        x = emb.float().to(torch.bfloat16).float() @ self.w[0].float().t()
        for l in range(4):
            z = x + self.b[l].float() / float(dq[l])
            if l < 3:
                y = z * float(f32(dq[l] * qs[l]))
                x = torch.relu(y).clamp(max=self.E4M3_MAX).to(e4).float()
                x = x @ f["w8"][l].float().t()
            else:
                x = torch.relu(z * float(dq[3])).to(torch.bfloat16).float()
        return x @ self.w[4].float().t() + self.b[4]
