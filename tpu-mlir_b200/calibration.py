"""Activation calibration on the GPU: running min/max, streaming histogram and KLD threshold per tensor.

Mirrors the statistics half of the reference's ``ActivationCalibrator``
(python/calibration/kld_calibrator.py:364-477 ``process_statistic``, :321-347 ``find_threshold``) and its math
object (python/calibration/cali_math.py:27-143).  Two things differ in form, not in result:

* ``CaliMathB200`` offers the reference's ``prepare / histogram / combine_histogram`` protocol, computed by the
  kernels in libb200q.so.
* ``ShardedCalibrator`` runs the same statistics over samples that are sharded across ranks.  The reference's
  streaming histogram depends on the sample order only through the running abs-max (cali_math.py:82-103 keeps
  old counts in their bins when it grows the histogram), so it equals the sum over samples of per-sample
  histograms taken with a (threshold, bins) schedule derived from the per-sample min/max alone.  Pass 1 gathers
  the min/max of every sample (all-gather), every rank derives the identical schedule on the host, pass 2
  histograms the local samples into a buffer of the final size, one all-reduce (sum, int32) merges the ranks.
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass
from typing import Callable, Dict, Iterable, List, Optional, Sequence

import numpy as np

from . import _lib as L

MAX_GROWN_BINS = 8000000   # cali_math.py:96
MAX_KLD_BINS = 64 * 2048   # kld_calibrator.py:338
ALL_ZERO_EPS = 1e-8        # kld_calibrator.py:395


# ----------------------------------------------------------------------------------------------- host logic
@dataclass
class Schedule:
    """What each sample contributes to one tensor's histogram, and the final histogram geometry."""
    th: np.ndarray          # float32 [S] threshold used for sample s (0 where it contributes nothing)
    nbins: np.ndarray       # int32 [S] bins used for sample s (0 = skipped)
    final_bins: int         # length of the final histogram (0 if no sample contributed)
    width: np.float32       # bin width handed to the KLD search
    min: np.float32
    max: np.float32
    abs_max: np.float32


def bin_schedule(sample_min: Sequence[float], sample_max: Sequence[float], bin_num: int = 2048) -> Schedule:
    """Replays process_statistic + combine_histogram (kld_calibrator.py:391-398,:462-476; cali_math.py:82-103)
    on the per-sample (min, max) of one tensor, in sample order, in float32 like the reference."""
    smin = np.asarray(sample_min, dtype=np.float32)
    smax = np.asarray(sample_max, dtype=np.float32)
    S = len(smin)
    th_s = np.zeros(S, np.float32)
    nb_s = np.zeros(S, np.int32)
    run_min, run_max = float("inf"), float("-inf")
    th: Optional[np.float32] = None
    nb = 0
    width = np.float32(0)
    last_reset = 0
    for i in range(S):
        run_min = min(smin[i], run_min)
        run_max = max(smax[i], run_max)
        abs_value = max(abs(run_min), abs(run_max))
        if max(abs(smin[i]), abs(smax[i])) < ALL_ZERO_EPS:      # np.abs(activation).max() < 1e-8: no histogram
            continue
        if th is None:
            th, nb = np.float32(abs_value), bin_num
            width = np.float32(th / (nb - 1))
        elif abs_value > th:
            old_step = np.float32(th / nb)
            inc = int((np.float32(abs_value) - th) // old_step + 1)
            if inc + nb > MAX_GROWN_BINS:
                th, nb = np.float32(abs_value), bin_num          # starts over with this sample only
                last_reset = i
            else:
                th = np.float32(inc * old_step + th)
                nb = inc + nb
            width = np.float32(th / (nb - 1))
        th_s[i], nb_s[i] = th, nb
    nb_s[:last_reset] = 0
    th_s[:last_reset] = 0
    amax = np.float32(max(abs(run_min), abs(run_max))) if S else np.float32(0)
    return Schedule(th=th_s, nbins=nb_s, final_bins=int(nb), width=np.float32(width), min=np.float32(run_min),
                    max=np.float32(run_max), abs_max=amax)


# b200q_bin_state: the recurrence's state of one tensor
_BIN_STATE = np.dtype([("min", np.float32), ("max", np.float32), ("th", np.float32), ("width", np.float32), ("bins", np.int64),
                       ("last_reset", np.int64), ("started", np.int64)])


class BinScheduler:
    """``bin_schedule`` for T tensors at once, fed with any number of samples at a time (native code, identical results)."""

    def __init__(self, tensors: int, bin_num: int = 2048):
        self.bin_num, self.samples = bin_num, 0
        self.state = np.zeros(tensors, _BIN_STATE)
        self.state["min"], self.state["max"] = np.inf, -np.inf

    def advance(self, minmax: np.ndarray):
        """``minmax`` float32 [T, S, 2] of the next S samples -> their (threshold, bins), float32 / int32 [T, S].  Where
        ``state["last_reset"]`` moved into these samples, everything counted for earlier ones is void."""
        mm = np.ascontiguousarray(minmax, dtype=np.float32)
        T, S = mm.shape[:2]
        th, nb = np.empty((T, S), np.float32), np.empty((T, S), np.int32)
        L.check(L.lib().b200q_calib_bin_schedule(self.state.ctypes.data, T, S, mm.ctypes.data, self.samples, self.bin_num, MAX_GROWN_BINS,
                                                 th.ctypes.data, nb.ctypes.data))
        self.samples += S
        return th, nb


def bin_schedule_many(sample_min: np.ndarray, sample_max: np.ndarray, bin_num: int = 2048) -> List[Schedule]:
    """``bin_schedule`` for T tensors at once: ``sample_min / sample_max`` are float32 [T, S], the results are identical
    to the scalar form (tested)."""
    T, S = np.shape(sample_min)
    bs = BinScheduler(T, bin_num)
    th, nb = bs.advance(np.stack([sample_min, sample_max], axis=2))
    st = bs.state
    amax = np.maximum(np.abs(st["min"]), np.abs(st["max"])) if S else np.zeros(T, np.float32)
    return [Schedule(th=th[t], nbins=nb[t], final_bins=int(st["bins"][t]), width=st["width"][t], min=st["min"][t], max=st["max"][t],
                     abs_max=np.float32(amax[t])) for t in range(T)]


def table_threshold(kl: float, abs_max: float) -> float:
    """calibration_result.canonicalize (python/calibration/utils.py:53-69) and the 1e-5 floor of
    dump_cali_table (kld_calibrator.py:848-851)."""
    th = min(float(kl), float(abs_max))
    return th if th > 1e-5 else 1e-5


# ----------------------------------------------------------------------------------------------- GPU math
class CaliMathB200:
    """The reference's math_impl protocol (cali_math.py:27-143: prepare / histogram / combine_histogram) on the
    GPU.  Arrays passed to ``prepare`` stay on the device; histograms come back as int32 numpy arrays."""

    def __init__(self, device: Optional[int] = None):
        import torch
        self.torch = torch
        if not torch.cuda.is_available():
            raise L.B200QError(L.ERR_NO_DEVICE, "CaliMathB200 needs a CUDA device (there is no CPU fallback)")
        self.device = torch.device("cuda", torch.cuda.current_device() if device is None else device)
        self.ctx = C.c_void_p()
        L.check(L.lib().b200q_calib_create(C.byref(self.ctx)))

    def __del__(self):
        try:
            if self.ctx:
                L.lib().b200q_calib_destroy(C.byref(self.ctx))
        except Exception:
            pass

    # -- device helpers
    def _dev(self, a):
        t = self.torch
        if isinstance(a, t.Tensor):
            if a.dtype is t.float32 and a.device == self.device and a.is_contiguous():
                return a
            return a.to(self.device, dtype=t.float32).contiguous()
        return t.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(self.device)

    def _stream(self):
        return C.c_void_p(self.torch.cuda.current_stream(self.device).cuda_stream)

    def prepare(self, array):
        return self._dev(array)

    def minmax(self, x, samples: int = 1):
        """Per-sample (min, max) of a device tensor viewed as [samples, -1]; returns a device tensor [samples, 2]."""
        x = self._dev(x)
        n = x.numel() // samples
        out = self.torch.empty((samples, 2), dtype=self.torch.float32, device=self.device)
        L.check(L.lib().b200q_calib_minmax(self.ctx, C.c_void_p(x.data_ptr()), n, samples,
                                           C.c_void_p(out.data_ptr()), self._stream()))
        return out

    def histogram_into(self, hist, x, th: np.ndarray, nbins: np.ndarray):
        """hist (device int32) += per-sample histograms of x viewed as [len(th), -1]."""
        x = self._dev(x)
        S = len(th)
        th = np.ascontiguousarray(th, dtype=np.float32)
        nbins = np.ascontiguousarray(nbins, dtype=np.int32)
        L.check(L.lib().b200q_calib_histogram(self.ctx, C.c_void_p(x.data_ptr()), x.numel() // S, S,
                                              th.ctypes.data_as(C.POINTER(C.c_float)),
                                              nbins.ctypes.data_as(C.POINTER(C.c_int32)),
                                              C.c_void_p(hist.data_ptr()), hist.numel(), self._stream()))

    def _tensors(self, xs, samples):
        """Pointer and per-sample size arrays of device tensors viewed as [samples, -1]."""
        return (np.fromiter((x.data_ptr() for x in xs), np.uint64, len(xs)),
                np.fromiter((x.numel() // samples for x in xs), np.int64, len(xs)))

    def minmax_many(self, xs, samples: int) -> np.ndarray:
        """``minmax`` of many device tensors with one launch; float32 [T, samples, 2] on the host."""
        p, n = self._tensors(xs, samples)
        out = np.empty((len(xs), samples, 2), np.float32)
        L.check(L.lib().b200q_calib_minmax_many(self.ctx, len(xs), p.ctypes.data, n.ctypes.data, samples, out.ctypes.data, self._stream()))
        return out

    def histogram_many_into(self, hists, xs, th: np.ndarray, nbins: np.ndarray):
        """``histogram_into`` for many device tensors with one launch: ``hists`` is (addresses, lengths), th / nbins [T, samples]."""
        T, S = th.shape
        p, n = self._tensors(xs, S)
        L.check(L.lib().b200q_calib_histogram_many(self.ctx, T, p.ctypes.data, n.ctypes.data, S, th.ctypes.data, nbins.ctypes.data,
                                                   hists[0].ctypes.data, hists[1].ctypes.data, self._stream()))

    def histogram(self, ndarray, abs_max, bin_num: int = 2048):
        """CaliMathCpu.histogram (cali_math.py:68-80): returns (int32 counts, float32 width)."""
        hist = self.torch.zeros(bin_num, dtype=self.torch.int32, device=self.device)
        abs_max = np.float32(abs_max)
        self.histogram_into(hist, self._dev(ndarray).reshape(-1), np.array([abs_max]), np.array([bin_num]))
        return hist.cpu().numpy(), np.float32(abs_max / np.float32(bin_num - 1))

    def combine_histogram(self, old_hist, arr, new_min, new_max, new_th, bin_num: int = 2048):
        """CaliMathCpu.combine_histogram (cali_math.py:82-103) with the histogram taken on the GPU."""
        (old, old_edges, old_min, old_max, old_th) = old_hist
        if new_th <= old_th:
            hist, _ = self.histogram(arr, old_th, len(old))
            return (old + hist, old_edges, min(old_min, new_min), max(old_max, new_max), old_th)
        old_bins = len(old)
        old_step = old_th / old_bins
        inc = int((new_th - old_th) // old_step + 1)
        new_bins = inc + old_bins
        if new_bins > MAX_GROWN_BINS:
            hist, edges = self.histogram(arr, new_th, bin_num)
            return (hist, edges, min(old_min, new_min), max(old_max, new_max), new_th)
        new_th = inc * old_step + old_th
        hist, edges = self.histogram(arr, new_th, new_bins)
        hist[0:old_bins] += old
        return (hist, edges, min(old_min, new_min), max(old_max, new_max), new_th)

    def find_thresholds(self, hists, widths, dst_bins: int = 128, return_kl: bool = False):
        """find_threshold (kld_calibrator.py:321-347) for a list of device int32 histograms."""
        T = len(hists)
        ptrs = (C.c_void_p * T)(*[h.data_ptr() for h in hists])
        nb = (C.c_int64 * T)(*[h.numel() for h in hists])
        w = (C.c_float * T)(*[float(np.float32(x)) for x in widths])
        out = (C.c_float * T)()
        kl = (C.c_float * (T * 1024))() if return_kl else None
        L.check(L.lib().b200q_calib_find_thresholds(self.ctx, T, ptrs, nb, w, dst_bins, out, kl, self._stream()))
        th = np.frombuffer(out, dtype=np.float32).copy()
        if return_kl:
            return th, np.frombuffer(kl, dtype=np.float32).reshape(T, 1024).copy()
        return th


def kld_threshold_host(hist: np.ndarray, width, dst_bins: int = 128) -> np.float32:
    """BaseKldCalibrator.kld_threshold (kld_calibrator.py:55-59) through the reference's own C symbol, served
    by libb200q.so."""
    h = np.ascontiguousarray(hist, dtype=np.int32)
    return np.float32(L.lib().kl_diversity_hist(h.ctypes.data_as(C.POINTER(C.c_int)), C.c_float(float(width)),
                                                C.c_longlong(h.size), C.c_longlong(dst_bins)))


# ----------------------------------------------------------------------------------------------- sharded driver
@dataclass
class TensorResult:
    name: str
    min: float
    max: float
    abs_max: float
    bins: int
    width: float
    kl: float
    threshold: float     # what the calibration table would hold (min(kl, abs_max), floor 1e-5)


class ShardedCalibrator:
    """Statistics + KLD thresholds for the activations of a forward function, samples sharded across ranks.

    ``forward(batch) -> dict name -> device float32 tensor [B, ...]`` produces every activation of interest for a
    batch of samples; if it has a ``check_status``, that is called once after the last batch and raises if a kernel gave up
    (min / max and the histogram pass over NaN, so a lost activation would end as a plausible threshold); ``shard`` is the local contiguous range of the global sample order.  ``math`` defaults to
    the GPU implementation; ``dist`` is a torch.distributed-like module (None = single process).
    """

    def __init__(self, forward: Callable, math=None, dist=None, bin_num: int = 2048, dst_bins: int = 128):
        self.forward = forward
        self.math = math if math is not None else CaliMathB200()
        self.dist = dist if (dist is not None and dist.is_initialized() and dist.get_world_size() > 1) else None
        self.bin_num = bin_num
        self.dst_bins = dst_bins

    def _check_forward(self, device):
        """Raises on every rank if the forward of one reports that its activations are not valid."""
        import torch
        failed = None
        try:
            getattr(self.forward, "check_status", lambda: None)()
        except Exception as e:      # the ranks learn of it from each other before the next collective
            failed = e
        if self.dist:
            count = torch.tensor([int(failed is not None)], dtype=torch.int32, device=device)
            self.dist.all_reduce(count)
            if failed is None and int(count.item()):
                raise RuntimeError(f"the forward of {int(count.item())} other rank(s) failed")
        if failed is not None:
            raise failed

    def _world(self):
        return (self.dist.get_rank(), self.dist.get_world_size()) if self.dist else (0, 1)

    def run(self, batches: Iterable, samples_per_rank: int, cache_bytes: Optional[int] = None) -> Dict[str, TensorResult]:
        """``batches`` must cover exactly ``samples_per_rank`` local samples in order, and be re-iterable over several ranks or
        with ``cache_bytes`` (it may be walked twice then); rank r holds global samples [r*samples_per_rank, (r+1)*samples_per_rank).

        In a single process a sample's bins depend only on the samples before it, so every batch is forwarded and
        histogrammed once (``_run_streaming``) unless ``cache_bytes`` is given.  Over several ranks (or with
        ``cache_bytes``) the activations of the first pass stay on the device for the second pass while they fit in
        ``cache_bytes`` (default: the device memory that is free when the run starts less 24 GB); batches past that
        budget are forwarded a second time, as the reference does for every batch (kld_calibrator.py:629-760 runs the
        network once for min/max and once more for the histograms).  ``self.timings`` holds the seconds spent per
        phase, ``self.cached_bytes`` the bytes of activations that did not need a second forward."""
        import time
        import torch
        rank, world = self._world()
        m = self.math
        if world == 1 and cache_bytes is None and isinstance(m, CaliMathB200):
            return self._run_streaming(batches, samples_per_rank)
        tm: Dict[str, float] = {}
        cuda = torch.cuda.is_available()

        def lap(key, t0):
            if cuda:
                torch.cuda.synchronize()
            tm[key] = tm.get(key, 0.0) + time.perf_counter() - t0
            return time.perf_counter()

        if cache_bytes is None:
            # what the driver has free plus what torch's allocator holds without using (blocks of an earlier run), less
            # 24 GB for the forward
            idle = torch.cuda.memory_reserved() - torch.cuda.memory_allocated() if cuda else 0
            cache_bytes = max(0, torch.cuda.mem_get_info()[0] + idle - (24 << 30)) if cuda else 0
        # ---- pass 1: per-sample min/max of every tensor
        t0 = time.perf_counter()
        names: List[str] = []
        local: Dict[str, List] = {}
        cache: List[Optional[Dict]] = []
        held = 0
        # The kept activations are copied into a few large slabs: holding the forward's own tensors would make the
        # allocator ask the driver for fresh memory on every batch (slow once peer access is enabled by NCCL), while a
        # copy costs a fraction of the forward and lets the forward reuse its blocks.
        SLAB = 4 << 30
        slabs: List = []
        slab_off = 0

        def keep(acts):
            nonlocal slab_off
            out = {}
            for n in names:
                a = acts[n]
                if not a.is_cuda or a.dtype != torch.float32 or not a.is_contiguous():
                    out[n] = a
                    continue
                nbytes = (a.numel() * 4 + 255) & ~255
                if not slabs or slab_off + nbytes > slabs[-1].numel():
                    ta = time.perf_counter()
                    slabs.append(torch.empty(max(SLAB, nbytes), dtype=torch.uint8, device=a.device))
                    tm["cache_alloc"] = tm.get("cache_alloc", 0.0) + time.perf_counter() - ta
                    slab_off = 0
                v = slabs[-1][slab_off:slab_off + a.numel() * 4].view(torch.float32).view(a.shape)
                v.copy_(a)
                slab_off += nbytes
                out[n] = v
            return out

        # When the activations of the WHOLE shard fit, every tensor gets one region [samples, ...] and the kernels run
        # once per tensor over all its samples (at most CHUNK samples per launch) instead of once per tensor and batch:
        # 2 x 73 launches for ResNet-50 instead of 2 x 73 per batch, whose fixed cost (not their bytes) set the pace.
        CHUNK = 1024
        store: Optional[Dict] = None
        filled = 0
        for batch in batches:
            acts = self.forward(batch)
            if not names:
                names = list(acts.keys())
                local = {n: [] for n in names}
                per_sample = sum(acts[n][0].numel() * 4 for n in names)
                if all(acts[n].is_cuda and acts[n].dtype == torch.float32 for n in names) and per_sample * samples_per_rank <= cache_bytes:
                    ta = time.perf_counter()
                    store = {n: torch.empty((samples_per_rank,) + tuple(acts[n].shape[1:]), dtype=torch.float32, device=acts[n].device)
                             for n in names}
                    tm["cache_alloc"] = time.perf_counter() - ta
                    held = per_sample * samples_per_rank
            if store is not None:
                B = acts[names[0]].shape[0]
                for n in names:
                    store[n][filled:filled + B].copy_(acts[n])
                filled += B
                cache.append(None)
                del acts
                continue
            for n in names:
                a = acts[n]
                local[n].append(m.minmax(a, samples=a.shape[0]))
            need = sum(acts[n].numel() * acts[n].element_size() for n in names)
            if held + need <= cache_bytes and (not cache or cache[-1] is not None):
                cache.append(keep(acts))
                held += need
            else:
                cache.append(None)
            del acts
        if store is not None:
            assert filled == samples_per_rank, "batches do not cover samples_per_rank samples"
            for n in names:
                for c0 in range(0, samples_per_rank, CHUNK):
                    c1 = min(c0 + CHUNK, samples_per_rank)
                    local[n].append(m.minmax(store[n][c0:c1], samples=c1 - c0))
        mm_local = torch.stack([torch.cat(local[n], dim=0) for n in names])            # [T, S_local, 2]
        assert mm_local.shape[1] == samples_per_rank, "batches do not cover samples_per_rank samples"
        t0 = lap("pass1_forward_minmax", t0)
        if self.dist:
            gathered = [torch.empty_like(mm_local) for _ in range(world)]
            self.dist.all_gather(gathered, mm_local.contiguous())
            mm_all = torch.cat(gathered, dim=1)                                          # rank-major = sample order
        else:
            mm_all = mm_local
        mm_all = mm_all.cpu().numpy()
        t0 = lap("gather_minmax", t0)
        # ---- identical schedule on every rank
        sched = dict(zip(names, bin_schedule_many(mm_all[:, :, 0], mm_all[:, :, 1], self.bin_num)))
        t0 = lap("bin_schedule", t0)
        # ---- pass 2: histograms of the local samples into final-size buffers (one flat allocation)
        sizes = [max(sched[n].final_bins, 1) for n in names]
        offs = np.concatenate(([0], np.cumsum(sizes)))
        flat = torch.zeros(int(offs[-1]), dtype=torch.int32, device=mm_local.device)
        views = {n: flat[int(offs[t]):int(offs[t + 1])] for t, n in enumerate(names)}
        s0 = rank * samples_per_rank
        done = 0
        if store is not None:
            for n in names:
                sc = sched[n]
                for c0 in range(0, samples_per_rank, CHUNK):
                    c1 = min(c0 + CHUNK, samples_per_rank)
                    if sc.final_bins and sc.nbins[s0 + c0:s0 + c1].any():
                        m.histogram_into(views[n], store[n][c0:c1], sc.th[s0 + c0:s0 + c1], sc.nbins[s0 + c0:s0 + c1])
        for bi, batch in enumerate(batches if store is None else []):
            acts = cache[bi] if cache[bi] is not None else self.forward(batch)
            cache[bi] = None
            for n in names:
                a = acts[n]
                B = a.shape[0]
                sc = sched[n]
                lo = s0 + done
                if sc.final_bins and sc.nbins[lo:lo + B].any():
                    m.histogram_into(views[n], a, sc.th[lo:lo + B], sc.nbins[lo:lo + B])
            done += next(iter(acts.values())).shape[0]
            del acts
        store = None
        self._check_forward(mm_local.device)
        t0 = lap("pass2_histograms", t0)
        # this rank's own contribution, kept for save_shard (the all-reduce below overwrites `flat` with the sum)
        self._shard = dict(names=list(names), minmax=mm_local.cpu().numpy(), hist=flat.cpu().numpy().copy(), sizes=np.asarray(sizes, np.int64),
                           rank=rank, world=world, samples_per_rank=int(samples_per_rank), bin_num=int(self.bin_num))
        self.allreduce_bytes = int(flat.numel() * 4) if self.dist else 0
        self.cached_bytes = int(held)
        if self.dist:
            self.dist.all_reduce(flat)                                                   # sum of int32 counts
        t0 = lap("allreduce_histograms", t0)
        # ---- KLD
        live = [n for n in names if sched[n].final_bins]
        kl = m.find_thresholds([views[n] for n in live], [sched[n].width for n in live], self.dst_bins) if live else []
        out: Dict[str, TensorResult] = {}
        for n in names:
            sc = sched[n]
            k = float(kl[live.index(n)]) if n in live else 0.0
            out[n] = TensorResult(name=n, min=float(sc.min), max=float(sc.max), abs_max=float(sc.abs_max),
                                  bins=sc.final_bins, width=float(sc.width), kl=k,
                                  threshold=table_threshold(k, sc.abs_max) if n in live else 1e-5)
        lap("kld", t0)
        self.timings = tm
        self.histograms = {n: views[n] for n in names}
        return out


    @staticmethod
    def _samples(name, x, B):
        """The activation as a tensor of B samples: its first dimension is B, or 1 for what is the same in every sample."""
        if x.dim() and x.shape[0] == B:
            return x
        if x.dim() and x.shape[0] == 1:
            return x.expand((B,) + tuple(x.shape[1:])).contiguous()
        raise ValueError(f"{name}: the first dimension of {tuple(x.shape)} is not the batch ({B})")

    def _run_streaming(self, batches: Iterable, samples: int) -> Dict[str, TensorResult]:
        """One pass: per batch the forward, ONE min/max launch over all its activations, the bin schedule of its samples on
        the host (native code, one small copy back), ONE histogram launch over the activations where they lie.  Against
        keeping every activation for a second pass (64 samples of ResNet-50, 2.8 GB of activations: 12.0 ms) nothing is
        copied and the launches do not grow with the number of tensors."""
        import time
        import torch
        m: CaliMathB200 = self.math
        tm: Dict[str, float] = {}

        def lap(key, t0):
            torch.cuda.synchronize()
            t1 = time.perf_counter()
            tm[key] = tm.get(key, 0.0) + t1 - t0
            return t1
        t0 = time.perf_counter()
        names: List[str] = []
        minmax, held, done = [], 0, 0
        sched = None
        CAP = 1 << 16           # bins of a row of the shared histogram matrix at most; longer histograms get buffers of their own
        rows = None             # int32 [T, capacity]
        own: Dict[int, "torch.Tensor"] = {}
        addr = lens = None

        def make_room(need):
            nonlocal rows, addr, lens
            fit = need[need <= CAP]
            cap = int(fit.max()) if fit.size else 0
            if rows is None or cap > rows.shape[1]:
                grown = torch.zeros((len(names), min(CAP, max(4096, 2 * cap))), dtype=torch.int32, device=m.device)
                if rows is not None:
                    grown[:, :rows.shape[1]] = rows
                rows = grown
                addr = rows.data_ptr() + np.arange(len(names), dtype=np.uint64) * np.uint64(4 * rows.shape[1])
                lens = np.full(len(names), rows.shape[1], np.int64)
                for t, h in own.items():
                    addr[t], lens[t] = h.data_ptr(), h.numel()
            for t in np.flatnonzero(need > lens):
                h = torch.zeros(int(need[t] + need[t] // 2), dtype=torch.int32, device=m.device)
                old = own.get(int(t), rows[t])
                h[:old.numel()] = old
                own[int(t)] = h
                addr[t], lens[t] = h.data_ptr(), h.numel()

        for batch in batches:
            acts = self.forward(batch)
            if not names:
                names = list(acts.keys())
                sched = BinScheduler(len(names), self.bin_num)
            B = acts[names[0]].shape[0]
            xs = [self._samples(n, m._dev(acts[n]), B) for n in names]
            held += sum(x.numel() for x in xs) * 4
            mm = m.minmax_many(xs, B)
            minmax.append(mm)
            th, nb = sched.advance(mm)
            make_room(sched.state["bins"])
            for t in np.flatnonzero(sched.state["last_reset"] >= max(done, 1)):    # started over inside this batch
                own.get(int(t), rows[t]).zero_()
            m.histogram_many_into((addr, lens), xs, th, nb)
            done += B
            del acts, xs
        assert done == samples, "batches do not cover samples_per_rank samples"
        self._check_forward(m.device)
        t0 = lap("pass_forward_statistics", t0)
        st = sched.state
        views = {n: own.get(t, rows[t])[:max(int(st["bins"][t]), 1)] for t, n in enumerate(names)}
        host = rows.cpu().numpy()
        self._shard = dict(names=list(names), minmax=np.concatenate(minmax, axis=1), sizes=np.maximum(st["bins"], 1).astype(np.int64),
                           hist=np.concatenate([own[t].cpu().numpy()[:views[n].numel()] if t in own else host[t, :views[n].numel()]
                                                for t, n in enumerate(names)]),
                           rank=0, world=1, samples_per_rank=int(samples), bin_num=int(self.bin_num))
        self.allreduce_bytes = 0
        self.cached_bytes = int(held)
        live = np.flatnonzero(st["bins"])
        kl = np.zeros(len(names), np.float32)
        if live.size:
            kl[live] = m.find_thresholds([views[names[t]] for t in live], st["width"][live], self.dst_bins)
        amax = np.maximum(np.abs(st["min"]), np.abs(st["max"]))
        out: Dict[str, TensorResult] = {}
        for t, n in enumerate(names):
            k = float(kl[t])
            out[n] = TensorResult(name=n, min=float(st["min"][t]), max=float(st["max"][t]), abs_max=float(amax[t]), bins=int(st["bins"][t]),
                                  width=float(st["width"][t]), kl=k, threshold=table_threshold(k, amax[t]) if st["bins"][t] else 1e-5)
        lap("kld", t0)
        self.timings = tm
        self.histograms = views
        return out


def save_shard(calibrator: ShardedCalibrator, path: str) -> None:
    """Persist this rank's part of a finished ``run``: its per-sample (min, max) pairs and its local histograms (before
    the all-reduce), so that a calibration can be re-merged without the ranks, or one shard recomputed after a failure
    (the reference keeps only the final table, kld_calibrator.py:804-884)."""
    sh = calibrator._shard
    np.savez(path, names=np.array(sh["names"]), minmax=sh["minmax"], hist=sh["hist"], sizes=sh["sizes"],
             meta=np.array([sh["rank"], sh["world"], sh["samples_per_rank"], sh["bin_num"]], np.int64))


def merge_shards(paths: Sequence[str], math=None, dst_bins: int = 128) -> Dict[str, TensorResult]:
    """Rebuild the result of a sharded run from the files ``save_shard`` wrote, one per rank: the bin schedule is
    recomputed from all ranks' (min, max) pairs in rank order, the int32 histograms are summed (what the all-reduce
    does) and the thresholds searched again.  Raises if a shard is missing or was histogrammed under another schedule
    (e.g. recomputed with different samples)."""
    import torch
    shards = sorted((dict(np.load(p)) for p in paths), key=lambda d: int(d["meta"][0]))
    world = int(shards[0]["meta"][1])
    if [int(d["meta"][0]) for d in shards] != list(range(world)):
        raise ValueError(f"need one shard per rank 0..{world - 1}, got ranks {[int(d['meta'][0]) for d in shards]}")
    names = [str(n) for n in shards[0]["names"]]
    bin_num = int(shards[0]["meta"][3])
    for d in shards:
        if [str(n) for n in d["names"]] != names or int(d["meta"][3]) != bin_num or int(d["meta"][2]) != int(shards[0]["meta"][2]):
            raise ValueError("shards disagree on tensors, samples per rank or bin count")
    mm_all = np.concatenate([d["minmax"] for d in shards], axis=1)
    sched = bin_schedule_many(mm_all[:, :, 0], mm_all[:, :, 1], bin_num)
    sizes = np.array([max(sc.final_bins, 1) for sc in sched], np.int64)
    for d in shards:
        if not np.array_equal(d["sizes"], sizes):
            raise ValueError("a shard's histograms were built under a different bin schedule: recompute it with the same samples")
    flat = np.sum([d["hist"].astype(np.int64) for d in shards], axis=0).astype(np.int32)
    offs = np.concatenate(([0], np.cumsum(sizes)))
    m = math if math is not None else CaliMathB200()
    dev = "cuda" if isinstance(m, CaliMathB200) else "cpu"
    tflat = torch.from_numpy(flat).to(dev)
    views = [tflat[int(offs[t]):int(offs[t + 1])] for t in range(len(names))]
    live = [t for t, sc in enumerate(sched) if sc.final_bins]
    kl = m.find_thresholds([views[t] for t in live], [sched[t].width for t in live], dst_bins) if live else []
    out: Dict[str, TensorResult] = {}
    for t, n in enumerate(names):
        sc = sched[t]
        k = float(kl[live.index(t)]) if t in live else 0.0
        out[n] = TensorResult(name=n, min=float(sc.min), max=float(sc.max), abs_max=float(sc.abs_max), bins=sc.final_bins,
                              width=float(sc.width), kl=k, threshold=table_threshold(k, sc.abs_max) if t in live else 1e-5)
    return out


def dump_cali_table(path: str, results: Dict[str, TensorResult], *, order: Optional[List[str]] = None, mlir_file: str = "",
                    num_samples: int = 0, tune_num: int = 0, histogram_bin_num: int = 2048) -> None:
    """Write the results of ``ShardedCalibrator.run`` as a calibration table in the reference's text format
    (kld_calibrator.py:804-884): tensors in graph order, ``threshold min max`` with seven decimals."""
    from .cali_table import write_cali_table
    names = order if order is not None else list(results.keys())
    rows = [(n, float(results[n].threshold), float(results[n].min), float(results[n].max)) for n in names if n in results]
    write_cali_table(path, rows, mlir_file=mlir_file, method="use_kl", histogram_bin_num=histogram_bin_num,
                     num_samples=num_samples, tune_num=tune_num)
