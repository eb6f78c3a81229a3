"""Filtered ranking and top-k over an entity table without materialising the score matrix.

``rank = 1 + #{j : s_j > s_target} − #{j ∈ known answers, j ≠ target : s_j > s_target}``: the dense count comes
from the tcgen05 kernel ``dice_rank_count`` (GEMM tiles in TMEM, counting epilogue), which leaves out the known answers
through a bit mask where that is cheaper; otherwise they are counted by gather-dots (``dice_eval_sparse``), like the target
scores.  With a process group every rank holds a row shard of the
table (contiguous or cyclic); target scores, counts and top-k candidates are merged across ranks by merge kernels that
read the ranks' buffers in a symmetric heap through peer loads, ordered by the bounded device barrier: the hot loop
holds no library collective and no host round trip.

The reference sorts a dense ``[B, |E|]`` matrix per batch (``dicee/evaluation/evaluator.py:484-508``) and uses
``torch.topk`` over all scores for ``predict_topk`` (``dicee/knowledge_graph_embeddings.py:533-607``).
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import kernels

SUPPORTED_D = (64, 128, 256)


def pad_dim(d: int) -> Optional[int]:
    for s in SUPPORTED_D:
        if d <= s:
            return s
    return None


def to_kernel_operand(x: torch.Tensor, d_pad: int) -> torch.Tensor:
    """bf16, contiguous, zero-padded to ``d_pad`` columns."""
    x = x.detach()
    if x.shape[1] == d_pad:
        return x.to(torch.bfloat16).contiguous()
    out = torch.zeros(x.shape[0], d_pad, dtype=torch.bfloat16, device=x.device)
    out[:, :x.shape[1]] = x
    return out


class FusedRanker:
    """Holds one (shard of an) entity table in kernel layout and answers rank / top-k queries against it.

    ``table`` rows are entities ``y_offset + c * y_stride``; ``col_bias`` (fp32, per local row) is added to every
    score of that entity.  ``group``: process group over which the table is sharded (``None`` = whole table here).
    """

    def __init__(self, table: torch.Tensor, col_bias: Optional[torch.Tensor] = None, y_offset: int = 0,
                 y_stride: int = 1, group=None, exact: bool = False, band_capacity: int = 1 << 24):
        """``exact``: ranks equal those of an fp32 scoring of the same operands.  The tensor cores still do the bulk of the
        work, on operands split into two bf16 terms each; such a score differs from its fp32 value by at most
        ``MARGIN[d] · ‖q‖ · ‖e‖`` (plus the rounding of the bias), so only entities within that margin of the target are
        undecided, and exactly those (0.2 percent for targets in the middle of a random table, far fewer near its top) are
        re-scored in fp32 by a second, sparse pass."""
        assert table.is_cuda, "the fused ranker runs on a CUDA device"
        self.d = table.shape[1]
        self.d_pad = pad_dim(self.d)
        if self.d_pad is None:
            raise ValueError(f"embedding width {self.d} exceeds the kernel's limit of {SUPPORTED_D[-1]}")
        self.exact = bool(exact)
        if self.exact:
            t32 = table.detach().float()
            self.table, self.table_lo, copy, _ = kernels.split_rows(t32, self.d_pad, want_copy=self.d != self.d_pad)
            self.table_f32 = copy if copy is not None else t32.contiguous()
            self.row_norm_max = float(self.table_f32.norm(dim=1).max()) if table.shape[0] else 0.0
            self.band_rows = torch.empty(band_capacity, dtype=torch.int32, device=table.device)
            self.band_cols = torch.empty(band_capacity, dtype=torch.int32, device=table.device)
        else:
            self.table = to_kernel_operand(table, self.d_pad)
        self.col_bias = None if col_bias is None else col_bias.detach().float().contiguous()
        self.bias_max = 0.0
        if self.exact and self.col_bias is not None and table.shape[0]:
            self.bias_max = float(self.col_bias.abs().nan_to_num(0.0, 0.0).max())   # a column at -inf is undecided for no one
        self.y_offset, self.y_stride, self.group = int(y_offset), int(y_stride), group
        self.device = table.device
        self._flags = torch.zeros(2, dtype=torch.int32, device=self.device)
        self.status = self._flags[0:1]      # kernel status word
        self.overflow = self._flags[1:2]    # set when a top-k candidate list ran full
        self._scan_done = {}
        self._whole_table = False           # top-k thresholds from the whole table: set once a list of the two-stage search ran full
        self.W, self.rank = 1, 0
        self._heap = None
        if group is not None:
            import torch.distributed as dist
            self.W, self.rank = dist.get_world_size(group), dist.get_rank(group)
            if self.W == 1:
                self.group = None
            elif self.exact:   # the margin of the band mode needs the largest row norm and bias over all shards: once, here
                emax = torch.tensor([self.row_norm_max, self.bias_max], device=self.device)
                dist.all_reduce(emax, op=dist.ReduceOp.MAX, group=group)
                self.row_norm_max, self.bias_max = emax.tolist()

    # ------------------------------------------------------------------ cross-rank merge (symmetric heap + barrier)
    K_CAP = 32

    def _merge_buffers(self, B: int):
        """Symmetric buffers for ``B`` queries (collective when they have to grow: every rank calls with the same
        ``B``).  Two candidate sets alternate between top-k calls, so one barrier per call is enough."""
        if self._heap is None or self._heap_rows < B:
            from ..parallel.symm import SymmetricHeap
            rows = max(B, 1024)
            heap = SymmetricHeap(self.group, self.device, multicast=False)
            heap.plan("tgt", (rows,), torch.float32)
            heap.plan("greater", (rows,), torch.int32)
            heap.plan("filtered", (rows,), torch.int32)
            for par in (0, 1):
                heap.plan(f"cs{par}", (rows, self.K_CAP), torch.float32)
                heap.plan(f"ci{par}", (rows, self.K_CAP), torch.int64)
            heap.plan("sig", (64,), torch.int32)
            heap.commit()
            self._heap, self._heap_rows = heap, rows
            self._tab = {n: heap.table(n) for n in ("tgt", "greater", "filtered", "cs0", "ci0", "cs1", "ci1", "sig")}
            self._bar_count = torch.zeros(1, dtype=torch.int32, device=self.device)
            self._topk_parity = 0
            heap.host_barrier()
        return self._heap

    def _barrier(self) -> None:
        kernels.p2p_barrier(self._tab["sig"], self.rank, self.W, self._bar_count, self.status)

    def check(self) -> None:
        """Raise if a kernel reported a failure or a candidate list overflowed.  This is the one place where the ranker
        waits for the GPU: :meth:`ranks` and :meth:`topk` only queue work."""
        code, over = self._flags.tolist()
        if code != 0 or over != 0:
            self._flags.zero_()
        if code != 0:
            raise kernels.KernelError(f"kernel status {code} ({kernels.STATUS_TEXT.get(code, '?')}) in the fused ranker"
                                      " (band list full: raise band_capacity or use smaller batches)")
        if over != 0:
            self._whole_table = True
            raise kernels.KernelError("a top-k candidate list ran full (the sample of the table gave too low a threshold); call "
                                      "topk again: this ranker takes its thresholds from the whole table from here on")

    #: relative error of a split score for each padded width: the terms left out of (hi + lo)(hi + lo) are at most
    #: 3 · 2^-16, the accumulation of 3 d products and of the fp32 reference at most 4 d · 2^-23
    MARGIN = {d: 3 * 2.0 ** -16 + 4 * d * 2.0 ** -23 for d in SUPPORTED_D}
    #: error relative to the largest column bias: the sum with it is rounded once for either score and once for the bounds of
    #: the band, by 2^-24 of it each (the score's share of those sums is far inside MARGIN)
    BIAS_MARGIN = 2.0 ** -22
    #: largest bit mask of known answers (bytes); beyond it the known answers are scored one by one
    MASK_LIMIT = 512 << 20

    def _mask_words(self) -> int:
        return (self.table.shape[0] + 127) // 128 * 4

    def _mask_pays(self, B: int, entries: int) -> bool:
        """A bit mask of the known answers costs clearing, setting and reading ``B · |E| / 8`` bytes; scoring them one by
        one reads a row of the table for each.  Queries of a popular pair have thousands of known answers, and the warps
        that walked them took 10 of the 21 ms of an evaluation of 20 466 queries against 14 541 entities; with 16 answers
        per query against two million rows the lists cost 41 us and the mask would be 2 GB."""
        mask = B * self._mask_words() * 4
        row = self.d_pad * (4 if self.exact else 2)
        return self.group is None and mask <= self.MASK_LIMIT and entries * row > 4 * mask

    @torch.no_grad()
    def ranks(self, q: torch.Tensor, target: torch.Tensor, filt_ptr: Optional[torch.Tensor] = None,
              filt_cols: Optional[torch.Tensor] = None) -> torch.Tensor:
        """Filtered ranks ``[B]`` (int64) of entity ``target[i]`` for query vector ``q[i]``.  The filter of query
        ``i`` is ``filt_cols[filt_ptr[i]:filt_ptr[i+1]]`` (global entity ids; the target itself is ignored).  An answer that
        beats the target is subtracted as often as its list names it (see ``filtered_rank_from_scores``); the lists of a
        :class:`PairCSR` name every answer once."""
        B = q.shape[0]
        if filt_ptr is not None:
            filt_ptr = filt_ptr.to(torch.int64).contiguous()
            filt_cols = filt_cols.to(torch.int32).contiguous()
            if self.y_offset == 0 and self.y_stride == 1 and self._mask_pays(B, filt_cols.numel()):
                cleared, mask = self._cleared(B, self._mask_words())
                repeated = torch.empty(filt_cols.numel() // 32 + B, dtype=torch.int32, device=self.device)
                kernels.filter_mask(mask, self.table.shape[0], ptr=filt_ptr, cols=filt_cols, repeated=repeated)
                return self._ranks(q, target, filt_ptr, filt_cols, mask, cleared, repeated=repeated)
        return self._ranks(q, target, filt_ptr, filt_cols, None)

    def _cleared(self, B: int, words: int):
        """Zeros for one batch in one fill: target scores and counts (and the band's counter) and the mask ``[B, words]``."""
        rows = (B + 3) // 4 * 4
        buf = torch.zeros(2 * rows + 4 + B * words, dtype=torch.int32, device=self.device)
        small, mask = buf[:2 * rows + 4], buf[2 * rows + 4:].view(B, words)
        return (small[:B].view(torch.float32), small[rows:rows + B], small[2 * rows:2 * rows + 2].view(torch.int64)), mask

    @torch.no_grad()
    def ranks_of_pairs(self, q: torch.Tensor, target: torch.Tensor, ab: torch.Tensor, num_b: int, keys: torch.Tensor,
                       offsets: torch.Tensor, values: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
        """:meth:`ranks` with the filter of query ``i`` given as the pair in the first two columns of ``ab[i]``, looked up on
        the device in a CSR over sorted keys ``a * num_b + b`` (whole table on this device)."""
        assert self.group is None and self.y_offset == 0 and self.y_stride == 1
        cleared, mask = self._cleared(q.shape[0], self._mask_words())
        kernels.filter_mask(mask, self.table.shape[0], ab=ab, num_b=num_b, keys=keys, offsets=offsets, values=values)
        return self._ranks(q, target, None, None, mask, cleared, out)

    def _ranks(self, q, target, filt_ptr, filt_cols, mask, cleared=None, out=None, repeated=None) -> torch.Tensor:
        B = q.shape[0]
        tgt_idx = target.to(torch.int32).contiguous()
        sharded = self.group is not None
        if sharded:   # partial results live in the symmetric heap, where the merge kernels of every rank read them
            heap = self._merge_buffers(B)
            tgt_part, greater, filtered = heap.local("tgt")[:B], heap.local("greater")[:B], heap.local("filtered")[:B]
            tgt_part.zero_()   # the count buffers are cleared behind the first barrier: a slower rank may still be
            tgt_score = torch.empty(B, dtype=torch.float32, device=self.device)   # merging the previous call's counts
        else:
            tgt_score, greater, band_count = cleared if cleared is not None else self._cleared(B, 0)[0]
            tgt_part = tgt_score
            # with a mask the lists are only looked at for repeated answers, whose further mentions come off the counts directly
            filtered = torch.zeros(B, dtype=torch.int32, device=self.device) if filt_ptr is not None and mask is None else None
        kw = dict(col_bias=self.col_bias, y_offset=self.y_offset, y_stride=self.y_stride)
        band = {}
        if self.exact:
            # target scores and filtered counts from the fp32 operands, dense counts from the split ones
            q32 = q.detach().float()
            qk, q_lo, copy, margin = kernels.split_rows(q32, self.d_pad, want_copy=self.d != self.d_pad,
                                                        margin_factor=self.row_norm_max * self.MARGIN[self.d_pad],
                                                        margin_offset=self.bias_max * self.BIAS_MARGIN)
            qs, table = copy if copy is not None else q32.contiguous(), self.table_f32
            if sharded:
                band_count = torch.zeros(1, dtype=torch.int64, device=self.device)
            band = dict(x_lo=q_lo, y_lo=self.table_lo, margin=margin, band_rows=self.band_rows, band_cols=self.band_cols,
                        band_count=band_count)
        else:
            qk = to_kernel_operand(q, self.d_pad)
            qs, table = qk, self.table
        if sharded:  # phase 1: owners score their targets, phase 2: everybody counts against the merged scores
            kernels.eval_sparse(qs, table, tgt_idx, tgt_part, None, **kw)
            self._barrier()
            kernels.peer_sum_f32(self._tab["tgt"], self.W, tgt_score, B, self.status)
            greater.zero_()
            filtered.zero_()
            if filt_ptr is not None:
                kernels.eval_sparse(qs, table, tgt_idx, None, filtered, filt_ptr, filt_cols, target_in=tgt_score, **kw)
        else:
            kernels.eval_sparse(qs, table, tgt_idx, tgt_score, filtered if mask is None else greater, filt_ptr, filt_cols,
                                repeated=repeated, **kw)
        kernels.rank_count(qk, self.table, tgt_score, tgt_idx, greater, self.status, mask=mask, **band, **kw)
        if self.exact:
            kernels.eval_band_exact(qs, table, self.band_rows, self.band_cols, band_count, tgt_score, greater, **kw)
        if self.group is None:
            if filtered is not None:
                greater.sub_(filtered)
            return torch.add(greater, 1, out=out if out is not None else
                             torch.empty(B, dtype=torch.int64, device=self.device))
        out = torch.empty(B, dtype=torch.int64, device=self.device)
        self._barrier()                       # every rank's counts are complete
        kernels.merge_ranks(self._tab["greater"], self._tab["filtered"], self.W, out, B, self.status)
        return out

    #: tables with more rows than this are searched in two stages (threshold from a sample, then one collecting pass)
    TWO_STAGE_ROWS = 131072
    SAMPLE_ROWS = 32768

    #: queries per pass, and what the group maxima of a pass may take (16 KB per query at 131 072 rows)
    TOPK_QUERIES = 8192
    GROUP_MAX_BYTES = 1 << 30

    def _sample_rows(self) -> torch.Tensor:
        """One row out of each of ``SAMPLE_ROWS`` equally long ranges of the table, at a place a hash of the range's number
        gives: the whole table is covered, and no order of the rows (sorted, periodic) can keep a class of them out."""
        n, S = self.table.shape[0], self.SAMPLE_ROWS
        i = torch.arange(S + 1, dtype=torch.int64, device=self.device)
        edge = i * n // S
        h = (i[:S] + 1) * 0x9E3779B97F4A7C1            # odd multipliers and shifts: Fibonacci hashing, twice
        h = (h ^ (h >> 29)) * 0x5851F42D4C957F2D
        return edge[:S] + ((h >> 33) & 0x7fffffff) % (edge[1:] - edge[:S])

    def _list_capacity(self, kk: int) -> int:
        """Room for the scores above the ``kk``-th best of the sample.  In units of ``n / S`` their number follows a gamma
        distribution of order ``kk`` (exponential for 1); it is above ``kk + 6 sqrt(kk) + 24`` of them with probability 6e-13
        or less for every ``kk`` up to 32, so that a call of 8192 queries meets a full list once in 200 million calls."""
        return int((kk + 6 * kk ** 0.5 + 24) * (self.table.shape[0] / self.SAMPLE_ROWS)) + 64

    def _done(self) -> torch.Tensor:
        """Block counter of the scan: calls on one stream follow one another, so there is one per stream."""
        if not torch.cuda.is_current_stream_capturing():
            key = torch._C._cuda_getCurrentRawStream(self.device.index)
            if key in self._scan_done:
                return self._scan_done[key]
            if len(self._scan_done) < 64:
                self._scan_done[key] = torch.zeros(1, dtype=torch.int32, device=self.device)
                return self._scan_done[key]
        return torch.zeros(1, dtype=torch.int32, device=self.device)

    def _topk_local(self, q: torch.Tensor, kk: int):
        n_local, B = self.table.shape[0], q.shape[0]
        kw = dict(col_bias=self.col_bias, y_offset=self.y_offset, y_stride=self.y_stride)
        # up to four queries: one launch that reads the table once on the ordinary cores.  Everything else goes through the
        # tensor cores, where a tile costs the same for 1 query as for 128.
        if kk and B and q.dtype in (torch.float32, torch.bfloat16) and q.stride(1) == 1 and kernels.topk_scan_blocks(B, n_local):
            return kernels.topk_scan(q, self.table, kk, self._done(), **kw)
        if kk == 0 or B == 0:
            return (torch.empty(B, kk, dtype=torch.float32, device=self.device),
                    torch.empty(B, kk, dtype=torch.int64, device=self.device))
        two_stage = n_local > self.TWO_STAGE_ROWS and not self._whole_table
        most = self.TOPK_QUERIES if two_stage else max(1, min(self.TOPK_QUERIES, self.GROUP_MAX_BYTES // (16 * ((n_local + 127) // 128))))
        if B > most:
            parts = [self._topk_local(q[i:i + most], kk) for i in range(0, B, most)]
            return torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
        qk = to_kernel_operand(q, self.d_pad)
        if not two_stage:
            return kernels.topk_bounded(qk, self.table, kk, self.status, self.overflow, **kw)
        # stage 1: the k-th best score over a sample of the table (copied once per ranker) is a lower bound of the k-th best
        # overall
        if getattr(self, "_sample", None) is None:
            rows = self._sample_rows()
            self._sample_bias = None if self.col_bias is None else self.col_bias[rows]
            self._sample = self.table[rows]
        floor = kernels.topk_bounded(qk, self._sample, kk, self.status, self.overflow, col_bias=self._sample_bias, kth_only=True)
        # stage 2: one pass over the whole table that collects what reaches the bound (few per row).  A list that ran full is
        # recorded on the device and reported by check()
        return kernels.topk_bounded(qk, self.table, kk, self.status, self.overflow, floor=floor,
                                    cand_cap=self._list_capacity(kk), **kw)

    @torch.no_grad()
    def topk(self, q: torch.Tensor, k: int) -> Tuple[torch.Tensor, torch.Tensor]:
        """``(scores [B, k], entity ids [B, k])`` of the best entities per query, best first."""
        n_local = self.table.shape[0]
        if k > 32:  # beyond the in-kernel list: plain matmul in slices (rare; interactive use)
            s = to_kernel_operand(q, self.d_pad).float() @ self.table.float().t()
            if self.col_bias is not None:
                s = s + self.col_bias
            sc, ix = torch.topk(s, min(k, n_local), dim=1)
            ix = ix * self.y_stride + self.y_offset
        else:
            kk = min(k, n_local)
            sc, ix = self._topk_local(q.detach(), kk)
        if self.group is not None:
            sc, ix = self._merge_topk(sc, ix, k)
        return sc, ix

    def _merge_topk(self, sc: torch.Tensor, ix: torch.Tensor, k: int):
        """Every rank publishes its local best ``k`` in the symmetric heap; after one barrier a merge kernel picks the
        best ``k`` of the ``W · k`` candidates per query by peer loads.  The candidate buffers alternate between calls,
        so the next call's writes cannot meet a slower rank's reads of this one."""
        B = sc.shape[0]
        if k > self.K_CAP or self.W * k > 256:   # beyond the merge kernel: library path (interactive use only)
            import torch.distributed as dist
            all_s = [torch.empty_like(sc) for _ in range(self.W)]
            all_i = [torch.empty_like(ix) for _ in range(self.W)]
            dist.all_gather(all_s, sc.contiguous(), group=self.group)
            dist.all_gather(all_i, ix.contiguous(), group=self.group)
            cat_s, cat_i = torch.cat(all_s, 1), torch.cat(all_i, 1)
            s2, pos = torch.topk(cat_s, min(k, cat_s.shape[1]), dim=1)
            return s2, torch.gather(cat_i, 1, pos)
        heap = self._merge_buffers(B)
        par = self._topk_parity
        self._topk_parity ^= 1
        cs, ci = heap.local(f"cs{par}")[:B], heap.local(f"ci{par}")[:B]
        cs.fill_(float("-inf"))
        ci.fill_(-1)
        cs[:, :sc.shape[1]].copy_(sc)
        ci[:, :ix.shape[1]].copy_(ix)
        out_s = torch.empty(B, k, dtype=torch.float32, device=self.device)
        out_i = torch.empty(B, k, dtype=torch.int64, device=self.device)
        self._barrier()
        kernels.merge_topk(self._tab[f"cs{par}"], self._tab[f"ci{par}"], self.W, k, self.K_CAP, out_s, out_i, B,
                           self.status)
        return out_s, out_i


def supports(model) -> bool:
    """True when ``model`` can be ranked by the fused path: bilinear contract, CUDA parameters, width ≤ 256."""
    try:
        w = model.entity_embeddings.weight
    except AttributeError:
        return False
    return bool(getattr(model, "bilinear", False)) and w.is_cuda and pad_dim(w.shape[1]) is not None \
        and kernels._lib.available()


def ranker_for_model(model, exact: bool = True) -> FusedRanker:
    """Ranker over the model's entity table; ``exact`` (default) gives the ranks of an fp32 evaluation."""
    return FusedRanker(model.entity_embeddings.weight, exact=exact)


@torch.no_grad()
def model_queries(model, hr: torch.Tensor) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """``(q, bias)`` of the model's bilinear form for index pairs ``hr [B, 2]``."""
    h, r = model.get_head_relation_representation(hr)
    return model.compose(h, r)
