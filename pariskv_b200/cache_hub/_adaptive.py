"""Shared body of the two adaptive-k cache variants: value-norm bookkeeping and the adaptive selection step.

Both variants keep all C rerank candidates, weight them by exp(logit - max) * ||v|| together with the window
rows, and attend the shortest benefit-ordered prefix that reaches a share `threshold` of the total benefit
(reference: cache_hub/polar_cache_atten_value_indices_adaptive_k.py:1510-1589,
cache_hub/polar_cache_adaptivek_varlen.py:1684-1812).  Here the selection is one kernel
(adaptive_select), which makes the window logits and gathers the value norms of the candidates itself, and the
attention kernel takes per-head row counts, so there is no host synchronisation, no index packing and no staging copy.
"""
import math

import torch

from .. import _lib, ops
from .polar_cache import polar_cache as _base_cache


class AdaptiveKCache(_base_cache):
    # (candidate_ratio, collision_ratio) by zone length, adaptive variants
    # (cache_hub/polar_cache_adaptivek_varlen.py:2115-2126)
    def _ratio_rows(self):
        return [(0.5, 0.5), (0.25, 0.3), (0.2, 0.25), (0.05, 0.2)]

    def _max_selected_rows(self):
        return max(super()._max_selected_rows(), 4096)   # the adaptive selection may attend up to 4096 rows per head

    def _init_adaptive(self, threshold, min_k, max_k, per_head):
        self.adaptive_topk_threshold = float(threshold)
        self._min_k, self._max_k, self._per_head = int(min_k), int(max_k), bool(per_head)
        if self._max_k > 4096:
            raise ValueError("adaptive top-k supports at most 4096 rows per head")
        dev, bs, H = self.device, self.batch_size, self.kv_head
        self._attn_scale = 1.0 / math.sqrt(self.head_dim)
        # ||v|| of the window rows and of the zone rows (zone-relative index), fp32.  The window norms are the staging
        # array that the append kernel fills for every cache; the zone norms are published by its flush.
        self._sl_vnorm_cache = self._win_vnorm
        self.value_norm_gpu = [torch.zeros(bs, H, self.zone_capacity, dtype=torch.float32, device=dev)
                               for _ in range(self.layer_num)]
        self._last_adaptive = None
        self.fixed_shapes = False   # True: capacity-shaped tensors on eager steps too (what a stream capture uses)

    @property
    def last_adaptive(self):
        """(adaptive_k, topk_indices, n_sel, sl_logits, cand, cand_scores) of the last compute, the scores as the bf16
        values that were ranked."""
        last = self._last_adaptive
        return last and (*last[:5], last[5].to(torch.bfloat16))

    def _zone_vnorm(self, layer):
        return self.value_norm_gpu[layer]

    # ---- decode attention ---------------------------------------------------------------------------------
    def compute(self, queries, layer_idx):
        queries = queries.contiguous()
        self._wait_offload(layer_idx)
        N = self.cpu_valid_end[layer_idx]
        n_win = self._window_len[layer_idx]
        total = self.current_seq_len[layer_idx]
        if total < max(self.FULL_ATTENTION_THRESHOLD, self.steady_size + 2 * self.final_topk) or N <= 0:
            return super().compute(queries, layer_idx)
        wk, wv = self.unified_keys_gpu[layer_idx], self.unified_values_gpu[layer_idx]
        # rows of the candidate lists are c_max long; a sample's own count follows from its zone length, read on the
        # device, and the rest of its row carries score -inf (no weight in the adaptive selection)
        _, _, ex = ops.retrieve_ex(queries, self.srht_diagonal_signs, self._mag_centers, self.codebook_gpu[layer_idx],
                                   self.key_block_weight_gpu[layer_idx], self.key_4bit_packed_gpu[layer_idx],
                                   self.cluster_key_counts_gpu[layer_idx], self._c_max, 0, kv_len=self._zone_len_dev[layer_idx],
                                   schedule=self._zone_schedule, want=("cand", "scores_f32", "query_avg"),
                                   scratch=self._retrieve_scratch)
        cand, cand_scores = ex["cand"], ex["scores_f32"]
        C = self.retrieval_plan(N)[1]          # candidates of the longest sample
        # Shapes that follow the host's view of the lengths (the reference's shapes) on eager steps; inside a stream
        # capture, or with fixed_shapes set, every shape is a capacity and the lengths act on the device only: window
        # rows beyond the filled part get logit -inf, candidate rows keep their -inf tail, and a head never attends
        # more rows than it has candidates.  Both forms attend the same rows.
        fixed = self.fixed_shapes or torch.cuda.is_current_stream_capturing()
        equal = min(self.zone_len[layer_idx]) == N
        if fixed:
            n_rows, C = self.window_capacity, cand.shape[2]
        else:
            n_rows = n_win
            if equal:   # equal lengths: the lists as the reference shapes them, [bs,H,C]
                cand, cand_scores = cand[:, :, :C], cand_scores[:, :, :C]
        K_out = min(self._max_k, C)
        # rows longer than a sample's candidate list: its count caps what the head attends
        capped = fixed or not equal
        adaptive_k, topk, n_sel, sl_logits = _lib.native().adaptive_select(
            ex["query_avg"], wk, self._window_rows_dev[layer_idx] if fixed else None, n_rows, cand_scores, ex["n_cand"] if capped else None,
            self._attn_scale, self._sl_vnorm_cache[layer_idx][:, :, :n_rows], cand, self.value_norm_gpu[layer_idx],
            self.adaptive_topk_threshold, K_out, max(1, min(self._min_k, K_out)), max(1, K_out))
        if not self._per_head:  # dense variant: every head attends the first max-over-heads rows of its own ranking
            n_sel = adaptive_k.max().to(torch.int32).expand_as(adaptive_k).contiguous()
            if capped:
                n_sel = torch.minimum(n_sel, ex["n_cand"])
        self._last_adaptive = (adaptive_k, topk, n_sel, sl_logits, cand, cand_scores)
        self.last_topk_indices = topk
        if fixed:
            return self._attend(queries, wk, wv, self.window_capacity, self._store_k[layer_idx], self._store_v[layer_idx],
                                topk, n_sel=n_sel, n_window_dev=self._window_rows_dev[layer_idx], n_window_add=0)
        return self._attend(queries, wk, wv, n_win, self._store_k[layer_idx], self._store_v[layer_idx], topk,
                            n_sel=n_sel)
