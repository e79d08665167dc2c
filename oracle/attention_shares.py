"""CPU checker of batched attention by shares (opcode 10): which cached positions a share takes, and its arithmetic.

TEST INFRASTRUCTURE, NOT A PRODUCT PATH.  A restatement of how the kernel cuts a layer's attention: a unit is four, two or one
neighbouring key/value heads of a sequence, as long as its stages and ``UNIT_COST`` more; units stand in line (sequence, heads), and
share ``r`` of ``R`` is the r-th part of the line.  No counterpart in the reference, which decodes one sequence.
"""

from __future__ import annotations

from dataclasses import dataclass

import numpy as np
import torch
from torch import Tensor

UNIT_COST, STAGE_ELEMENTS, MOST_PARTS = 12, 8192, 23
STAGE_COST = {4: 1.0, 2: 1.01, 1: 1.05}


@dataclass(frozen=True)
class Piece:
    seq: int
    head: int  # first key/value head
    heads: int
    first: int  # stages first .. last - 1 of `stages`
    last: int
    stages: int
    parts: int
    part: int


@dataclass(frozen=True)
class LineUp:
    heads: int
    shares: int  # at most
    units: int  # of a sequence
    stages: tuple[int, ...]
    starts: tuple[int, ...]

    @classmethod
    def of(cls, positions: list[int], kv_heads: int, head_dim: int, max_partials: int, sms: int) -> "LineUp":
        def stages(h):
            run = STAGE_ELEMENTS // head_dim // h
            return [-(-p // run) for p in positions]

        rows, best = min(MOST_PARTS, max_partials - 1), None
        for h in (4, 2, 1):
            if kv_heads % h:
                continue
            lengths = [n + UNIT_COST for n in stages(h)]
            line = kv_heads // h * sum(lengths)
            most = max(1, min(line, rows * line // max(lengths)))
            time = np.float32(line) * np.float32(STAGE_COST[h]) / np.float32(min(most, sms))
            if best is None or time < best[0]:
                best = (time, h, most)
        _, heads, most = best
        units, starts = kv_heads // heads, [0]
        for n in stages(heads):
            starts.append(starts[-1] + units * (n + UNIT_COST))
        return cls(heads, most, units, tuple(stages(heads)), tuple(starts))

    def pieces(self, rank: int, ranks: int) -> list[Piece]:
        total, shares = self.starts[-1], min(ranks, self.shares)
        if rank >= shares:
            return []
        begin, end, out = total * rank // shares, total * (rank + 1) // shares, []
        for seq, n in enumerate(self.stages):
            for unit in range(self.units):
                at, length = self.starts[seq] + unit * (n + UNIT_COST), n + UNIT_COST
                # cuts at or before this one leave the unit whole behind them
                edge = at + min(UNIT_COST, length - 1)
                if at + length <= begin or end <= edge:
                    continue
                share_of = lambda x: ((x + 1) * shares - 1) // total  # noqa: E731
                if rank < share_of(edge):
                    continue
                first = 0 if begin <= edge else begin - at - UNIT_COST
                out.append(Piece(seq, unit * self.heads, self.heads, first, min(n, end - at - UNIT_COST), n,
                                 share_of(at + length - 1) - share_of(edge) + 1, rank - share_of(edge)))
        return out


def attend(q: Tensor, k: Tensor, v: Tensor, positions: list[int], scale: float, max_partials: int, sms: int, ranks: int) -> Tensor:
    """q [B, Hq, D], k and v [B, T, Hkv, D] with the tokens' own rows at ``positions``: every share's parts, merged."""
    B, Hq, D = q.shape
    Hkv = k.shape[2]
    line = LineUp.of(positions, Hkv, D, max_partials, sms)
    run, gqa = STAGE_ELEMENTS // D // line.heads, Hq // Hkv
    parts: dict[tuple[int, int], list[tuple[Tensor, Tensor]]] = {}
    for rank in range(ranks):
        for p in line.pieces(rank, ranks):
            rows = list(range(p.first * run, min(p.last * run, positions[p.seq]))) + [positions[p.seq]] * (p.last == p.stages)
            for head in range(p.head * gqa, (p.head + p.heads) * gqa):
                score = k[p.seq, rows, head // gqa].double() @ q[p.seq, head].double() * scale
                parts.setdefault((p.seq, head), []).append((torch.logsumexp(score, 0), torch.softmax(score, 0) @ v[p.seq, rows, head // gqa].double()))
    out = torch.zeros(B, Hq, D, dtype=torch.float64)
    for (seq, head), rows in parts.items():
        weights = torch.softmax(torch.stack([lse for lse, _ in rows]), 0)
        out[seq, head] = sum(w * o for w, (_, o) in zip(weights, rows))
    return out
