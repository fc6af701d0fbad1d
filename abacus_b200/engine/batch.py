"""The rows of one step, as the kernels see them.

A step carries, for each sequence, its next tokens (a whole prompt, or one
token), flattened into rows. Token-parallel kernels see only the rows; the
mixers and the cache write also read which sequence and position a row belongs
to. All index arrays of a step live in one int32 buffer, filled on the host and
sent to the device in one copy.

Rows beyond the step's tokens (padding up to a fixed size, for a captured
graph) carry sequence index -1; kernels skip them and no result depends on them.

A mixer whose kernels need more than these arrays (work lists, tiles, whatever it
derives from the step's sequences on the host) brings a *step plan*: an object with
    name                              what the mixer looks its part of the step up by
    layout(n_rows, n_seqs) -> layout  an object with `.words`, the int32 words the plan needs at most in a
                                      StepBatch with this room, and whatever else the plan wants to remember
                                      about such a StepBatch (offsets of its lists)
    fill(layout, sequences, words, is_decode, exact) -> info
                                      writes its words (a numpy view of the host buffer) and returns
                                      what the mixer wants to know on the host (counts and the like)
The plan's words travel in the same buffer, at an address that is fixed for the StepBatch's
life (a captured graph holds it); `batch.plan[name]` gives the mixer its words on the device
with its layout and the info of the last fill. Nothing here knows what any plan holds.
"""
import struct
from dataclasses import dataclass

import numpy as np
import torch


@dataclass
class Sequence:
    """One sequence's share of a step."""
    slot: int
    tokens: list  # its next tokens
    start: int  # how many tokens the slot already holds
    want: list  # places among `tokens` whose logits are wanted


@dataclass
class PlanView:
    """A step plan's part of a filled StepBatch."""
    plan: object
    layout: object
    words: torch.Tensor  # int32, on the device, at a fixed address
    info: object         # what the plan's fill returned


def _put_words(words, at, values):
    """words[at:at + len(values)] = values; a list of ints goes in packed (a third of what numpy takes for it)."""
    if type(values) is list and len(values) >= 64:
        try:
            struct.pack_into(f"{len(values)}i", words, 4 * at, *values)
            return
        except struct.error:  # (something numpy converts and struct does not, or refuses in its own words)
            pass
    words[at:at + len(values)] = values


CORE = ["tokens", "token_seq", "token_pos", "seq_slot", "seq_start", "seq_pos0", "seq_len_after", "logit_rows"]


class StepBatch:
    """Device-side index arrays of a step, with room for n_rows rows and n_seqs sequences."""

    def __init__(self, n_rows, n_seqs, n_logit_rows, device, plans=()):
        """plans: the step plans of the model's mixers (see above), each under a name of its own."""
        self.device = torch.device(device)
        self.cap_rows, self.cap_seqs, self.cap_logits = n_rows, n_seqs, max(1, n_logit_rows)
        self.plans = {}
        for p in plans:
            self.plans.setdefault(p.name, p)
        sizes = [n_rows, n_rows, n_rows, n_seqs, n_seqs + 1, n_seqs, n_seqs, self.cap_logits]
        self._layouts = {name: p.layout(n_rows, n_seqs) for name, p in self.plans.items()}
        sizes += [max(1, int(self._layouts[name].words)) for name in self.plans]
        offsets = np.concatenate([[0], np.cumsum([-(-s // 4) * 4 for s in sizes])])  # 16-byte aligned parts
        self._host = torch.zeros(int(offsets[-1]), dtype=torch.int32)
        if self.device.type == "cuda":
            self._host = self._host.pin_memory()
        self._dev = torch.zeros(int(offsets[-1]), dtype=torch.int32, device=self.device)
        names = CORE + [f"plan:{name}" for name in self.plans]
        self._h, self._parts = {}, {}
        for name, off, size in zip(names, offsets[:-1], sizes):
            self._h[name] = self._host[int(off):int(off) + size].numpy()
            self._parts[name] = self._dev[int(off):int(off) + size]
        for name in CORE:
            setattr(self, name, self._parts[name])
        self.plan = {}
        self.n_rows = n_rows
        self.n_tokens = self.n_seqs = self.n_logit_rows = 0
        self.max_position = 0
        self.max_len_after = 0
        self.longest = 0  # tokens of the sequence that brings most
        self.is_decode = False
        self.any_continuation = False
        self._sent, self._sent_on = None, set()

    def fill(self, sequences, pad_logits=False, exact=False):
        """Write the step described by `sequences` (list of Sequence) and send it to the device.
        pad_logits: logits are made for as many rows as this StepBatch has room for (a captured graph
        needs a fixed number); the rows beyond the wanted ones repeat row 0 and are ignored.
        exact: the step has as many rows, sequences and logit rows as `sequences` bring, not as many as
        there is room for (an engine keeps one StepBatch for steps of every size)."""
        h = self._h
        if self._sent is not None:
            self._sent.synchronize()  # the last copy must have read the host buffer before it is rewritten
        lens, starts, wants = [len(s.tokens) for s in sequences], [s.start for s in sequences], [s.want for s in sequences]
        n_tokens, n_logits = sum(lens), sum(map(len, wants))
        if n_tokens > self.cap_rows or len(sequences) > self.cap_seqs or n_logits > self.cap_logits:
            raise ValueError("step is larger than this StepBatch")
        n_seqs = len(sequences)
        lens_a, starts_a = np.array(lens, dtype=np.int64), np.array(starts, dtype=np.int64)
        ends = np.cumsum(lens_a)
        first = ends - lens_a
        one_each = n_tokens == n_seqs and (n_seqs == 0 or min(lens) == 1)
        if one_each:  # a decode step: a row a sequence
            h["tokens"][:n_seqs] = [s.tokens[0] for s in sequences]
            h["token_seq"][:n_seqs] = np.arange(n_seqs)
            h["token_pos"][:n_seqs] = starts_a
        elif n_seqs == 1:
            _put_words(h["tokens"], 0, sequences[0].tokens)
            h["token_seq"][:n_tokens] = 0
            h["token_pos"][:n_tokens] = np.arange(starts[0], starts[0] + n_tokens)
        else:
            for s, row in zip(sequences, first.tolist()):
                _put_words(h["tokens"], row, s.tokens)
            h["token_seq"][:n_tokens] = np.repeat(np.arange(n_seqs), lens_a)
            h["token_pos"][:n_tokens] = np.arange(n_tokens) + np.repeat(starts_a - first, lens_a)
        if n_tokens < self.cap_rows:
            h["tokens"][n_tokens:] = 0
            h["token_seq"][n_tokens:] = -1
            h["token_pos"][n_tokens:] = 0
        lens_after = starts_a + lens_a
        for name, values in (("seq_slot", [s.slot for s in sequences]), ("seq_pos0", starts_a), ("seq_len_after", lens_after)):
            h[name][:n_seqs] = values
            if n_seqs < self.cap_seqs:
                h[name][n_seqs:] = 0
        h["seq_start"][:n_seqs] = first
        h["seq_start"][n_seqs:] = n_tokens
        logit_rows = []
        if n_logits:
            for want, n, row in zip(wants, lens, first.tolist()):
                for wpos in want:
                    if not 0 <= wpos < n:
                        raise ValueError(f"wanted place {wpos} is outside the {n} tokens given")
                    logit_rows.append(row + wpos)
            h["logit_rows"][:n_logits] = logit_rows
        h["logit_rows"][n_logits:] = 0
        self.n_tokens, self.n_seqs, self.n_logit_rows = n_tokens, len(sequences), n_logits
        if pad_logits:
            self.n_logit_rows = self.cap_logits
        if exact:
            self.n_rows = n_tokens
            for name, n in (("tokens", n_tokens), ("token_seq", n_tokens), ("token_pos", n_tokens), ("seq_slot", n_seqs),
                            ("seq_start", n_seqs + 1), ("seq_pos0", n_seqs), ("seq_len_after", n_seqs),
                            ("logit_rows", max(1, n_logits))):
                whole = self._parts[name]
                setattr(self, name, whole if whole.shape[0] == n else whole[:n])
        self.sequences = list(sequences)  # host view, for mixers that walk the sequences themselves
        self.is_decode = one_each
        self.longest = 1 if one_each else max(lens, default=0)
        for name, p in self.plans.items():
            info = p.fill(self._layouts[name], self.sequences, h[f"plan:{name}"], self.is_decode, exact)
            self.plan[name] = PlanView(p, self._layouts[name], self._parts[f"plan:{name}"], info)
        self.max_position = int(lens_after.max()) - 1 if n_seqs else 0
        self.max_len_after = self.max_position + 1
        self.any_continuation = n_seqs > 0 and max(starts) > 0
        self._send()
        return self

    def _send(self):
        """The host's words to the device, in the order of the device's current stream."""
        # The first copy on a stream is torch's: its allocator then keeps the pinned words, should they be freed, until that stream has read
        # them. A copy and an event by torch cost the host four times as long, so the later ones go straight to the runtime.
        index = self._dev.get_device()
        if index >= 0:
            stream = torch._C._cuda_getCurrentRawStream(index)
            if stream in self._sent_on and index == torch.cuda.current_device():
                from ..kernels import ops
                ops.send_words(self._dev, self._host, self._sent)
                return
            self._sent_on.add(stream)
        self._dev.copy_(self._host, non_blocking=True)
        if self.device.type == "cuda":
            # (the event stays with the batch's device, whichever device is the current one)
            self._sent = self._sent or torch.cuda.Event()
            self._sent.record(torch.cuda.current_stream(self._dev.device))

    def advance_on_device(self):
        """Every sequence moves one position on (a decode step follows a decode step); the tokens are
        left as they are on the device. The host's view follows."""
        from ..kernels import ops
        ops.advance_decode(self)
        for s in self.sequences:
            s.start += 1
        self.max_position += 1
        self.max_len_after += 1
        self.any_continuation = True
        return self
