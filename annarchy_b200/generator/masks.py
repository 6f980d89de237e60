"""Small spiking networks on one thread-block cluster, every warp on its own.

CTA r owns the neurons [r * chunk, (r + 1) * chunk) of every population, a
warp 32 of them, a lane one, whose state stays in registers for a whole run.
The CTA's shared memory holds, per pre-synaptic neuron and warp, a 32-bit mask
of the lanes it has a synapse on; all synapses of a projection carry one
weight. A step of a warp:

  1. wait until every warp's spikes of the previous step have arrived in this
     CTA's copy of the spike bitmaps (an mbarrier counting the bytes from the
     other CTAs and one arrival per own warp);
  2. every lane takes a few words of the bitmap and loads the mask of the spike
     it finds; the masks that are not empty are packed into a short list per
     projection (a second round takes the second spikes of the words, and so
     on), and every lane adds the projection's weight once per listed mask with
     its bit. The reference adds them in ascending pre rank (ANNarchy/generator/
     Projection/OpenMP/CSR.py:870-902): with one weight per projection that is
     the same sequence of additions;
  3. update its neurons, store the ballot of the new spikes in the own copy
     and send it to every other CTA (st.async: the bytes land and are counted
     in one trip).

Synaptic delays (the network is the grid engine's by name, and keeps its
arrays): a lane counts, per projection, the events that arrive in each of the
coming steps (16 bits per neuron and step, all of one weight), and adds the
weight as often as counted when the step comes. Delays per synapse lie next to
the masks, one byte per synapse, found by the first position of a row's warp
and the mask's bits below the lane's; where they do not fit, a byte per pair of
neurons in global memory (14 MB, in L2, for 4000 neurons on 16 CTAs). The spike
history stays in memory as the other engines keep it; a run begins by going
through the steps whose spikes may still be on their way, so delays, times and
states set between runs act as they do there. Weights that become different
send the network to the grid engine's plan.

No CTA or cluster barrier in the loop: a warp that has received all words of
step s knows that every warp has finished reading those of step s - 1, so two
copies of the bitmaps (by step parity) are enough. What bounds a step is this
chain, and the instructions of eight warps per SM: the control flow is
uniform, since forms in which the warp went through the spikes one after
another (100 cycles per spike), lanes looped over their own spikes (shared-
memory counters: 1000 cycles) or one warp listed them for the CTA were slower.

Measured per step against the form with a cluster barrier per step and the
synapses listed per pre-synaptic neuron (CodeGenerator.cluster_module, which
remains for projections with several weights and for larger populations): 4000
neurons, 8 spikes per step 1.19 us (2.56) in double and 0.99 us (1.69) in single
precision; 1000 neurons 0.66 and 0.46 us; 400 neurons 0.62 and 0.44 us. With delays, against
the grid engine's launches per step: 3000 neurons, 1 to 20 steps per synapse,
1.8 us (9.4) in double precision (2.0 with the delays in global memory and a
list per projection); 400 neurons, uniform, 1.1 (7.4) in double and 0.7 (5.4) in
single precision. Runs of one step take 95 to 130 us with the wait
(144 to 146 us through the plan), so every run length gains.

A step costs about one mask per spike and warp, so that very active networks gain
less, and with delays lose: 3000 neurons with 60 synapses each, 1 % / 5 % / 20 % of
the neurons spiking in a step, us per step here and through the plan: uniform
delays 1.5, 3.0, 7.3 and 5.2, 5.4, 6.0 in double, 1.4, 2.9, 7.2 and 6.3, 8.0, 12.0
in single precision; delays per synapse 3.0, 9.0, 28 and 8.3, 11.2, 16.3 in double,
3.0, 9.0, 28 and 6.2, 6.4, 7.0 in single precision.
"""
from __future__ import annotations

import re

import numpy as np

from .codegen import CodeGenerator, Module, compensated_vars

SMEM_LIMIT = 220 * 1024
MAX_WORDS = 256            # bitmap words of a population (8 per lane)


class Masks:
    def __init__(self, c):
        self.c = c
        self.net = c.net

    def possible(self) -> bool:
        """One weight per projection, populations of up to 8192 neurons."""
        net = self.net
        if any((p.size + 31) // 32 > MAX_WORDS for p in net.populations):
            return False
        for p in net.projections:
            d = p._csr.data
            if d.size and not np.all(d == d[0]):
                return False
            # (a mask has one bit per pair of neurons)
            if any(np.unique(x).size != np.size(x) for x in (p.pre_ranks, p.post_ranks_view)):
                return False
        return True

    def slots(self):
        """Projections grouped into mask tables: one joins the table before it
        when both populations are the same and their pre-synaptic words are
        disjoint. Tables keep the projections' order. Without delays the
        projections of a table are added round by round, so that two of one
        target would mix their additions: each then has its own table. (With
        delays the events are counted and added projection by projection.)"""
        out = []
        delayed = any(p.max_delay > 1 for p in self.net.projections)
        for p in self.net.projections:
            lay = self.c.layout[p.id]
            w0, w1 = lay["w0"], lay["w1"]
            if out:
                s = out[-1]
                if s["pre"] is p.pre_pop and s["post"] is p.post_pop and all(
                        (w1 <= a or b <= w0) and (delayed or q.target != p.target)
                        for q, a, b in s["projs"]):
                    s["projs"].append((p, w0, w1))
                    s["w0"], s["w1"] = min(s["w0"], w0), max(s["w1"], w1)
                    continue
            out.append({"pre": p.pre_pop, "post": p.post_pop, "projs": [(p, w0, w1)], "w0": w0, "w1": w1})
        return out

    def layout(self, C: int):
        """Shared memory of a CTA of a C-CTA cluster, or None."""
        a16 = lambda x: (int(x) + 15) // 16 * 16
        off, lay = 64, {"pop": {}, "slots": self.slots()}             # two mbarriers first
        # with delays: counters of the events arriving in the next steps
        delayed = any(p.max_delay > 1 for p in self.net.projections)
        lay["S"] = S = max(self.c.slots.values()) + 1 if delayed else 0
        for pop in self.net.populations:
            chunk = -(-(-(-pop.size // C)) // 32) * 32
            words = (pop.size + 31) // 32
            per = -(-words // 32)                                     # words a lane takes
            d = {"chunk": chunk, "words": words, "per": per, "rep": []}
            for _ in (0, 1):
                d["rep"].append(off)
                off += a16(per * 32 * 4)
            # with delays: the steps before the run
            ring = self.c.slots.get(pop.id, 1)
            d["hist"] = off
            if ring > 1:
                off += a16(ring * words * 4)
            lay["pop"][pop.id] = d
        lay["block"] = max(d["chunk"] for d in lay["pop"].values())
        if lay["block"] > 1024:
            return None
        # no CTA without neurons: one that sends nothing would not be waited for
        lay["C"] = max(-(-p.size // lay["pop"][p.id]["chunk"]) for p in self.net.populations)
        for s in lay["slots"]:
            s["warps"] = lay["pop"][s["post"].id]["chunk"] // 32
            s["rows"] = (s["w1"] - s["w0"]) * 32
            s["off"], off = off, off + a16(s["rows"] * s["warps"] * 4)
            # per warp and projection, the masks of one round
            s["cap"] = lay["pop"][s["pre"].id]["per"] * 32 + 8
            # (one list, with the positions of the delays, for all projections with delays per synapse)
            s["synapse"] = [q for q, (p, _, _) in enumerate(s["projs"]) if p._delay_steps is not None]
            s["lists"] = len(s["projs"]) - len(s["synapse"]) + (2 if s["synapse"] else 0)
            s["list"], off = off, off + 4 * s["cap"] * s["lists"] * s["warps"]
            s["cnt"], off = off, off + a16(2 * S * 32 * s["warps"] * len(s["projs"]))
        if off > SMEM_LIMIT:
            return None
        for s in lay["slots"]:
            # the delays of the synapses next to the masks, where they fit
            s["packed"] = False
            if s["synapse"]:
                positions, delays = self.packed(s, lay)
                n = delays.shape[1]
                more = a16(positions.shape[1] * 2) + a16(n)
                if n < 65536 and off + more <= SMEM_LIMIT:
                    s["packed"], s["nbytes"], s["arrays"] = True, n, (positions, delays)
                    s["pos"], off = off, off + a16(positions.shape[1] * 2)
                    s["bytes"], off = off, off + a16(n)
        lay["smem"] = off
        return lay

    def choose(self):
        """Layouts to try, the preferred one first: about 128 neurons per CTA
        (four warps: one per scheduler), at most 16 CTAs. 1000 neurons on 1, 2,
        4, 8 and 16 CTAs: 1.37, 0.82, 0.70, 0.66, 0.69 us per step in double."""
        want = self.net._config.get("cluster_size")
        if want:
            lays = [self.layout(int(want))]
        else:
            total = max(p.size for p in self.net.populations)
            first = next((c for c in (1, 2, 4, 8) if total <= 128 * c), 16)
            lays = (self.layout(c) for c in (1, 2, 4, 8, 16) if c >= first)
        return (x for x in lays if x)

    def tables(self, slot, lay):
        """(C x rows x warps) masks of a table."""
        chunk, W, rows = lay["pop"][slot["post"].id]["chunk"], slot["warps"], slot["rows"]
        m = np.zeros(lay["C"] * rows * W)
        for proj, _, _ in slot["projs"]:
            post_rank, row_ptr, cols, _ = proj.csr_population_ranks()
            post = np.repeat(post_rank, np.diff(row_ptr)).astype(np.int64)
            q = post % chunk
            idx = ((post // chunk) * rows + (cols - 32 * slot["w0"])) * W + (q >> 5)
            m += np.bincount(idx, weights=np.ldexp(1.0, (q & 31).astype(np.int32)), minlength=m.size)
        return m.astype(np.uint32)

    def create_arrays(self, lay):
        nat = self.c.native
        for i, s in enumerate(lay["slots"]):
            nat.create(f"net__masks{i}", self.tables(s, lay))
            for proj, _, _ in s["projs"]:
                w = proj._csr.data
                nat.create(f"proj{proj.id}__mw", self.c._w(np.array([w[0] if w.size else 0.0])))
            self._delay_arrays(i, s, lay, nat.create)
        self.lay = lay

    def free_arrays(self):
        for name in [n for n in self.c.native.arrays if n.startswith("net__") or n.endswith("__mw")]:
            self.c.native.free(name)

    def _delay_arrays(self, i, slot, lay, put):
        if slot["packed"]:
            positions, delays = slot.pop("arrays", None) or self.packed(slot, lay)
            put(f"net__dpos{i}", positions.reshape(-1))
            put(f"net__dby{i}", delays.reshape(-1))
        elif slot["synapse"]:
            put(f"net__dby{i}", self.delays(slot, lay))

    def _synapses(self, slot, lay):
        """((CTA x row x lane) index, delay) of the synapses of a table's
        projections with delays per synapse."""
        chunk, at, steps = lay["pop"][slot["post"].id]["chunk"], [], []
        for q in slot["synapse"]:
            proj = slot["projs"][q][0]
            post_rank, row_ptr, cols, _ = proj.csr_population_ranks()
            post = np.repeat(post_rank, np.diff(row_ptr)).astype(np.int64)
            at.append(((post // chunk) * slot["rows"] + (cols - 32 * slot["w0"])) * chunk + post % chunk)
            steps.append(np.asarray(proj._delay_steps))
        return np.concatenate(at), np.concatenate(steps)

    def delays(self, slot, lay):
        """(C x rows x chunk) delays (steps, one byte each; at most 63)."""
        d = np.zeros(lay["C"] * slot["rows"] * lay["pop"][slot["post"].id]["chunk"], dtype=np.uint8)
        at, steps = self._synapses(slot, lay)
        d[at] = steps
        return d

    def packed(self, slot, lay):
        """Per CTA the first positions (rows x warps) and the delays of the
        synapses in the order of rows and lanes."""
        C, per = lay["C"], slot["rows"] * slot["warps"]
        at, steps = self._synapses(slot, lay)
        order = np.argsort(at, kind="stable")
        count = np.bincount(at // 32, minlength=C * per).reshape(C, per)
        total = count.sum(axis=1)
        first = np.cumsum(count, axis=1) - count
        d = np.zeros((C, int(total.max())), dtype=np.uint8)
        ends = np.cumsum(total)
        for c in range(C):
            d[c, :total[c]] = steps[order[ends[c] - total[c]:ends[c]]]
        return first.astype(np.uint16), d

    def write_delays(self, proj):
        """The delays set after compile() (uniform ones are read from their
        array at the start of a run)."""
        for i, s in enumerate(self.lay["slots"]):
            if any(s["projs"][q][0] is proj for q in s["synapse"]):
                self._delay_arrays(i, s, self.lay, self.c.native.write)

    def write_weights(self, proj) -> bool:
        """The weights set after compile(); False when they differ."""
        w = proj._csr.data
        if not w.size:
            return True
        if not np.all(w == w[0]):
            return False
        self.c.native.write(f"proj{proj.id}__mw", self.c._w(np.array([w[0]])))
        return True

    def module(self, lay) -> Module:
        # (the update code of a kernel that neither lists spikes nor has inboxes)
        c = self.c
        lists, inbox = c.spike_lists, c.inbox
        c.spike_lists, c.inbox = False, set()
        try:
            return self._module(lay, lists)
        finally:
            c.spike_lists, c.inbox = lists, inbox

    def _module(self, lay, lists: bool) -> Module:
        c, net = self.c, self.net
        gen = CodeGenerator(c)
        R, C, block = gen.real, lay["C"], lay["block"]
        regs, load, store, ranges, ups, deliver, words_sent = [], [], [], [], [], "", 0
        for pop in net.populations:
            k, d = pop.id, lay["pop"][pop.id]
            words_sent += d["words"]
            ranges += [f"const int anb_base{k} = (int)anb_rank * {d['chunk']};",
                       f"const int anb_cnt{k} = max(0, min({pop.size} - anb_base{k}, {d['chunk']}));",
                       f"anb_u32* const anb_rep{k}0 = reinterpret_cast<anb_u32*>(anb_smem + {d['rep'][0]});",
                       f"anb_u32* const anb_rep{k}1 = reinterpret_cast<anb_u32*>(anb_smem + {d['rep'][1]});"]
            spk = gen.ptr(f"pop{k}__spk")
            ring = c.slots.get(k, 1)
            # the spikes before the run are read from the bitmaps in memory
            last = f"{spk} + (size_t)anb_ring_slot(anb_t0 - 1, {ring}) * {d['words']}"
            load.append(f"#pragma unroll 1\n    for (int q = threadIdx.x; q < {32 * d['per']}; q += {block}) {{ "
                        f"anb_rep{k}1[q] = q < {d['words']} ? ({last})[q] : 0u; anb_rep{k}0[q] = 0u; }}")
            if ring > 1:
                load.append(f"#pragma unroll 4\n    for (int q = threadIdx.x; q < {ring * d['words']}; q += {block}) "
                            f"reinterpret_cast<anb_u32*>(anb_smem + {d['hist']})[q] = {spk}[q];")
            if lists and lay["S"]:
                # (the grid engine's spike lists are emptied when the time is set)
                spn = gen.ptr(f"pop{k}__spn")
                regs.append(f"const bool anb_had{k} = {spn}[(anb_t0 - 1) & 1] != 0;")
                store.append(f"if (anb_rank == 0 && threadIdx.x < 2) {spn}[threadIdx.x] = 1;")
            if ring == 1:
                store.append(f"if (anb_tid < anb_cnt{k} && anb_lane == 0) {spk}[(anb_base{k} + anb_tid) >> 5] = "
                             f"(anb_steps & 1 ? anb_rep{k}0 : anb_rep{k}1)[(anb_base{k} + anb_tid) >> 5];")
            smem = {}
            names = [(n, "int" if pop._ctype.get(n) in ("int", "bool") else R) for n in c._local_vars(pop)]
            names.append(("refractory_remaining", "int"))
            if pop._has_refractory:
                names.append(("refractory", "int"))
            names += [("kc_" + n, R) for n in compensated_vars(pop, c.exact, net._config)]
            for n, ct in names:
                reg = f"anb_rg{k}_{n}"
                smem[n] = reg
                regs.append(f"{ct} {reg} = ({ct})0;")
                if n.startswith("kc_") and not lay["S"]:
                    continue        # without delays a run starts without carried errors
                g = gen.ptr(f"pop{k}__{n}")
                load.append(f"if (anb_tid < anb_cnt{k}) {reg} = {g}[anb_base{k} + anb_tid];")
                if n != "refractory":
                    store.append(f"if (anb_tid < anb_cnt{k}) {g}[anb_base{k} + anb_tid] = {reg};")
            ups.append(self._update(gen, pop, smem, lay))
        for i, s in enumerate(lay["slots"]):
            a, b = s["pre"].id, s["post"].id
            per = lay["pop"][a]["per"]
            n4 = s["rows"] * s["warps"]
            load.append(f"#pragma unroll 4\n    for (int q = threadIdx.x; q < {n4}; q += {block}) "
                        f"reinterpret_cast<anb_u32*>(anb_smem + {s['off']})[q] = "
                        f"{gen.ptr(f'net__masks{i}')}[(size_t)anb_rank * {n4} + q];")
            regs.append(f"const anb_u32* const anb_mask{i} = reinterpret_cast<const anb_u32*>(anb_smem + {s['off']}) + anb_warp;")
            regs.append(f"anb_u32* const anb_li{i} = reinterpret_cast<anb_u32*>(anb_smem + {s['list']}) + "
                        f"anb_warp * {s['cap'] * s['lists']};")
            S, chunk = lay["S"], lay["pop"][b]["chunk"]
            if S:
                n2 = S * chunk * len(s["projs"])
                load.append(f"#pragma unroll 1\n    for (int q = threadIdx.x; q < {n2}; q += {block}) "
                            f"reinterpret_cast<unsigned short*>(anb_smem + {s['cnt']})[q] = 0;")
            pack, adds, drain, place = "", "", "", ""
            uniform = [q for q in range(len(s["projs"])) if q not in s["synapse"]]
            if s["synapse"]:
                dby = f"anb_li{i} + {len(uniform) * s['cap']}"
                dat = f"anb_li{i} + {(len(uniform) + 1) * s['cap']}"
                pack += """
            int anb_nd = 0;"""
                if s["packed"]:
                    n16 = s["rows"] * s["warps"]
                    for what, ct, at, n in (("dpos", "unsigned short", s["pos"], n16),
                                            ("dby", "unsigned char", s["bytes"], s["nbytes"])):
                        load.append(f"#pragma unroll 4\n    for (int q = threadIdx.x; q < {n}; q += {block}) "
                                    f"reinterpret_cast<{ct}*>(anb_smem + {at})[q] = "
                                    f"{gen.ptr(f'net__{what}{i}')}[(size_t)anb_rank * {n} + q];")
                    regs.append(f"const unsigned short* const anb_dp{i} = "
                                f"reinterpret_cast<const unsigned short*>(anb_smem + {s['pos']}) + anb_warp;")
                    row = f"(int)anb_dp{i}[anb_row * {s['warps']}]"
                    where = f"anb_smem + {s['bytes']}, 0"
                else:
                    row = "anb_row"
                    where = f"{gen.ptr(f'net__dby{i}')} + (size_t)anb_rank * {s['rows'] * chunk} + anb_tid, {chunk}"
                # the delays' position, and above it the projection
                place = f"""
              anb_r[j] = 0;
              if (anb_m[j]) {{
                const int anb_row = (j * 32 + anb_lane) * 32 + __ffs(anb_x[j]) - {s['w0'] * 32 + 1};
                anb_r[j] = {row}{''.join(f" + (j * 32 + anb_lane >= {s['projs'][q][1]} && j * 32 + anb_lane < {s['projs'][q][2]} ? {q << 24} : 0)" for q in s["synapse"] if q)};
              }}"""
                adds += f"""
            anb_mask_delays<{'true' if s['packed'] else 'false'}>({dby}, {dat}, anb_nd, {where},
                            reinterpret_cast<anb_u32*>(anb_smem + {s['cnt']}), {S * chunk}, {chunk},
                            anb_cur - 1, {S}, 1 - anb_s);"""
            for q, (proj, w0, w1) in enumerate(s["projs"]):
                pk = proj.id
                regs.append(f"const {R} anb_w{pk} = ({R})anb_wf({gen.ptr(f'proj{pk}__mw')}[0]);")
                synapse = q in s["synapse"]
                n, at = ("anb_nd", dby) if synapse else (f"anb_n{q}", f"anb_li{i} + {uniform.index(q) * s['cap']}")
                if not synapse:
                    pack += f"""
            int anb_n{q} = 0;"""
                for j in range(w0 // 32, (w1 - 1) // 32 + 1):
                    # (words outside the projection's range belong to others)
                    inside = "" if w0 <= 32 * j and 32 * j + 32 <= w1 else \
                        f" && anb_lane >= {max(0, w0 - 32 * j)} && anb_lane < {min(32, w1 - 32 * j)}"
                    if synapse:
                        pack += f"""
            {{ int n = anb_nd; anb_pack((anb_u32)anb_r[{j}], anb_m[{j}] != 0u{inside}, {dat}, &n); }}"""
                    pack += f"""
            anb_pack(anb_m[{j}], anb_m[{j}] != 0u{inside}, {at}, &{n});"""
                if not synapse:
                    pack += f"""
            if (anb_lane < 4) ({at})[anb_n{q} + anb_lane] = 0u;"""
                g = f"anb_rg{b}_g_{proj.target}"
                if not S:
                    adds += f"""
            {g} = anb_mask_add({g}, anb_w{pk}, {at}, anb_n{q});  // {proj.name}"""
                    continue
                cnt = f"anb_cn{i} + {q * S * chunk}"
                drain += f"""
          {g} = anb_mask_drain({g}, anb_w{pk}, {cnt} + anb_cur * {chunk});  // {proj.name}"""
                if synapse:
                    continue
                least = "1 - anb_s"
                if proj.max_delay > 1:
                    regs.append(f"const int anb_d{pk} = {gen.ptr(f'proj{pk}__delay')}[0];")
                else:
                    regs.append(f"const int anb_d{pk} = 1;")
                    if lists:
                        least = f"(anb_s > 0 || anb_had{a} ? 1 - anb_s : 2)"
                adds += f"""
            if (anb_d{pk} >= {least}) {{  // {proj.name}
              const int c = anb_mask_add(0, 1, {at}, anb_n{q}), at = anb_cur - 1 + anb_d{pk};
              if (c) ({cnt})[(at >= {S} ? at - {S} : at) * {chunk}] += (unsigned short)c;
            }}"""
            if s["synapse"]:
                pack += f"""
            if (anb_lane < 8) ({dby})[anb_nd + anb_lane] = 0u;
            if (anb_lane < 8) ({dat})[anb_nd + anb_lane] = 0u;"""
            if S:
                regs.append(f"unsigned short* const anb_cn{i} = reinterpret_cast<unsigned short*>(anb_smem + {s['cnt']}) + anb_tid;\n    (void)anb_cn{i};")
            word = "anb_rep[j * 32 + anb_lane]"
            used = [(w0, w1) for _, w0, w1 in s["projs"]]
            if len(used) != 1 or used[0] != (0, lay["pop"][a]["words"]):
                word = " || ".join(f"(j * 32 + anb_lane >= {w0} && j * 32 + anb_lane < {w1})"
                                   for w0, w1 in used) + " ? " + word + " : 0u"
            any_x = " | ".join(f"anb_x[{j}]" for j in range(per))
            rowdecl = f"\n          int anb_r[{per}];" if s["synapse"] else ""
            if drain:
                drain = f"""
          if (anb_s >= 0) {{{drain}
          }}"""
            ring, words = c.slots.get(a, 1), lay["pop"][a]["words"]
            inside = " || ".join(f"(i >= {w0} && i < {w1})" for w0, w1 in used)
            history = f"-anb_s < {ring} && ({inside}) ? anb_hist[i] : 0u" if ring > 1 else "0u"
            earlier = f"""
          if (anb_s < 0) {{
            // steps before the run: spikes still on their way
            const anb_u32* anb_hist = reinterpret_cast<const anb_u32*>(anb_smem + {lay['pop'][a]['hist']}) +
                                      {f'(anb_at{a} == 0 ? {ring - 1} : anb_at{a} - 1)' if ring > 1 else '0'} * {words};
            (void)anb_hist;
#pragma unroll
            for (int j = 0; j < {per}; ++j) {{
              const int i = j * 32 + anb_lane;
              anb_x[j] = {history};
            }}
          }}""" if lay["S"] else ""
            deliver += f"""
        if (anb_warp < {s['warps']}) {{  // population {a}'s spikes of the previous step (word j * 32 + lane: lane's j-th)
          const anb_u32* anb_rep = (anb_s & 1) ? anb_rep{a}0 : anb_rep{a}1;
          anb_u32 anb_x[{per}], anb_m[{per}];{rowdecl}
#pragma unroll
          for (int j = 0; j < {per}; ++j) anb_x[j] = {word};{earlier}
#pragma unroll 1
          while (__any_sync(0xffffffffu, ({any_x}) != 0u)) {{
            // the mask of each word's first spike
#pragma unroll
            for (int j = 0; j < {per}; ++j) {{
              anb_m[j] = anb_x[j] ? anb_mask{i}[((j * 32 + anb_lane) * 32 + __ffs(anb_x[j]) - {s['w0'] * 32 + 1}) * {s['warps']}] : 0u;{place}
              anb_x[j] &= anb_x[j] - 1u;
            }}{pack}
            __syncwarp();{adds}
            __syncwarp();
          }}{drain}
        }}"""
        globals_ = [gen._scoped_globals(p)[0] for p in net.populations]
        mon_pre = "\n    ".join(
            f"const int anb_mon_on{m.id} = {gen.ptr(f'mon{m.id}__on')}[0];\n    "
            f"const long long anb_sl{m.id} = anb_t0 - {gen.ptr(f'mon{m.id}__t0')}[0];\n    "
            f"const int anb_slot0{m.id} = anb_sl{m.id} < -(1 << 30) || anb_sl{m.id} > (1 << 30) ? -(1 << 30) : (int)anb_sl{m.id};"
            for m in net.monitors)
        dt_t = "double" if c.exact else "float"
        warps = f"anb_cnt{net.populations[0].id}"
        for p in net.populations[1:]:
            warps = f"max({warps}, anb_cnt{p.id})"
        # with delays the steps before the run that still matter come first
        S = lay["S"]
        start = f"anb_steps > 0 ? {2 - S} : 0" if S else "0"
        # (positions in the rings are counted: a 64-bit remainder is 100 cycles)
        cursor = f"""
        anb_cur = anb_cur + 1 == {S} ? 0 : anb_cur + 1;""" if S else ""
        rings = f"int anb_cur = anb_ring_slot(anb_t0 + ({start}) - 1, {S});" if S else ""
        for pop in net.populations:
            ring = c.slots.get(pop.id, 1)
            if ring > 1:
                rings += f"\n      int anb_at{pop.id} = anb_ring_slot(anb_t0 + ({start}) - 1, {ring});"
                cursor += f"""
        anb_at{pop.id} = anb_at{pop.id} + 1 == {ring} ? 0 : anb_at{pop.id} + 1;"""
        skip = """
        if (anb_s < 0) continue;""" if S else ""
        own = " + ".join(f"(anb_cnt{p.id} + 31) / 32" for p in net.populations)
        nl = "\n    "
        err = gen.ptr("err")
        src = f"""
extern "C" __global__ void __launch_bounds__({block}, 1) anb_cluster_run(long long anb_t0, int anb_steps) {{
    extern __shared__ __align__(16) unsigned char anb_smem[];
    const unsigned anb_rank = anb_cluster_rank();
    const {dt_t} dt = ({dt_t})(*{gen.ptr('dt')});
    const int anb_tid = threadIdx.x, anb_lane = threadIdx.x & 31, anb_warp = threadIdx.x >> 5;
    // mbarriers: the words of even and of odd steps
    const unsigned anb_bar = anb_smem_addr(anb_smem);
    {nl.join(ranges)}
    // lane c: CTA c's shared memory (the mbarriers at its start)
    const unsigned anb_peer = anb_cluster_map(anb_bar, anb_lane < {C} ? anb_lane : 0);
    (void)anb_peer;
    const int anb_warps = ({warps} + 31) / 32;
    const unsigned anb_bytes = 4u * ({words_sent} - ({own}));
    {nl.join(regs)}
    {nl.join(g for g in globals_ if g)}
    {mon_pre}
    if (threadIdx.x == 0) {{
      // a phase: thread 0 (the bytes to expect) and every warp with neurons
      anb_mbar_init(anb_bar, 1 + anb_warps);
      anb_mbar_init(anb_bar + 8, 1 + anb_warps);
      anb_mbar_expect(anb_bar, anb_bytes);
      anb_mbar_expect(anb_bar + 8, anb_bytes);
    }}
    {nl.join(load)}
    anb_cluster_sync();
    // (warps without neurons send nothing, so nobody waits for them: they stay out)
    if (anb_warp < anb_warps) {{
      {rings}
#pragma unroll 1
      for (int anb_s = {start}; anb_s < anb_steps; ++anb_s) {{
        const long long t = anb_t0 + anb_s;{cursor}
        if (anb_s > 0) {{
          // the words of step s - 1; the barrier's next phase takes those of s + 1
          const unsigned b = anb_bar + 8u * ((anb_s - 1) & 1);
          if (!anb_mbar_wait(b, ((anb_s - 1) >> 1) & 1, {err})) break;
          if (threadIdx.x == 0) anb_mbar_expect(b, anb_bytes);
        }}{deliver}{skip}
        {''.join(ups)}
        __syncwarp();
        if (anb_lane == 0) anb_mbar_arrive(anb_bar + 8u * (anb_s & 1));
      }}
      // the last step's words have arrived everywhere before any CTA leaves
      if (anb_steps > 0) anb_mbar_wait(anb_bar + 8u * ((anb_steps - 1) & 1), ((anb_steps - 1) >> 1) & 1, {err});
      {nl.join(store)}
    }}
    __syncwarp();
    anb_cluster_sync();
    if (anb_rank == 0 && threadIdx.x == 0) *{gen.ptr('t')} = anb_t0 + anb_steps;
}}
"""
        return Module(gen.assemble([src]), gen.options(), "cluster",
                      local=("anb_cluster_run", C, block, lay["smem"], C), kernels=["anb_cluster_run"])

    def _update(self, gen, pop, smem, lay) -> str:
        k, d = pop.id, lay["pop"][pop.id]
        send = "" if lay["C"] == 1 else f"""
          if (anb_lane != (int)anb_rank && anb_lane < {lay['C']})
            anb_st_async(anb_peer + anb_off, anb_m, anb_peer + 8u * (anb_s & 1));"""
        rec, keep, ring = "", "", self.c.slots.get(k, 1)
        if ring > 1:
            # the history ring in memory, as the other engines keep it
            keep = f"""
          if (anb_lane == 30)
            {gen.ptr(f'pop{k}__spk')}[anb_at{k} * {d['words']} + ((anb_base + anb_q) >> 5)] = anb_m;"""
        for m in self.net.monitors:
            if m.population is pop and "spike" in m.variables:
                ml = self.c.mon_layout[m.id]
                rec += f"""
          if (anb_lane == 31 && anb_mon_on{m.id}) {{
            const int anb_slot = anb_slot0{m.id} + anb_s;
            if (anb_slot >= 0 && anb_slot < {ml['cap_spike']})
              {gen.ptr(f'mon{m.id}__spk')}[(unsigned)anb_slot * {ml['words']}u + ((unsigned)(anb_base + anb_q) >> 5)] = anb_m;
            else
              anb_report({gen.ptr('err')}, ANB_DEVERR_MONITOR_OVERFLOW);
          }}"""
        hook = f"""
      {{
        const anb_u32 anb_m = __ballot_sync(0xffffffffu, anb_spiked);
        if (anb_q - anb_lane < anb_cnt) {{
          const unsigned anb_off = ((anb_s & 1) ? {d['rep'][1]}u : {d['rep'][0]}u) + 4u * (unsigned)((anb_base + anb_q) >> 5);
          if (anb_lane == (int)anb_rank) *reinterpret_cast<anb_u32*>(anb_smem + anb_off) = anb_m;{send}{keep}{rec}
        }}
      }}"""
        code = gen.neuron_update(pop, local_engine=True, smem=smem, cluster={}, ballot_hook=hook)
        code = f"{{ {gen._scoped_globals(pop)[1]}{code}}}"
        code = re.sub(r"(anb_rg\d+_\w+)\[anb_q\]", r"\1", code)
        # one pass over the CTA's neurons, whose state is a register each
        loop = "for (int anb_q0 = 0; anb_q0 < anb_cnt; anb_q0 += blockDim.x) {"
        names = f"const int anb_base = anb_base{k}, anb_cnt = anb_cnt{k};"
        assert code.count(loop) == code.count(names) == 1 and not re.search(r"anb_rg\d+_\w+\[", code)
        return code.replace(loop, "{ const int anb_q0 = 0;").replace(names, names + " (void)anb_base;")
