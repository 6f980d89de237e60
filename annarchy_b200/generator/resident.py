"""Rate-coded networks that stay on chip: one persistent kernel per run.

A step of a small or middle-sized rate-coded network is a few hundred
thousand multiplications; as separate launches (one weighted sum per
projection, the update, the recording) it is launch and load latency. Here
every CTA owns a slice of each population with its state and the incoming
synapses of its neurons in shared memory for the whole run, and a copy of
the rates its synapses read. A step is: weighted sums and update of the own
neurons, the new rates to everybody, one barrier. The reference runs the same
phases as separate loops over all neurons (ANNarchy/generator/Template/
OpenMPBaseTemplate.py:131-484).

Two forms:

* cluster - up to 16 CTAs of one thread-block cluster: the new rates are
            stored into every CTA's shared memory (double-buffered by step
            parity), then the hardware cluster barrier. For small networks
            (CLUSTER_SYNAPSES).
* grid    - one CTA per SM (cooperative launch): the new rates go through a
            double-buffered global array, then a grid-wide barrier (bounded),
            then every CTA copies them into its shared memory.

Double precision adds every row's products one by one in stored order, one
lane per row; single precision splits a row over `lanes` lanes.

Measured per step against one launch per phase (5.9 to 18 us): 500 neurons
with 12,000 synapses 1.4 us in double, 1.0 us in single precision; 5000
neurons with 0.72 million 4.7 and 2.7 us; 9000 neurons with 0.96 million 4.5
and 3.3 us. The grid-wide barrier and the copy of the rates are 1.9 us of it.
"""
from __future__ import annotations

import re

import numpy as np

from ..core.monitor import source_name, array_name
from .codegen import CodeGenerator, Module, compensated_vars, global_equations

SMEM_LIMIT = 220 * 1024
# one CTA per SM: more than half of an SM's shared memory
SMEM_ALONE = 118 * 1024
GRID_CTAS = 148
# Most synapses of a network on one cluster. us per step, 16 CTAs of a cluster
# against 148 CTAs: double, 135,000 synapses 2.9 and 3.2, 50,000: 1.9 and 2.5;
# single, 135,000: 3.7 and 2.1, 50,000: 1.6 and 2.0, 12,000: 1.1 and 1.8. (The
# engine of launches takes 5.8 to 9 us for these.)
CLUSTER_SYNAPSES = {"double": 160_000, "float": 64_000}


def unroll(lanes: int) -> int:
    """Steps whose loads are in flight together (anb_rate_row)."""
    return 8 if lanes == 1 else 4


def updated(pop) -> bool:
    return any(v.get("cpp") for v in pop.desc["variables"])


def possible(c) -> bool:
    """Rate-coded populations and plain weighted sums w * pre.r without
    delays, learning or storage formats chosen by the user; no equations or
    reductions over a whole population, stop conditions or input schedules;
    single-network runs (not shards or copies sharing weights)."""
    net = c.net
    if c.shard or not net.projections or net._config.get("persistent"):
        return False
    for p in net.populations:
        if (p.neuron_type.type != "rate" or hasattr(p, "_ta_schedule_ms") or global_equations(p)
                or p._globalops or getattr(p, "stop_condition", None) or c.slots.get(p.id, 1) > 1):
            return False
    if not any(updated(p) for p in net.populations):
        return False
    for p in net.projections:
        if (p.synapse_type.type != "rate" or getattr(p, "_batched", None) is not None
                or getattr(p, "_device_conn", None) or p._csr is None or p.max_delay > 1
                or p._delay_steps is not None or CodeGenerator.continuous_update(p)
                or CodeGenerator.custom_psp(p) or p.desc["variables"] and any(
                    v.get("cpp") for v in p.desc["variables"])
                or p._storage_format not in ("csr", "auto") or p.pre_pop.size > 65535
                or not updated(p.post_pop)):
            return False
    for m in net.monitors:
        names = [source_name(v) for v in m.variables]
        if any(not n.startswith("_last_sum_") and m.population._locality.get(n) != "local" for n in names):
            return False
        if m.ranks is not None and len(np.unique(m.ranks)) != len(m.ranks):
            return False
    return True


def _pow2(n) -> int:
    return 1 << max(0, int(np.ceil(np.log2(max(1, n)))))


class Resident:
    """Layout and kernel of one network."""

    def __init__(self, c):
        self.c = c
        self.net = c.net
        self.rb = np.dtype(c.real).itemsize
        self.wb = np.dtype(c.wdtype).itemsize
        self.pops = [p for p in self.net.populations if updated(p)]
        self.pres = {p.pre_pop.id: p.pre_pop for p in self.net.projections}
        self.nnz = sum(int(p._csr.nnz) for p in self.net.projections)
        self.state = {p.id: self._state(p) for p in self.pops}

    def _projs(self, pop):
        return [p for p in self.net.projections if p.post_pop is pop]

    def _state(self, pop):
        """(name, C type, stored back) of the attributes kept in shared memory."""
        gen = CodeGenerator(self.c)
        body, modified = gen._neuron_body(pop, None, False)
        rec = {source_name(v) for m in self.net.monitors if m.population is pop for v in m.variables}
        local = [p["name"] for p in pop.desc["parameters"] + pop.desc["variables"]
                 if p["locality"] == "local"]
        body += gen._random_draws(pop)
        out = []
        for n in local:
            if n == "r" or n in rec or re.search(rf"\b{re.escape(n)}\b", body):
                ct = "int" if pop._ctype.get(n) in ("int", "bool") else gen.real
                out.append((n, ct, n in modified))
        for n in compensated_vars(pop, self.c.exact, self.net._config):
            out.append(("kc_" + n, gen.real, True))
        for t in pop.targets:
            out.append(("_last_sum_" + t, gen.real, True))
        return out

    # ----------------------------------------------------------------- layout
    def layout(self, ctas: int, cluster: bool):
        """Offsets in a CTA's shared memory with the network on `ctas` CTAs;
        None when it does not fit."""
        a16 = lambda x: (int(x) + 15) // 16 * 16
        off = 0
        # threads per CTA: more warps share the items of a whole SM's neurons
        # (single precision, 9000 neurons: 4.5 us per step with 512, 3.2 with 1024)
        lay = {"ctas": ctas, "cluster": cluster, "block": 512 if cluster else 1024,
               "x": {}, "pop": {}, "proj": {}}
        own = {p.id for p in self.pops}
        for k, pop in self.pres.items():
            # one element more: a zero for the padding of the rows
            copies = 2 if (cluster and k in own) else 1
            lay["x"][k] = (off, a16((pop.size + 1) * self.rb), copies)
            off += copies * a16((pop.size + 1) * self.rb)
        for pop in self.pops:
            chunk = -(-pop.size // ctas)
            d = {"chunk": chunk, "state": {}}
            for name, ct, _ in self.state[pop.id]:
                d["state"][name] = off
                off += a16(chunk * (4 if ct == "int" else self.rb))
            fan = np.zeros(pop.size)
            for p in self._projs(pop):
                fan[p.post_ranks_view] += np.diff(p._csr.indptr)
            typical = float(np.median(fan[fan > 0])) if fan.any() else 0.0
            # lanes per row: one in double precision (ordered sum), in single
            # precision about eight products per lane of a typical row (every
            # lane's first product is rounded by itself: chosen by the mean, 50
            # rows of 2000 among 1950 of 20 had 16 lanes, 3.8 us per step, and an
            # error 1.12 times the launch plan's). Rows per item: full warps
            # (a load instruction for few lanes costs the SM as much as for 32);
            # double precision with one item per SM halves it, for two warps: 4000
            # neurons with 180 synapses each 4.7 us per step with 16 rows, 5.1 with
            # 32 (8000 neurons: 4.8 and 4.4)
            lanes = 1 if self.c.exact else min(16, _pow2(typical / 8))
            rows = 32 // lanes
            if self.c.exact and not cluster and chunk <= 32:
                rows = 16
            d["lanes"], d["rows"] = lanes, rows
            d["items"] = -(-chunk // rows)
            lay["pop"][pop.id] = d
        pool = np.zeros(ctas, dtype=np.int64)
        for proj in self.net.projections:
            d = lay["pop"][proj.post_pop.id]
            chunk, lanes, rows, items = d["chunk"], d["lanes"], d["rows"], d["items"]
            length = np.zeros(ctas * chunk, dtype=np.int64)
            length[proj.post_ranks_view] = np.diff(proj._csr.indptr)
            length = np.pad(length.reshape(ctas, chunk), ((0, 0), (0, items * rows - chunk)))
            steps = -(-length.reshape(ctas, items, rows).max(axis=2) // lanes)
            U = unroll(lanes)
            steps = -(-steps // U) * U
            first = pool[:, None] + np.cumsum(steps, axis=1) * (rows * lanes) - steps * (rows * lanes)
            lay["proj"][proj.id] = np.stack([first, steps], axis=2).astype(np.int32)
            pool = pool + steps.sum(axis=1) * (rows * lanes)
        # (the loads of columns run ahead by two blocks of 8 x 32 elements)
        lay["pool"] = n = int(pool.max())
        lay["w"], off = off, off + a16(n * self.wb)
        lay["col"], off = off, off + a16((n + 512) * 2)
        lay["smem"] = off
        return lay if off <= SMEM_LIMIT else None

    def choose(self):
        """The layout to use, None when the network does not fit. A cluster
        (up to 16 CTAs, about 2000 synapses each: below that its barrier is
        the larger part of a step) while its CTAs' shared-memory gathers take
        less than the grid-wide barrier, else one CTA per SM."""
        want = self.net._config.get("resident_ctas")
        if want:
            return self.layout(int(want), int(want) <= 16)
        if self.nnz <= CLUSTER_SYNAPSES["double" if self.c.exact else "float"]:
            c = min(16, _pow2(self.nnz / 2048))
            while c <= 16:
                lay = self.layout(c, True)
                if lay:
                    return lay
                c *= 2
        from ..runtime.lib import DryNative, device_sm_count
        sms = (GRID_CTAS if isinstance(self.c.native, DryNative)
               else device_sm_count(self.net._config.get("device", 0)))
        return self.layout(min(GRID_CTAS, sms), False)

    # ----------------------------------------------------------------- kernel
    def create_arrays(self, lay):
        """The items' places in the CTAs' pools (rs: first element, steps) and,
        per projection, the pool positions of its synapses: for every element
        of its items its place in the CSR arrays (ri, -1 past a row's end)."""
        nat = self.c.native
        for proj in self.net.projections:
            k, tab = proj.id, lay["proj"][proj.id]
            d = lay["pop"][proj.post_pop.id]
            chunk, lanes, rows, items = d["chunk"], d["lanes"], d["rows"], d["items"]
            # the projection's part of every CTA's pool is one run of elements
            part = tab[:, :, 1].sum(axis=1, dtype=np.int64) * (rows * lanes)
            start = np.concatenate(([0], np.cumsum(part)))
            lengths = np.diff(proj._csr.indptr)
            full = lengths > 0
            post, lengths = proj.post_ranks_view[full], lengths[full].astype(np.int32)
            cta, q = np.divmod(post, chunk)
            item, q = np.divmod(q, rows)
            base = (start[cta] + tab[cta, item, 0] - tab[cta, 0, 0] + q * lanes).astype(np.int32)
            first = (np.cumsum(lengths) - lengths).astype(np.int32)
            j = np.arange(int(lengths.sum()), dtype=np.int32)
            e = j - np.repeat(first, lengths)
            if lanes > 1:
                e, g = e // lanes, e % lanes
                at = np.repeat(base, lengths) + e * np.int32(rows * lanes) + g
            else:
                at = np.repeat(base, lengths) + e * np.int32(rows)
            ri = np.full(int(start[-1]), -1, dtype=np.int32)
            ri[at] = j
            nat.create(f"proj{k}__rs", tab)
            nat.create(f"proj{k}__ri", ri)
            nat.create(f"proj{k}__rb", np.stack([start[:-1], part, tab[:, 0, 0]], axis=1).astype(np.int32))
        if not lay["cluster"]:
            nat.create("gbar", np.zeros(2, dtype=np.uint32))
            for pop in self.pops:
                if pop.id in self.pres:
                    nat.create_empty(f"pop{pop.id}__rx", self.c.real, (2 * self._stride(pop),))
        for m in self.net.monitors:
            if m.ranks is not None:
                pos = np.full(m.population.size, -1, dtype=np.int32)
                pos[np.asarray(m.ranks)] = np.arange(len(m.ranks), dtype=np.int32)
                nat.create(f"mon{m.id}__pos", pos)

    @staticmethod
    def _stride(pop) -> int:
        """Elements per buffer of exchanged rates (16-byte aligned)."""
        return -(-pop.size // 4) * 4

    def module(self, lay) -> Module:
        gen = CodeGenerator(self.c)
        c, net, R = self.c, self.net, gen.real
        W = c.wctype
        C, cluster, BLOCK = lay["ctas"], lay["cluster"], lay["block"]
        carve, load, store, ranges, fill, steps = [], [], [], [], [], []
        own = {p.id for p in self.pops}

        def smem(name, ct, off):
            carve.append(f"{ct}* const anb_s_{name} = reinterpret_cast<{ct}*>(anb_smem + {off});")

        for k, pop in self.pres.items():
            off, size, copies = lay["x"][k]
            smem(f"x{k}", R, off)
            if copies == 2:
                smem(f"x{k}b", R, off + size)
            load.append(f"#pragma unroll 1\n    for (int q = threadIdx.x; q < {pop.size}; q += blockDim.x) anb_s_x{k}[q] = "
                        f"{gen.ptr(f'pop{k}__r')}[q];")
            load.append(f"if (threadIdx.x == 0) anb_s_x{k}[{pop.size}] = ({R})0;")
            if copies == 2:
                load.append(f"if (threadIdx.x == 0) anb_s_x{k}b[{pop.size}] = ({R})0;")
        smem("w", W, lay["w"])
        smem("c", "unsigned short", lay["col"])
        for pop in self.pops:
            k, d = pop.id, lay["pop"][pop.id]
            ranges.append(f"const int anb_base{k} = anb_rank * {d['chunk']};")
            ranges.append(f"const int anb_cnt{k} = max(0, min({pop.size} - anb_base{k}, {d['chunk']}));")
            for name, ct, back in self.state[k]:
                smem(f"p{k}_{name}", ct, d["state"][name])
                g = gen.ptr(f"pop{k}__{name}")
                load.append(f"#pragma unroll 1\n    for (int q = threadIdx.x; q < anb_cnt{k}; q += blockDim.x) "
                            f"anb_s_p{k}_{name}[q] = {g}[anb_base{k} + q];")
                if back:
                    store.append(f"#pragma unroll 1\n    for (int q = threadIdx.x; q < anb_cnt{k}; q += blockDim.x) "
                                 f"{g}[anb_base{k} + q] = anb_s_p{k}_{name}[q];")
        for proj in net.projections:
            k, b = proj.id, proj.post_pop.id
            d = lay["pop"][b]
            p = lambda n, k=k: gen.ptr(f"proj{k}__{n}")
            fill.append(f"""
    anb_rate_fill<{W}>({p('rb')} + 3 * anb_rank, {p('ri')}, {p('col')}, {p('w')}, {proj.pre_pop.size}, anb_s_w, anb_s_c);""")
            # a warp with one item keeps its place in registers
            if d["items"] <= lay["block"] // 32:
                ranges.append(f"const int anb_rf{k} = {p('rs')}[2 * (anb_rank * {d['items']} + min(anb_warp, {d['items'] - 1}))];")
                ranges.append(f"const int anb_rn{k} = {p('rs')}[2 * (anb_rank * {d['items']} + min(anb_warp, {d['items'] - 1})) + 1];")
        for pop in self.pops:
            steps.append(self._pop_step(gen, pop, lay, own))
        recs = []
        for m in net.monitors:
            pre = self._record_test(gen, m)
            if not updated(m.population):
                for v in m.variables:
                    src = gen.ptr(f"pop{m.population.id}__{source_name(v)}")
                    ranks = f"{gen.ptr(f'mon{m.id}__ranks')}[q]" if m.ranks is not None else "q"
                    pre += f"""
      if (anb_rec{m.id}) for (int q = anb_rank * {BLOCK} + (int)threadIdx.x; q < {c.mon_layout[m.id]['n']}; q += {C * BLOCK})
        {gen.ptr(f'mon{m.id}__{array_name(v)}')}[anb_slot{m.id} * {c.mon_layout[m.id]['n']} + q] = (double){src}[{ranks}];"""
            recs.append(pre)
        mon_pre = "\n    ".join(
            f"const int anb_on{m.id} = {gen.ptr(f'mon{m.id}__on')}[0]; "
            f"const long long anb_start{m.id} = {gen.ptr(f'mon{m.id}__start')}[0], "
            f"anb_t0v{m.id} = {gen.ptr(f'mon{m.id}__t0v')}[0];" for m in net.monitors)
        if cluster:
            meet = "anb_cluster_sync();"
            rank, guard = "(int)anb_cluster_rank()", ""
            first = "anb_cluster_sync();"
        else:
            rank, guard = "(int)blockIdx.x", f"if (blockIdx.x >= {C}) return;\n    "
            first = "__syncthreads();"
            copies = "".join(f"""
        {{
          const uint4* src = reinterpret_cast<const uint4*>({gen.ptr(f'pop{p.id}__rx')} + (anb_s & 1) * {self._stride(p)});
          uint4* dst = reinterpret_cast<uint4*>(anb_s_x{p.id});
#pragma unroll 4
          for (int q = threadIdx.x; q < {-(-p.size * self.rb // 16)}; q += blockDim.x) dst[q] = __ldcg(src + q);
        }}""" for p in self.pops if p.id in self.pres)
            meet = f"""if (!anb_grid_meet({gen.ptr('gbar')}, {C}u * (unsigned)(anb_s + 1), {gen.ptr('err')})) break;{copies}
      __syncthreads();"""
        dt_t = "double" if c.exact else "float"
        globals_ = [gen._globals_preamble(p, lambda n, k=p.id: gen.ptr(f"pop{k}__{n}"))
                    for p in self.pops] if self._hoisted(gen) else []
        nl = "\n    "
        name = "anb_rate_run"
        src = f"""
extern "C" __global__ void __launch_bounds__({BLOCK}, 1) {name}(long long anb_t0, int anb_steps) {{
    extern __shared__ __align__(16) unsigned char anb_smem[];
    {guard}const int anb_rank = {rank};
    const {dt_t} dt = ({dt_t})(*{gen.ptr('dt')});
    const int anb_lane = threadIdx.x & 31, anb_warp = threadIdx.x >> 5;
    {nl.join(carve)}
    const unsigned anb_aw = anb_smem_addr(anb_s_w), anb_ac = anb_smem_addr(anb_s_c);
    {nl.join(ranges)}
    {mon_pre}
    {nl.join(globals_)}
    {nl.join(load)}{''.join(fill)}
    {first}
#pragma unroll 1
    for (int anb_s = 0; anb_s < anb_steps; ++anb_s) {{
      const long long t = anb_t0 + anb_s;
      {''.join(recs)}{''.join(steps)}
      {meet}
    }}
    __syncthreads();
    {nl.join(store)}
    if (anb_rank == 0 && threadIdx.x == 0) *{gen.ptr('t')} = anb_t0 + anb_steps;
}}
"""
        smem_bytes = lay["smem"] if cluster else max(lay["smem"], SMEM_ALONE)
        return Module(gen.assemble([src]), gen.options(), "resident",
                      local=(name, C, BLOCK, smem_bytes, C if cluster else -1), kernels=[name])

    def _hoisted(self, gen) -> bool:
        """One population's parameters are read before the step loop (those of
        several may share names)."""
        return len(self.pops) == 1

    def _record_test(self, gen, m) -> str:
        cap = self.c.mon_layout[m.id]["cap_var"]
        return f"""
      const bool anb_due{m.id} = anb_on{m.id} && (t - anb_start{m.id}) % {m.period_steps} == {m.period_offset_steps % m.period_steps};
      const long long anb_slot{m.id} = (t - anb_t0v{m.id}) / {m.period_steps};
      const bool anb_rec{m.id} = anb_due{m.id} && anb_slot{m.id} >= 0 && anb_slot{m.id} < {cap};
      if (anb_due{m.id} && !anb_rec{m.id} && threadIdx.x == 0) anb_report({gen.ptr('err')}, ANB_DEVERR_MONITOR_OVERFLOW);"""

    def _pop_step(self, gen, pop, lay, own) -> str:
        c, R, W = self.c, gen.real, self.c.wctype
        k, d = pop.id, lay["pop"][pop.id]
        lanes, rows, items = d["lanes"], d["rows"], d["items"]
        body, _ = gen._neuron_body(pop, None, False)
        body = gen._use_reciprocals(pop, body)
        draws = gen._random_draws(pop)
        if draws:
            body = draws + "\n" + body
        sums = [f"{R} _sum_{t} = ({R})0;" for t in pop.targets]
        for proj in self._projs(pop):
            a = proj.pre_pop.id
            x = f"anb_s_x{a}"
            if lay["x"][a][2] == 2:
                x = f"((anb_s & 1) ? anb_s_x{a}b : anb_s_x{a})"
            rs = f"{gen.ptr(f'proj{proj.id}__rs')}[2 * (anb_rank * {items} + anb_it)"
            place = (f"anb_rf{proj.id}, anb_rn{proj.id}" if items <= lay["block"] // 32
                     else f"{rs}], {rs} + 1]")
            sums.append(f"_sum_{proj.target} += anb_rate_row<{R}, {W}, {lanes}, {rows}>("
                        f"{place}, anb_aw, anb_ac, anb_smem_addr({x}));  // {proj.name}")
        loads, stores = [], []
        for name, ct, back in self.state[k]:
            s = f"anb_s_p{k}_{name}[anb_q]"
            if name.startswith("_last_sum_"):
                stores.append(f"{s} = _sum_{name[len('_last_sum_'):]};")
                continue
            var = "anb_" + name if name.startswith("kc_") else name
            loads.append(f"{ct} {var} = {s};")
            if back:
                stores.append(f"{s} = {var};")
        recs = []
        for m in self.net.monitors:
            if m.population is not pop:
                continue
            n = c.mon_layout[m.id]["n"]
            at = f"{gen.ptr(f'mon{m.id}__pos')}[anb_i]" if m.ranks is not None else "anb_i"
            puts = " ".join(
                f"{gen.ptr(f'mon{m.id}__{array_name(v)}')}[anb_slot{m.id} * {n} + anb_p] = (double)"
                + (source_name(v).replace("_last_sum_", "_sum_")) + ";" for v in m.variables)
            recs.append(f"if (anb_rec{m.id}) {{ const int anb_p = {at}; if (anb_p >= 0) {{ {puts} }} }}")
        if k in self.pres:
            if lay["cluster"]:
                recs.append(f"""{{
            {R}* anb_dst = ((anb_s & 1) ? anb_s_x{k} : anb_s_x{k}b) + anb_i;
            for (int anb_c = 0; anb_c < {lay['ctas']}; ++anb_c)
              anb_cluster_st(anb_cluster_map(anb_smem_addr(anb_dst), (unsigned)anb_c), r);
          }}""")
            else:
                recs.append(f"__stcg({gen.ptr(f'pop{k}__rx')} + (anb_s & 1) * {self._stride(pop)} + anb_i, r);")
        nl = "\n          "
        one = "" if lanes == 1 else f" && anb_lane % {lanes} == 0"
        return f"""
      {{  // population {pop.name}: weighted sums and update of the own neurons
        {"" if self._hoisted(gen) else gen._globals_preamble(pop, lambda n: gen.ptr(f'pop{k}__{n}'))}
#pragma unroll 1
        for (int anb_it = anb_warp; anb_it < {items}; anb_it += {lay['block'] // 32}) {{
          const int anb_q = anb_it * {rows} + anb_lane / {lanes};
          {nl.join(sums)}
          if (anb_lane < {rows * lanes} && anb_q < anb_cnt{k}{one}) {{
          const int anb_i = anb_base{k} + anb_q; (void)anb_i;
          {nl.join(loads)}
          {body.replace(chr(10), nl)}
          {nl.join(stores)}
          {nl.join(recs)}
          }}
        }}
      }}"""
