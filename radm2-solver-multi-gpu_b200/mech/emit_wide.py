#!/usr/bin/env python3
"""Emit the fragments of the wide tensor-memory solver (csrc/radm2_wide.cuh): straight-line
code for a block of 128 threads, one cell per thread, with every word of a cell's working set
placed at compile time.

  shared memory   state (59), the distinct rate constants, some LU slots
  tensor memory   the 256 most used LU slots (a 512-column row per thread)
  global scratch  the other LU slots, K1, K2 and the saved state: 1 KB per word and block

The mechanism's 156 rate constants are 99 distinct expressions, 11 of them plain numbers
(mgpu.cu:763-918 repeats the peroxy-radical rates); only the 88 others need a word.

Two things bound this kernel and shape the code:

  instruction fetch  Every phase is unrolled, far more than a scheduler's instruction cache,
      so an SM streams its code once per step attempt: 6 to 12 cycles per instruction beyond
      128 KB of code, by how far the warps run together.  Fewer instructions are faster,
      whatever they do.
  memory latency     A warp has no neighbour on its scheduler to hide behind.  Global loads
      are therefore issued a fixed distance (in emitted operations) before their value is
      used, and each group of tensor-memory loads while the previous group is being used.

The arithmetic is that of the plain fragments: the same operations on each value in the same
order.

Fragments talk to their caller through macros: V(i), RC(k), FIX(k), X(i); SL(k) shared word k;
GLD(var, w) / GST(w, value) global word w; TLDn(column, vars...) / TSTn(column, values...) n
doubles of tensor memory, TLD_WAIT and TLD_GET(var) before a loaded value is used, TST_WAIT
before a stored one is loaded; LU_PIVOT_CHECK(value); FMAC(c, a, b) c += a b and
FNMA(c, a, b) c -= a b, fused where the build contracts multiply-adds.
  radm2_wide_map.h             placement tables
  radm2_wide_tmem.h            the TLDn / TSTn macros
  radm2_wide_fun.inc           X(i) = F(V)
  radm2_wide_jac.inc           G = -J + ghinv I into the LU slots
  radm2_wide_lu{_rcp,}.inc     in-place LU (reciprocal pivots / pivot divisions)
  radm2_wide_solve{_rcp,}.inc  X(i) = G^-1 X(i)

Usage:  python emit_wide.py
"""
import json
import os

import emit
from emit import BANNER, CSRC_GEN, Renderer, fused_add, is_zero, kernel_var, lit, slot_chain, term_b

THREADS = 128
SMEM_WORDS = 226        # doubles per thread: 226 KB of the 227 KB a block may have
TMEM_SLOTS = 256
LOAD_AHEAD = 100        # operations a global load is issued before its use
TM_GROUP = 16           # doubles per tensor-memory load group
# Slots that start at zero, and whose first two updates the plain fragments leave to the compiler
# as one sum of two products (it sees the stored zero): it fuses the first product.
FILL_FIRST = (197, 201, 209, 212)
GK1, GK2, GY, GLU = 0, 59, 118, 177  # global words: K1, K2, saved state, LU slots


class Stream:
    """Operations in program order.  text(): the code with global loads moved LOAD_AHEAD
    operations forward (never above the last store to the same word) and each tensor-memory
    load group issued right after the previous group has arrived (never above the last store
    to one of its slots)."""

    def __init__(self, w):
        self.col, self.run_of = w.col, w.run_of
        self.ops = []
        self.names = []
        self.under_way = set()  # slots with a tensor-memory store not waited for yet

    def code(self, text, cost=1):
        self.ops.append(("code", text, cost))

    def gload(self, var, word):
        self.names.append(var)
        self.ops.append(("gload", var, word))

    def gstore(self, word, value):
        self.ops.append(("gstore", word, value))

    def tload(self, pairs):
        """pairs [(slot, var)] in slot order, in groups of TM_GROUP doubles."""
        for i in range(0, len(pairs), TM_GROUP):
            part = pairs[i:i + TM_GROUP]
            self.names += [v for _, v in part]
            self.ops.append(("tload", part))

    def tstore(self, pairs):
        """pairs [(slot, value)] in slot order; waited for before the next load of one of them."""
        if pairs:
            self.ops.append(("tstore", pairs))

    def text(self):
        # 1. global loads: where each is issued
        cost = {"code": lambda o: o[2], "gload": lambda o: 1, "gstore": lambda o: 1,
                "tload": lambda o: 1 + len(o[1]) // 4, "tstore": lambda o: 2 + len(o[1]) // 4}
        at, t = [], 0
        for o in self.ops:
            at.append(t)
            t += cost[o[0]](o)
        stored, place, issue = {}, [], {}
        for i, o in enumerate(self.ops):
            if o[0] == "gstore":
                stored[o[1]] = i
            elif o[0] == "gload":
                j = i
                low = stored.get(o[2], -1)
                while j - 1 > low and at[j - 1] >= at[i] - LOAD_AHEAD:
                    j -= 1
                issue.setdefault(j, []).append(o)
        # 2. tensor-memory groups: issued after the previous group's arrival or the last store to a slot
        groups = [i for i, o in enumerate(self.ops) if o[0] == "tload"]
        tissue, prev = {}, -1
        for g in groups:
            slots = {s for s, _ in self.ops[g][1]}
            low = max([i for i, o in enumerate(self.ops[:g]) if o[0] == "tstore" and slots & {s for s, _ in o[1]}] + [-1])
            tissue.setdefault(("after", max(prev, low)), []).append(g)
            prev = g
        out = []
        for g in tissue.get(("after", -1), []):
            out += self.t_issue(self.ops[g][1])
        for i, o in enumerate(self.ops):
            for ld in issue.get(i, []):
                out.append("GLD(%s, %d);\n" % (ld[1], ld[2]))
            if o[0] == "code":
                out.append(o[1] + "\n")
            elif o[0] == "gstore":
                out.append("GST(%d, %s);\n" % (o[1], o[2]))
            elif o[0] == "tload":
                out += self.t_arrive(o[1])
            elif o[0] == "tstore":
                out += self.t_store(o[1])
            for g in tissue.get(("after", i), []):
                out += self.t_issue(self.ops[g][1])
        decl = []
        for i in range(0, len(self.names), 12):
            decl.append("double %s;\n" % ", ".join(self.names[i:i + 12]))
        if self.under_way:
            out.append("TST_WAIT;\n")
        regs = sorted({v for o in self.ops if o[0] == "tload" for _, v in o[1]})
        for i in range(0, len(regs), 8):
            decl.append("unsigned %s;\n" % ", ".join("%s_l, %s_h" % (v, v) for v in regs[i:i + 8]))
        return decl + out

    def t_issue(self, pairs):
        var, lines, seen = dict(pairs), [], set()
        if any(x in self.under_way for s0, _ in pairs for x in self.run_of[s0]):
            lines.append("TST_WAIT;\n")
            self.under_way.clear()
        for s0, _ in pairs:
            run = self.run_of[s0]
            if run[0] in seen:
                continue
            seen.add(run[0])
            names = [var.get(s, "z%d" % s) for s in run]
            unused = [v for s, v in zip(run, names) if s not in var]
            pre = "{ unsigned %s; " % ", ".join("%s_l, %s_h" % (v, v) for v in unused) if unused else ""
            lines.append("%sTLD%d(%d, %s);%s\n" % (pre, len(run), self.col[run[0]], ", ".join(names), " }" if unused else ""))
        return lines

    def t_arrive(self, pairs):
        return ["TLD_WAIT;\n"] + ["TLD_GET(%s);\n" % v for _, v in pairs]

    def t_store(self, pairs):
        val, lines, seen = dict(pairs), [], set()
        for s0, _ in pairs:
            run = self.run_of[s0]
            if run[0] in seen:
                continue
            seen.add(run[0])
            i = 0
            while i < len(run):  # the stored slots of the run, in the widest aligned pieces
                w = len(run)
                while w > 1 and (i % w or i + w > len(run) or any(s not in val for s in run[i:i + w])):
                    w //= 2
                part = run[i:i + w]
                i += w
                if part[0] in val:
                    lines.append("TST%d(%d, %s);\n" % (w, self.col[part[0]], ", ".join(val[s] for s in part)))
        self.under_way.update(val)
        return lines


class Wide:
    def __init__(self, m):
        self.m = m
        lu = m["lu"]
        self.crow, self.diag, self.icol = lu["crow"], lu["diag"], lu["icol"]
        self.irow = lu["irow"]
        self.n = m["sizes"]["NVAR"]
        self.place_rc()
        self.place_lu()
        self.r = Renderer(self.ref, kernel_var)

    # ---- placement
    def place_rc(self):
        """rc_word[r]: the shared word of rate constant r, or None for a plain number; rc_rep: the
        reaction that stands for each word."""
        words, self.rc_rep, self.rc_word = {}, [], []
        for i, t in enumerate(self.m["rconst"]):
            key = json.dumps(t)
            if t[0] == "num":
                self.rc_word.append(None)
                continue
            if key not in words:
                words[key] = len(self.rc_rep)
                self.rc_rep.append(i)
            self.rc_word.append(words[key])

    def fill(self, sl):
        """A slot that the Jacobian leaves zero and the elimination fills: it is not stored before."""
        k = self.irow[sl]
        return is_zero(self.m["jvs"][sl]) and sl != self.diag[k] and self.icol[sl] in self.touched(k)

    def touched(self, k):
        """Row k's slots that the elimination updates (targets) and those it reads as multipliers."""
        c, d, ic = self.crow, self.diag, self.icol
        cols = set()
        for kk in range(c[k], d[k]):
            j = ic[kk]
            cols.add(j)
            cols.update(ic[jj] for jj in range(d[j] + 1, c[j + 1]))
        return cols

    def accesses(self):
        acc = [1 + 3] * len(self.icol)  # the Jacobian's store, three solves
        for k in range(self.n):
            cols = self.touched(k) | {k}
            for s in range(self.crow[k], self.crow[k + 1]):
                acc[s] += 0 if self.fill(s) else 2 if self.icol[s] in cols else 0
            for kk in range(self.crow[k], self.diag[k]):
                j = self.icol[kk]
                for jj in range(self.diag[j], self.crow[j + 1]):
                    acc[jj] += 1
        return acc

    def place_lu(self):
        """kind[s] / pos[s]: 'T' tensor-memory column, 'S' shared word, 'G' global word."""
        acc = self.accesses()
        order = sorted(range(len(acc)), key=lambda s: (-acc[s], s))
        nsm = SMEM_WORDS - 59 - len(self.rc_rep)
        # pivots of rows without eliminations: in shared memory, inverted there in one loop
        lone = {self.diag[k] for k in range(self.n) if self.crow[k] == self.diag[k]}
        self.lone = sorted(lone)
        order = [s for s in order if s not in lone]
        hot, warm = set(order[:TMEM_SLOTS]), lone | set(order[TMEM_SLOTS:TMEM_SLOTS + nsm - len(lone)])
        n = len(acc)
        self.kind = ["T" if s in hot else "S" if s in warm else "G" for s in range(n)]
        self.pos = [0] * n
        # Tensor memory: each row's multipliers and its U part (with the pivot) are read together, so
        # each is cut into runs of 16, 8, 4, 2 and 1 slots and the runs are laid out widest first:
        # every run starts on a multiple of its width and one instruction moves it.
        runs = []
        for k in range(self.n):
            for lo, hi in ((self.crow[k], self.diag[k]), (self.diag[k], self.crow[k + 1])):
                part = [s for s in range(lo, hi) if self.kind[s] == "T"]
                while part:
                    w = 1 << (min(len(part), TM_GROUP).bit_length() - 1)
                    runs.append(part[:w])
                    part = part[w:]
        self.run_of, self.col, at = {}, [-1] * n, 0
        for run in sorted(runs, key=lambda r: -len(r)):
            for q, s in enumerate(run):
                self.col[s] = self.pos[s] = at + 2 * q
                self.run_of[s] = run
            at += 2 * len(run)
        # shared memory: the pivots of the rows without eliminations first, side by side
        ns = 59 + len(self.rc_rep)
        self.sdiag = ns
        for s in sorted(warm, key=lambda s: (s not in lone, s)):
            self.pos[s] = ns
            ns += 1
        ng = GLU
        for s in range(n):
            if self.kind[s] == "G":
                self.pos[s] = ng
                ng += 1
        ns -= 59 + len(self.rc_rep)
        ng -= GLU
        self.nglobal = GLU + ng
        # the division form's reciprocal pivots, after everything else: first the pivots of rows
        # without eliminations, in the order of their shared words
        rows = [self.irow[sl] for sl in self.lone]
        rows += [k for k in range(self.n) if k not in set(rows)]
        self.gr = {k: self.nglobal + i for i, k in enumerate(rows)}
        self.smem_words = 59 + len(self.rc_rep) + ns
        self.acc = acc

    def ref(self, arr, i):
        if arr == "RCT":
            w = self.rc_word[i]
            return lit(self.m["rconst"][i][1]) if w is None else "RC(%d)" % w
        return {"V": "V(%d)", "F": "FIX(%d)", "A": "a%d", "B": "b%d"}[arr] % i

    # ---- fragments
    def emit_map(self):
        h = [BANNER, "#pragma once\n",
             "/* Working-set placement of the wide tensor-memory solver, in doubles per thread: RC_WORDS\n"
             " * distinct rate constants (word k holds the constant of reaction RC_REP[k]; the %d others are\n"
             " * numbers or repeats); LU slots by their loads and stores per step attempt: %d in tensor memory\n"
             " * (%d of %d accesses), %d in shared memory (%d), %d in global scratch (%d). */\n"
             % (156 - len(self.rc_rep), self.kind.count("T"), sum(a for a, k in zip(self.acc, self.kind) if k == "T"), sum(self.acc),
                self.kind.count("S"), sum(a for a, k in zip(self.acc, self.kind) if k == "S"),
                self.kind.count("G"), sum(a for a, k in zip(self.acc, self.kind) if k == "G")),
             "#define RADM2_WIDE_RC_WORDS %d\n" % len(self.rc_rep),
             "#define RADM2_WIDE_RC_REP_INIT {%s}\n" % ",".join(map(str, self.rc_rep)),
             "#define RADM2_WIDE_SMEM_WORDS %d\n" % self.smem_words,
             "#define RADM2_WIDE_GLOBAL_WORDS %d\n" % self.nglobal,
             "#define RADM2_WIDE_GRCP %d   /* division form: %d more words, the reciprocal pivots */\n"
             "#define RADM2_WIDE_GLOBAL_WORDS_DIV %d\n" % (self.nglobal, self.n, self.nglobal + self.n),
             "#define RADM2_WIDE_SPIVOT %d   /* the %d pivots of rows without eliminations, side by side */\n"
             "#define RADM2_WIDE_SPIVOTS %d\n" % (self.sdiag, len(self.lone), len(self.lone)),
             "#define RADM2_WIDE_GK1 %d\n#define RADM2_WIDE_GK2 %d\n#define RADM2_WIDE_GY %d\n" % (GK1, GK2, GY)]
        emit.write(os.path.join(CSRC_GEN, "radm2_wide_map.h"), [x.replace("emit.py", "emit_wide.py") for x in h])

    def emit_tmem(self):
        """The TLDn / TSTn macros: one tensor-memory instruction for n doubles."""
        h = [BANNER.replace("emit.py", "emit_wide.py"), "#pragma once\n",
             "/* n doubles of the thread's tensor-memory row in one warp-collective instruction.  A load's\n"
             " * registers (v_l, v_h of each variable v) may be read after TLD_WAIT and TLD_GET(v); a store\n"
             " * may be followed by a load of its columns after TST_WAIT.  TM_BASE: the row's first column. */\n"]
        for w in (1, 2, 4, 8, 16):
            vs = ["v%d" % i for i in range(w)]
            h.append('#define TLD%d(c, %s) asm volatile("tcgen05.ld.sync.aligned.32x32b.x%d.b32 {%s}, [%%%d];" : %s : "r"(TM_BASE + (c)))\n'
                     % (w, ", ".join(vs), 2 * w, ", ".join("%%%d" % i for i in range(2 * w)), 2 * w,
                        ", ".join('"=r"(%s##_l), "=r"(%s##_h)' % (v, v) for v in vs)))
            h.append('#define TST%d(c, %s) do { const double %s; asm volatile("tcgen05.st.sync.aligned.32x32b.x%d.b32 [%%0], {%s};" :: '
                     '"r"(TM_BASE + (c)), %s); } while (0)\n'
                     % (w, ", ".join(vs), ", ".join("%s_ = (%s)" % (v, v) for v in vs), 2 * w,
                        ", ".join("%%%d" % (i + 1) for i in range(2 * w)),
                        ", ".join('"r"(__double2loint(%s_)), "r"(__double2hiint(%s_))' % (v, v) for v in vs)))
        h.append('#define TLD_WAIT asm volatile("tcgen05.wait::ld.sync.aligned;")\n'
                 '#define TST_WAIT asm volatile("tcgen05.wait::st.sync.aligned;")\n'
                 '#define TLD_GET(v) do { asm volatile("" : "+r"(v##_l), "+r"(v##_h)); v = __hiloint2double((int)v##_h, (int)v##_l); } while (0)\n')
        emit.write(os.path.join(CSRC_GEN, "radm2_wide_tmem.h"), h)

    def emit_fun(self):
        s = Stream(self)
        m, r = self.m, self.r
        uses = {}
        for i, t in enumerate(m["vdot"]):
            for pos, (op, term) in enumerate(slot_chain(t)):
                refs = []

                def walk(x):
                    if x[0] == "ref" and x[1] == "A":
                        refs.append(x[2])
                    for y in x[1:]:
                        if isinstance(y, list):
                            walk(y)
                walk(term)
                uses.setdefault(refs[0], []).append((i, pos, op, term))
        for rx, t in enumerate(m["rates"]):
            if rx not in uses:
                continue
            lines = ["{ const double a%d = %s;" % (rx, r(t))]
            for (i, pos, op, term) in uses[rx]:
                lines.append("  X(%d) = %s;" % (i, r(term)) if pos == 0 else "  " + fused_add(r, "X(%d)" % i, op, term, t))
            s.code("\n".join(lines) + " }", 5 + len(uses[rx]))
        self.put("fun", s, "ODE right-hand side X(i) = F(V), mgpu.cu:1103-1385, reaction-major: each rate is formed\n"
                 " * once and added into the species it touches, in the reference's order of every sum")

    def emit_jac(self):
        s = Stream(self)
        m, r, dset = self.m, self.r, set(self.diag)
        juses, names = {}, []
        for sl, t in enumerate(m["jvs"]):
            if is_zero(t):
                if not self.fill(sl):
                    self.store(s, sl, "(-0.0) + ghinv" if sl in dset else "-0.0")
                continue
            chain = slot_chain(t)
            for pos, (op, term) in enumerate(chain):
                juses.setdefault(term_b(term), []).append((sl, pos, op, term, pos == len(chain) - 1))
        for k in sorted(m["bvals"], key=int):
            b = int(k)
            if b not in juses:
                continue
            s.code("const double b%d = %s;" % (b, r(m["bvals"][k])), 3)
            for (sl, pos, op, term, last) in juses[b]:
                if pos > 0:
                    s.code(fused_add(r, "js%d" % sl, op, term, m["bvals"][k]))
                    expr = "js%d" % sl
                else:
                    expr = r(term)
                    if not last:
                        names.append("js%d" % sl)
                        s.code("js%d = %s;" % (sl, expr))
                if last:
                    self.store(s, sl, "(-%s)%s" % (expr, " + ghinv" if sl in dset else ""))
        s.names += names
        self.put("jac", s, "G = -J + ghinv I into the LU slots, mgpu.cu:1685-2652, partial-major: each partial is formed\n"
                 " * once and added into the slots that use it, in the reference's order of every sum",
                 tail="TST_WAIT;\n")

    def store(self, s, sl, value):
        """One slot, from the Jacobian: no wait (nothing is read before the fragment's end)."""
        k, p = self.kind[sl], self.pos[sl]
        if k == "G":
            s.gstore(p, value)
        elif k == "S":
            s.code("SL(%d) = %s;" % (p, value))
        else:
            s.code("TST1(%d, %s);" % (p, value), 2)

    def read_group(self, s, slots, prefix):
        """Load slots; returns {slot: expression}."""
        ex = {}
        for sl in slots:
            if self.kind[sl] == "G":
                ex[sl] = "%s_%d" % (prefix, sl)
                s.gload(ex[sl], self.pos[sl])
            elif self.kind[sl] == "S":
                ex[sl] = "SL(%d)" % self.pos[sl]
            else:
                ex[sl] = "%s_%d" % (prefix, sl)
        s.tload([(sl, ex[sl]) for sl in slots if self.kind[sl] == "T"])
        return ex

    def emit_lu(self, recip):
        s = Stream(self)
        c, d, ic = self.crow, self.diag, self.icol
        for k in range(self.n):
            dk = d[k]
            cols = self.touched(k)
            row = [sl for sl in range(c[k], c[k + 1]) if ic[sl] in cols or ic[sl] == k]
            w = {ic[sl]: "w%d_%d" % (k, ic[sl]) for sl in row}
            if not cols:  # no elimination: pivot checked (and inverted) by the kernel's loop over SL(SPIVOT ...)
                continue
            s.tload([(sl, w[ic[sl]]) for sl in row if self.kind[sl] == "T" and not self.fill(sl)])
            seen, held = set(), {}

            def need(j):
                """Row element j in a register before its first use."""
                if j in seen:
                    return
                seen.add(j)
                sl = next(x for x in row if ic[x] == j)
                if self.fill(sl):
                    s.names.append(w[j])
                    s.code("%s = -0.0;" % w[j], 0)
                elif self.kind[sl] == "G":
                    s.gload(w[j], self.pos[sl])
                elif self.kind[sl] == "S":
                    s.names.append(w[j])
                    s.code("%s = SL(%d);" % (w[j], self.pos[sl]))
                if j == k:
                    s.code("LU_PIVOT_CHECK(%s);" % w[j])
            if self.kind[dk] == "T":
                need(k)
            for kk in range(c[k], dk):
                j = ic[kk]
                ex = self.read_group(s, list(range(d[j], c[j + 1])), "u%d" % k)
                need(j)
                self.divide(s, w[j], ex[d[j]], j, "q%d_%d" % (k, j), recip)
                self.put_slots(s, [(kk, w[j])], only="GS")
                for jj in range(d[j] + 1, c[j + 1]):
                    t = ic[jj]
                    sl = next(x for x in row if ic[x] == t)
                    if sl in FILL_FIRST and t not in seen:
                        seen.add(t)
                        s.names.append(w[t])
                        held[t] = (w[j], ex[jj])
                        continue
                    need(t)
                    if t in held:
                        s.code("%s = -(%s * %s);" % (w[t], w[j], ex[jj]))
                        s.code("FNMA(%s, %s, %s);" % ((w[t],) + held.pop(t)))
                        continue
                    s.code("FNMA(%s, %s, %s);" % (w[t], w[j], ex[jj]))
            need(k)
            outs = []
            for sl in row:
                j = ic[sl]
                if j < k and self.kind[sl] != "T":
                    continue  # stored at its pivot
                outs.append((sl, "1.0 / %s" % w[j] if (recip and j == k) else w[j]))
            if not recip and k not in cols:
                outs = [(sl, v) for sl, v in outs if sl != dk]
            self.put_slots(s, outs)
            if not recip:
                s.code("", 9)
                s.gstore(self.gr[k], "RCPR(%s)" % w[k])
        self.put("lu" + ("_rcp" if recip else ""), s,
                 "In-place pivot-free LU on the fixed fill pattern, mgpu.cu:2746-2779 order, %s.\n"
                 " * A row's slots that no elimination touches stay where they are" %
                 ("the diagonal slots holding 1/U(k,k) on exit" if recip else "pivot divisions"))

    def divide(self, s, var, pivot, j, name, recip):
        """var /= pivot of row j: by the reciprocal that the diagonal slot holds, or exactly, by pivot
        and its reciprocal."""
        if recip:
            s.code("%s = %s * %s;" % (var, var, pivot))
        else:
            s.gload(name, self.gr[j])
            s.code("%s = DIVR(%s, %s, %s);" % (var, var, pivot, name), 9)

    def put_slots(self, s, pairs, only="GST"):
        ts = []
        for sl, v in pairs:
            k = self.kind[sl]
            if k not in only:
                continue
            cost = 12 if "/" in v else 1
            if k == "G":
                s.gstore(self.pos[sl], v)
            elif k == "S":
                s.code("SL(%d) = %s;" % (self.pos[sl], v), cost)
            else:
                if "/" in v:
                    s.names.append("r_%d" % sl)
                    s.code("r_%d = %s;" % (sl, v), cost)
                    v = "r_%d" % sl
                ts.append((sl, v))
        s.tstore(ts)

    def emit_solve(self, recip):
        s = Stream(self)
        c, d, ic = self.crow, self.diag, self.icol
        for k in range(self.n):
            if c[k] == d[k]:
                continue
            ex = self.read_group(s, list(range(c[k], d[k])), "g")
            for sl in range(c[k], d[k]):
                s.code("FNMA(X(%d), %s, X(%d));" % (k, ex[sl], ic[sl]), 2 if self.kind[sl] == "S" else 1)
        for k in reversed(range(self.n)):
            ex = self.read_group(s, list(range(d[k], c[k + 1])), "g")
            for sl in range(d[k] + 1, c[k + 1]):
                s.code("FNMA(X(%d), %s, X(%d));" % (k, ex[sl], ic[sl]), 2 if self.kind[sl] == "S" else 1)
            self.divide(s, "X(%d)" % k, ex[d[k]], k, "q%d" % k, recip)
        self.put("solve" + ("_rcp" if recip else ""), s,
                 "X = (LU)^-1 X in place, mgpu.cu:2873-3090 order%s" % (", diagonal slots hold reciprocals" if recip else ""))

    def put(self, name, s, what, tail=""):
        body = [BANNER.replace("emit.py", "emit_wide.py"), "/* %s. */\n" % what] + s.text() + [tail]
        emit.write(os.path.join(CSRC_GEN, "radm2_wide_%s.inc" % name), body)


def main():
    w = Wide(emit.load())
    w.emit_map()
    w.emit_tmem()
    w.emit_fun()
    w.emit_jac()
    for recip in (False, True):
        w.emit_lu(recip)
        w.emit_solve(recip)
    print("wide: %d rate-constant words, %d shared, %d global words per thread; LU accesses T/S/G %s"
          % (len(w.rc_rep), w.smem_words, w.nglobal,
             [sum(a for a, k in zip(w.acc, w.kind) if k == q) for q in "TSG"]))


if __name__ == "__main__":
    main()
