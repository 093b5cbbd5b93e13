"""Derivatives of run-time compiled kernels: ``@parallel ∇=(A->Ā, B->B̄) f!(A, B, a)``.

The reference differentiates a kernel with Enzyme: `@parallel ∇=(A->Ā, B->B̄) f!(A, B, a)` expands
to `@parallel configcall=f!(A, B, a) AD.autodiff_deferred!(Enzyme.Reverse, f!,
DuplicatedNoNeed(A, Ā), DuplicatedNoNeed(B, B̄), Const(a))` (src/ParallelKernel/parallel.jl:265-301)
and every thread runs `Enzyme.autodiff_deferred(mode, f!, Const, args...)` on its own point
(src/ParallelKernel/EnzymeExt/autodiff_gpu.jl:35-40). Here the derivative kernel is generated from
the definition's source, like the kernel itself (ps_gb300.jit), and compiled for sm_103a:

- reverse mode (``ad_mode="reverse"``, Enzyme.Reverse): each thread runs its statements -- the
  primal stores happen, as in Enzyme's combined reverse mode -- keeping every intermediate value in
  registers, then walks them backwards: the shadow of a written element is read and zeroed (the
  element's old value no longer reaches the result) and the adjoint of every value read from a
  duplicated array is added to that array's shadow. A shadow element that other threads may also
  update takes an atomic addition (as Enzyme's gradient accumulation on the GPU does); a shadow
  that only its own thread touches is updated in place. Over the kernel's state map M -> F(M) of
  the duplicated arrays: shadow <- J_F(M)^T shadow.
- forward mode (``ad_mode="forward"``, Enzyme.Forward): the tangent of every value is carried
  beside it, and the shadow of a written element receives the tangent of its new value:
  shadow <- J_F(M) shadow (elements not written keep theirs).

Scalars are constants (Enzyme.Const), and so are the arrays not named in ∇. Supported bodies:
`@parallel` kernels (FiniteDifferences macros, on-the-fly arrays, masks of the left-hand
selections) and `@parallel_indices` kernels with explicit indexing, local variables and
if / elseif / else blocks (an early `return` included); arithmetic + - * /, literal and general
powers, max / min / abs / ifelse / inv and the kernel language's math functions. Loops and
kernel-language calls (shared memory, barriers, shuffles) are refused, and so is a duplicated
array that is written and also accessed at another index (its threads would race).
"""
from __future__ import annotations

import ast
import ctypes
import numbers
import re

from . import _lib
from ._lib import PSArray
from .core import ArgumentError, capturing, describe, require_initialized, stream_handle
from .fd import AV, DIFF, DIFF2, HARM, MAXLOC, MINLOC, SEL
from .jit import (_I32x3, _I64x3, _REALS, MAX_ARRAYS, MAX_SCALARS, VALUE_HELPERS, _MATH, JitKernel, _Gen, _lit, array_ndims, blocks_per_sm,
                  sweep_chunk, uses_kernel_language)
from .kernels import ranges_to_box

MODES = ("reverse", "forward")
SWEEP_MIN = 1 << 19  # points from which FP32 reverse kernels sweep
_ONE = "((R)1.0)"
_LITERAL = re.compile(r"^\(\(R\)[-+0-9.eE]+\)$")  # a number literal of the kernel's type
_SCALAR = re.compile(r"^s[0-9]+$")                  # a scalar argument


class _X:
    """A real value of the derivative kernel: an SSA register with an adjoint / tangent (`var`), or a
    value without derivative (a literal, a scalar argument, or a register holding a constant)."""

    __slots__ = ("code", "var")

    def __init__(self, code, var=False):
        self.code, self.var = code, var


# Shadow-memory helpers of the generated kernels (bounds-checked like the primal accesses: an index
# outside the array was already reported by the primal load, and its shadow is left alone).
_HELPERS = r"""
__device__ __forceinline__ bool ad_in(long long n0, long long n1, long long n2, long long i, long long j, long long k) {
    return (unsigned long long)i < (unsigned long long)n0 && (unsigned long long)j < (unsigned long long)n1 && (unsigned long long)k < (unsigned long long)n2; }
__device__ __forceinline__ E ad_ld(const E* d, long long n0, long long n1, long long n2, long long i, long long j, long long k) {
    return ad_in(n0, n1, n2, i, j, k) ? d[i + n0 * (j + n1 * k)] : (E)0; }
__device__ __forceinline__ void ad_st(E* d, long long n0, long long n1, long long n2, long long i, long long j, long long k, E v) {
    if (ad_in(n0, n1, n2, i, j, k)) d[i + n0 * (j + n1 * k)] = v; }
__device__ __forceinline__ E ad_take(E* d, long long n0, long long n1, long long n2, long long i, long long j, long long k) {
    if (!ad_in(n0, n1, n2, i, j, k)) return (E)0;
    const long long l = i + n0 * (j + n1 * k); const E g = d[l]; d[l] = (E)0; return g; }
__device__ __forceinline__ void ad_add(E* d, long long n0, long long n1, long long n2, long long i, long long j, long long k, E v, bool shared) {
    if (!ad_in(n0, n1, n2, i, j, k)) return;
    const long long l = i + n0 * (j + n1 * k);
    if (shared) atomicAdd(&d[l], v); else d[l] += v; }
"""


class _AdGen(_Gen):
    """Source of the derivative kernel of one definition (one point per thread)."""

    def __init__(self, kd, ndims, dup, mode):
        if mode not in MODES:
            raise ArgumentError(f"ad_mode must be one of {MODES}")
        if uses_kernel_language(kd):
            raise ArgumentError(f"{kd.name}: kernels that use the kernel language (@sharedMem, barriers, shuffles, "
                                "votes, thread indices) cannot be differentiated here")
        super().__init__(kd, ndims)
        unknown = [n for n in dup if n not in kd.arrays]
        if unknown:
            raise ArgumentError(f"∇: {unknown} are not array arguments of {kd.name}")
        self.dup = [n for n in kd.arrays if n in dup]
        self.didx = {n: len(kd.arrays) + i for i, n in enumerate(self.dup)}
        self.mode = mode
        self.nv = 0
        self.vars = []       # (register, C type) declared at the top of the kernel
        self.dvars = []      # registers with an adjoint (b...) or tangent (t...)
        self.tape = []       # (executed flag, nodes, store) per statement, in execution order
        self.nodes = None
        self.fresh = set()   # registers of the current statement whose adjoint nothing has been added to
        self.cur = {}        # real local variable -> its current value
        self.cache = None    # loads of one `@parallel` statement: (array, offsets) -> value
        self.keys = {}       # array -> access keys (offsets / index expressions) of all its accesses
        self.written = set()
        self.fw = []
        self.ind = "    "

    # ---- registers and nodes
    def _new(self, ctype):
        name = {"R": "v", "long long": "i", "bool": "f"}[ctype] + str(self.nv)
        self.nv += 1
        self.vars.append((name, ctype))
        return name

    def emit(self, line):
        self.fw.append(self.ind + line)

    def const(self, code):
        """A value without derivative; anything but a literal or a scalar is kept in a register
        (the reverse sweep must see the value of the forward sweep)."""
        if _LITERAL.match(code) or _SCALAR.match(code):
            return _X(code)
        c = self._new("R")
        self.emit(f"{c} = {code};")
        return _X(c)

    def node(self, op, code, ins, aux=None):
        if op != "load" and not any(x.var for x in ins):
            return self.const(code)
        v = self._new("R")
        self.dvars.append(v)
        self.emit(f"{v} = {code};")
        out = _X(v, True)
        self.nodes.append((op, out, ins, aux))
        if self.mode == "forward":
            self.emit(f"t{v} = {self.tangent(op, out, ins, aux)};")
        return out

    def bin(self, op, sym, a, b):
        return self.node(op, f"({a.code} {sym} {b.code})", [a, b])

    def flag(self, code):
        f = self._new("bool")
        self.emit(f"{f} = {code};")
        return f

    # ---- loads
    def key(self, name, key):
        self.keys.setdefault(name, set()).add(key)

    def leaf(self, name, idx, key=None):
        if name in self.shared or name not in self.aidx:
            raise ArgumentError(f"∇: {name} is not an array argument")
        self.key(name, key or ("i", tuple(idx)))
        ivs = []
        for x in idx:
            iv = self._new("long long")
            self.emit(f"{iv} = {x};")
            ivs.append(iv)
        code = self.load(name, ivs)
        if name in self.dup:
            return self.node("load", code, [], aux=(name, ivs))
        return self.const(code)

    def lval(self, name, o):
        if name in self.temps:  # on-the-fly array: its expression at the shifted index
            li, e = self.temps[name]
            return self.lo(e, tuple(o[d] - ((li >> d) & 1) for d in range(3)))
        if name not in self.aidx:
            raise ArgumentError(f"unknown array {name}")
        o3 = tuple(o[d] if d < self.nd else 0 for d in range(3))
        if self.cache is not None and (name, o3) in self.cache:
            return self.cache[(name, o3)]
        t = ("tx", "ty", "tz")
        idx = [f"{t[d]}+{o3[d]}" if o3[d] else t[d] for d in range(self.nd)]
        x = self.leaf(name, idx, ("o", o3[:self.nd]))
        if self.cache is not None:
            self.cache[(name, o3)] = x
        return x

    def lmacro(self, mname, name, off):
        """A FiniteDifferences macro as value nodes, in the operation order of the forward kernel."""
        if mname not in self.macros:
            raise ArgumentError(f"unknown macro @{mname} for {self.nd}-D")
        kind, opd, inn = self.macros[mname]
        b = [off[d] + ((inn >> d) & 1) for d in range(3)]

        def shift(d, s):
            o = list(b)
            o[d] += s
            return self.lval(name, o)

        dims = [d for d in range(3) if (opd >> d) & 1]
        if kind == SEL:
            return self.lval(name, b)
        if kind == DIFF:
            return self.bin("sub", "-", shift(dims[0], 1), self.lval(name, b))
        if kind == DIFF2:
            c = self.lval(name, b)
            return self.bin("sub", "-", self.bin("sub", "-", shift(dims[0], 1), c),
                            self.bin("sub", "-", c, shift(dims[0], -1)))
        if kind in (AV, HARM):
            terms = []
            for c in range(1 << len(dims)):
                o = list(b)
                for j, d in enumerate(dims):
                    o[d] += (c >> j) & 1
                v = self.lval(name, o)
                terms.append(self.bin("div", "/", _X(_ONE), v) if kind == HARM else v)
            s = terms[0]
            for t in terms[1:]:
                s = self.bin("add", "+", s, t)
            k = float(1 << len(dims))
            if kind == AV:
                return self.bin("mul", "*", s, _X(_lit(1.0 / k)))
            return self.bin("mul", "*", self.bin("div", "/", _X(_ONE), s), _X(_lit(k)))
        if kind in (MAXLOC, MINLOC):
            op, f = ("max", "jl_max") if kind == MAXLOC else ("min", "jl_min")

            def m(x, y):
                return self.node(op, f"{f}({x.code}, {y.code})", [x, y])
            r = m(m(shift(0, -1), shift(0, 1)), self.lval(name, b))
            for d in range(1, self.nd):
                r = m(r, m(shift(d, -1), shift(d, 1)))
            return r
        raise ArgumentError(f"macro @{mname} not supported")

    # ---- real expressions as value nodes
    def lo(self, e, off=(0, 0, 0)):
        t = self.etype(e)
        if t == "int":
            return self.const(self.expr(e, off, "real"))
        if t == "bool":
            return self.const(f"((R)({self.expr(e, off, 'auto')}))")
        if isinstance(e, ast.Constant):
            return _X(_lit(e.value))
        if isinstance(e, ast.Name):
            if e.id in self.sidx:
                return _X(f"s{self.sidx[e.id]}")
            if e.id in self.cur:
                return self.cur[e.id]
            if e.id in self.locals:
                raise ArgumentError(f"∇: local {e.id} is read before it is assigned")
            raise ArgumentError(f"unknown name {e.id} in an expression")
        if isinstance(e, ast.UnaryOp):
            if isinstance(e.op, ast.USub):
                a = self.lo(e.operand, off)
                return self.node("neg", f"(-{a.code})", [a])
            if isinstance(e.op, ast.UAdd):
                return self.lo(e.operand, off)
        if isinstance(e, ast.BinOp):
            if isinstance(e.op, ast.Pow):
                if isinstance(e.right, ast.Constant) and e.right.value in (2, 3) and not isinstance(e.right.value, bool):
                    x = self.lo(e.left, off)
                    sq = self.bin("mul", "*", x, x)
                    return sq if e.right.value == 2 else self.bin("mul", "*", sq, x)
                a, b = self.lo(e.left, off), self.lo(e.right, off)
                return self.node("pow", f"pow({a.code}, (R)({b.code}))", [a, b])
            if isinstance(e.op, ast.Mult) and (self.is_bool(e.left) or self.is_bool(e.right)):
                bl, x = (e.left, e.right) if self.is_bool(e.left) else (e.right, e.left)
                f = self.flag(self.expr(bl, off, "auto"))
                xv = self.lo(x, off)
                return self.node("bmul", f"jl_bmul({f}, {xv.code})", [xv], f)
            if isinstance(e.op, ast.Mod):
                a, b = self.lo(e.left, off), self.lo(e.right, off)
                return self.node("fmod", f"fmod({a.code}, {b.code})", [a, b])
            if isinstance(e.op, ast.FloorDiv):  # a step function: no derivative
                a, b = self.lo(e.left, off), self.lo(e.right, off)
                return self.const(f"trunc({a.code} / {b.code})")
            ops = {ast.Add: ("add", "+"), ast.Sub: ("sub", "-"), ast.Mult: ("mul", "*"), ast.Div: ("div", "/")}
            if type(e.op) not in ops:
                raise ArgumentError("unsupported operator")
            op, sym = ops[type(e.op)]
            return self.bin(op, sym, self.lo(e.left, off), self.lo(e.right, off))
        if isinstance(e, ast.Call) and isinstance(e.func, ast.Name):
            f = e.func.id
            if f.startswith("__m_"):
                if len(e.args) != 1 or not isinstance(e.args[0], ast.Name):
                    raise ArgumentError(f"@{f[4:]} takes one array")
                return self.lmacro(f[4:], e.args[0].id, off)
            if f in ("max", "min"):
                r = self.lo(e.args[0], off)
                for x in e.args[1:]:
                    xv = self.lo(x, off)
                    r = self.node(f, f"jl_{f}({r.code}, {xv.code})", [r, xv])
                return r
            if f == "abs":
                a = self.lo(e.args[0], off)
                return self.node("abs", f"fabs({a.code})", [a])
            if f == "inv":
                a = self.lo(e.args[0], off)
                return self.bin("div", "/", _X(_ONE), a)
            if f in ("one", "zero"):
                return _X("((R)1)" if f == "one" else "((R)0)")
            if f == "ifelse":
                c = self.flag(self.expr(e.args[0], off, "auto"))
                a, b = self.lo(e.args[1], off), self.lo(e.args[2], off)
                return self.node("select", f"({c} ? {a.code} : {b.code})", [a, b], c)
            if f in _MATH:
                a = self.lo(e.args[0], off)
                return self.node(f, f"{f}({a.code})", [a])
            raise ArgumentError(f"∇: unsupported function {f}")
        if isinstance(e, ast.Subscript):
            name, ix = self.subscript(e, off)
            return self.leaf(name, ix)
        raise ArgumentError(f"∇: unsupported expression {ast.dump(e)[:80]}")

    # ---- statements (forward sweep; the reverse sweep is built from the tape)
    def stmt(self, s, ind):
        saved = self.fw, self.ind
        self.fw, self.ind = [], "    " * ind
        try:
            self._stmt(s, ind)
            return self.fw
        finally:
            self.fw, self.ind = saved

    def begin(self):
        f = self.flag("true")
        self.nodes = []
        return f

    def end(self, f, store=None):
        self.tape.append((f, self.nodes, store))
        self.nodes = None

    def store(self, name, idx, rhs):
        """Primal store of rhs at idx (0-based index registers or expressions) and, in forward mode,
        of its tangent into the shadow."""
        k = self.aidx[name]
        i3 = list(idx) + ["0"] * (3 - len(idx))
        if self.checked:
            self.emit(f"jl_st(a{k}, n{k}_0, n{k}_1, n{k}_2, {i3[0]}, {i3[1]}, {i3[2]}, g.err, (E)({rhs.code}));")
        else:
            self.emit(f"{self.at(name, idx)} = (E)({rhs.code});")
        if self.mode == "forward" and name in self.dup:
            t = f"t{rhs.code}" if rhs.var else "(R)0"
            self.emit(f"ad_st(d{k}, n{k}_0, n{k}_1, n{k}_2, {i3[0]}, {i3[1]}, {i3[2]}, (E)({t}));")
        self.written.add(name)
        return (name, i3, rhs)

    def runs(self, lhs, point=("tx", "ty", "tz")):
        """The points at which a statement with this left-hand side (array, mask) runs."""
        name, li = lhs
        k = self.aidx[name]
        return " && ".join(f"{point[d]} < n{k}_{d} - {2 * ((li >> d) & 1)}" for d in range(self.nd))

    def _stmt(self, s, ind):
        if isinstance(s, ast.If):
            c = self.flag(f"({self.expr(s.test, ctx='auto')})")
            before = dict(self.cur)
            self.emit(f"if ({c}) {{")
            for b in s.body:
                self.fw += self.stmt(b, ind + 1)
            then = self.cur
            self.cur = dict(before)
            if s.orelse:
                self.emit("} else {")
                for b in s.orelse:
                    self.fw += self.stmt(b, ind + 1)
            self.emit("}")
            other = self.cur
            self.cur = dict(before)
            for name in sorted(set(then) | set(other)):
                a, b = then.get(name, _X("((R)0)")), other.get(name, _X("((R)0)"))
                if a is b:
                    self.cur[name] = a
                    continue
                f = self.begin()
                v = self.node("select", f"({c} ? {a.code} : {b.code})", [a, b], c)
                self.emit(f"v_{name} = {v.code};")
                self.end(f)
                self.cur[name] = v
            return
        if isinstance(s, (ast.For, ast.While)):
            raise ArgumentError("∇: kernels with loops cannot be differentiated here")
        if isinstance(s, ast.Pass):
            return
        if isinstance(s, ast.Return):
            if s.value is not None:
                raise ArgumentError("kernels return nothing")
            self.emit("goto ps_fwd_done_;")
            return
        if not isinstance(s, ast.Assign) or len(s.targets) != 1:
            raise ArgumentError("∇: kernel statements are assignments and if-blocks")
        t = s.targets[0]
        if isinstance(t, ast.Name):  # local variable
            if self.locals.get(t.id) == "int":
                self.emit(f"v_{t.id} = (long long)({self.expr(s.value, ctx='int')});")
                return
            f = self.begin()
            v = self.lo(s.value)
            self.emit(f"v_{t.id} = {v.code};")
            self.end(f)
            self.cur[t.id] = v
            return
        if isinstance(t, ast.Subscript) and isinstance(t.value, ast.Name) and t.value.id.startswith("__lhs_"):
            sel, name = t.value.id[6:], t.slice.id
            if sel not in self.sels:
                raise ArgumentError(f"@{sel} cannot be a left-hand side")
            if name in self.temps:
                return
            li = self.sels[sel]
            t3 = ("tx", "ty", "tz")
            self.emit(f"if ({self.runs((name, li))}) {{")
            saved = self.ind
            self.ind += "    "
            f = self.begin()
            self.cache = {}
            rhs = self.lo(s.value)
            self.cache = None
            o = tuple((li >> d) & 1 for d in range(self.nd))
            self.key(name, ("o", o))
            idx = [f"{t3[d]}+{o[d]}" if o[d] else t3[d] for d in range(self.nd)]
            st = self.store(name, idx, rhs)
            self.end(f, st)
            self.ind = saved
            self.emit("}")
            return
        if isinstance(t, ast.Subscript):  # @parallel_indices: A[i, j] = expr
            name, ix = self.subscript(t)
            if name in self.shared:
                raise ArgumentError("∇: @sharedMem arrays cannot be differentiated")
            f = self.begin()
            rhs = self.lo(s.value)
            self.key(name, ("i", tuple(ix)))
            ivs = []
            for x in ix:
                iv = self._new("long long")
                self.emit(f"{iv} = {x};")
                ivs.append(iv)
            st = self.store(name, ivs, rhs)
            self.end(f, st)
            return
        raise ArgumentError("unsupported left-hand side")

    # ---- derivative rules
    def tangent(self, op, out, ins, aux):
        a = ins[0] if ins else None
        b = ins[1] if len(ins) > 1 else None
        A, B, O = (a.code if a else ""), (b.code if b else ""), out.code

        def T(x):
            return f"t{x.code}" if x.var else "(R)0"
        if op == "load":
            name, ivs = aux
            k = self.aidx[name]
            i3 = list(ivs) + ["0"] * (3 - len(ivs))
            return f"(R)ad_ld(d{k}, n{k}_0, n{k}_1, n{k}_2, {i3[0]}, {i3[1]}, {i3[2]})"
        if op == "add":
            return f"({T(a)} + {T(b)})"
        if op == "sub":
            return f"({T(a)} - {T(b)})"
        if op == "neg":
            return f"(-{T(a)})"
        if op == "mul":
            return f"({T(a)} * {B} + {A} * {T(b)})"
        if op == "div":
            return f"(({T(a)} - {O} * {T(b)}) / {B})"
        if op == "select":
            return f"({aux} ? {T(a)} : {T(b)})"
        if op == "bmul":
            return f"({aux} ? {T(a)} : (R)0)"
        if op in ("max", "min"):
            sel = f"!signbit({A} - {B})" if op == "max" else f"signbit({A} - {B})"
            return f"(({sel}) ? {T(a)} : {T(b)})"
        if op == "abs":
            return f"(signbit({A}) ? -{T(a)} : {T(a)})"
        if op == "pow":
            s = f"{T(a)} * {B} * pow({A}, {B} - (R)1)"
            return f"({s} + {T(b)} * {O} * log({A}))" if b.var else f"({s})"
        if op == "fmod":
            return f"({T(a)} - {T(b)} * trunc({A} / {B}))"
        return f"({T(a)} * {self.dfun(op, A, O)})"

    def dfun(self, op, A, O):
        """d op(A) / dA, with O = op(A)."""
        return {"exp": O, "exp2": f"{O} * (R)0.6931471805599453", "log": f"((R)1 / {A})",
                "log10": f"((R)1 / ({A} * (R)2.302585092994046))", "sqrt": f"((R)1 / ({O} + {O}))",
                "cbrt": f"((R)1 / ((R)3 * {O} * {O}))", "sin": f"cos({A})", "cos": f"(-sin({A}))",
                "tan": f"((R)1 + {O} * {O})", "tanh": f"((R)1 - {O} * {O})", "sinh": f"cosh({A})",
                "cosh": f"sinh({A})", "atan": f"((R)1 / ((R)1 + {A} * {A}))",
                "asin": f"((R)1 / sqrt((R)1 - {A} * {A}))", "acos": f"(-(R)1 / sqrt((R)1 - {A} * {A}))"}[op]

    def adjoint(self, op, out, ins, aux):
        a = ins[0] if ins else None
        b = ins[1] if len(ins) > 1 else None
        A, B, O, bo = (a.code if a else ""), (b.code if b else ""), out.code, f"b{out.code}"
        lines = []

        def acc(x, expr):
            if x is not None and x.var:
                lines.append(self.add(x.code, expr))
        if op == "load":
            name, ivs = aux
            k = self.aidx[name]
            i3 = list(ivs) + ["0"] * (3 - len(ivs))
            lines.append(f"ad_add(d{k}, n{k}_0, n{k}_1, n{k}_2, {i3[0]}, {i3[1]}, {i3[2]}, (E){bo}, "
                         f"{'true' if self.is_shared(name) else 'false'});")
        elif op == "add":
            acc(a, bo)
            acc(b, bo)
        elif op == "sub":
            acc(a, bo)
            acc(b, f"-{bo}")
        elif op == "neg":
            acc(a, f"-{bo}")
        elif op == "mul":
            acc(a, f"{bo} * {B}")
            acc(b, f"{bo} * {A}")
        elif op == "div":
            acc(a, f"{bo} / {B}")
            acc(b, f"-({bo} * {O}) / {B}")
        elif op == "select":
            acc(a, f"({aux} ? {bo} : (R)0)")
            acc(b, f"({aux} ? (R)0 : {bo})")
        elif op == "bmul":
            acc(a, f"({aux} ? {bo} : (R)0)")
        elif op in ("max", "min"):
            sel = f"!signbit({A} - {B})" if op == "max" else f"signbit({A} - {B})"
            acc(a, f"(({sel}) ? {bo} : (R)0)")
            acc(b, f"(({sel}) ? (R)0 : {bo})")
        elif op == "abs":
            acc(a, f"(signbit({A}) ? -{bo} : {bo})")
        elif op == "pow":
            acc(a, f"{bo} * {B} * pow({A}, {B} - (R)1)")
            acc(b, f"{bo} * {O} * log({A})")
        elif op == "fmod":
            acc(a, bo)
            acc(b, f"-{bo} * trunc({A} / {B})")
        else:
            acc(a, f"{bo} * {self.dfun(op, A, O)}")
        return lines

    def add(self, v, expr):
        """Addition to the adjoint of register v; the first one of its statement sets it (an addition to zero is an
        instruction of its own: 60 of the 140 of the FP64 flux step, whose time is the FP64 pipe's)."""
        first = v in self.fresh
        self.fresh.discard(v)
        return f"b{v} {'' if first else '+'}= {expr};"

    def only_here(self, entry):
        """Registers of a statement whose adjoints receive nothing from the other statements."""
        mine = {o.code for _, o, _, _ in self.tape[entry][1]}
        for i, (_, nodes, store) in enumerate(self.tape):
            if i != entry:
                mine -= {x.code for _, _, ins, _ in nodes for x in ins}
                if store is not None:
                    mine.discard(store[2].code)
        return mine

    def is_shared(self, name):
        """Whether other threads may touch the shadow elements this thread touches: unless every
        access of the array in the kernel goes to one index of the thread's own (the same offsets /
        the same index expressions of the thread indices alone)."""
        ks = self.keys.get(name, set())
        if len(ks) != 1:
            return True
        (kind, k), = ks
        return kind == "i" and any("v_" in x for x in k)

    def check_races(self):
        for name in self.dup:
            if name in self.written and self.is_shared(name):
                raise ArgumentError(f"∇: {name} is written and also accessed at another index in {self.kd.name} "
                                    "(its threads would race)")

    def reverse_lines(self):
        out = []
        for entry in reversed(range(len(self.tape))):
            f, nodes, store = self.tape[entry]
            self.fresh = self.only_here(entry)
            blk = []
            if store is not None:
                name, i3, rhs = store
                if name not in self.dup:  # a constant array: nothing flows back from its elements
                    continue
                k = self.aidx[name]
                g = f"ad_take(d{k}, n{k}_0, n{k}_1, n{k}_2, {i3[0]}, {i3[1]}, {i3[2]})"
                blk.append(self.add(rhs.code, f"(R){g}") if rhs.var else f"(void){g};")
            for op, o, ins, aux in reversed(nodes):
                blk += self.adjoint(op, o, ins, aux)
            if blk:
                out += [f"    if ({f}) {{"] + ["        " + x for x in blk] + ["    }"]
        return out

    # ---- hooks of the kernel template
    def body_lines(self):
        fw = []
        for s in self.kd.body:
            fw += self.stmt(s, 1)
        self.check_races()
        out = fw + ["    if (0) goto ps_fwd_done_;", "ps_fwd_done_:;"]
        if self.mode == "reverse":
            out += self.reverse_lines()
        return out

    def extra_decl(self):
        decl = []
        for name in self.dup:
            decl.append(f"    E* const d{self.aidx[name]} = (E*)g.a[{self.didx[name]}];")
        init = {"R": "0", "long long": "0", "bool": "false"}
        for v, ctype in self.vars:
            decl.append(f"    {ctype} {v} = {init[ctype]};")
        p = "b" if self.mode == "reverse" else "t"
        for v in self.dvars:
            decl.append(f"    R {p}{v} = 0;")
        return decl

    def types(self, real):
        return super().types(real) + "\n" + _HELPERS


class _NoSweep(Exception):
    """The sweep form does not apply to this kernel; one point per thread is generated instead."""


class _AdSweepGen(_AdGen):
    """Reverse kernel of a 2-D or 3-D `@parallel` definition as a sweep along the last dimension.

    With one point per thread every value read from a duplicated array is an atomic addition of its own to
    that array's shadow: 14 per cell for the 3-D flux step with a conductivity array, and their index
    arithmetic and bounds checks, which is what the kernel spends its time on. Here a thread sums what
    flows to an element before it touches memory:

    - a thread keeps the contributions of its point in registers, one per array and offset;
    - those along x move to the thread of the element's column by warp shuffles, those along y through
      shared memory (two buffers in turn, one barrier per plane);
    - those along the sweep accumulate in registers until the sweep has passed the element, which then
      takes one atomic addition. Elements at the edge of a warp's rows, of a block's columns and of a
      chunk of the sweep take one from each side.

    So the flux step makes 2 additions per cell, and 4 one-lane ones per row and plane of a warp. The order
    in which an element's contributions are added was never fixed (atomics) and still is not.

    The values of arrays that the kernel only reads are loaded while the plane before is worked on, and handed from
    offset to offset along the sweep (left to itself the compiler sank the loads to their uses, where each
    waited for the one before: 390 us).

    Every access must be at fixed offsets from the thread's point; the caller (sweep_fits) has checked
    that all of them lie in their arrays, so nothing is checked here, and that 32-bit indices do.
    192^3, FP32: 477 us per launch with one point per thread, 100 so (10 words per cell take 42)."""

    TX, TY = 32, 8            # block of the 3-D form; 2-D: 128 x 1, whose warps exchange nothing
    SMEM = 40 * 1024          # bound on the exchange buffers

    def __init__(self, kd, ndims, dup):
        if kd.kind != "parallel" or ndims not in (2, 3):
            raise _NoSweep
        super().__init__(kd, ndims, dup, "reverse")
        self.access = set()   # (array, offset, left-hand array, its mask): what sweep_fits checks
        self.lhs = None
        self.regs = {}        # statement's left-hand side -> {(read-only array, offset) -> register}
        self.early = None     # the taken shadow's element, where it can be loaded with them

    # ---- accesses: `p<k>` points to the thread's point of array k
    def ref(self, name, o, p="p"):
        k = self.aidx[name]
        o = tuple(o) + (0,) * (3 - len(o))
        if self.lhs is None:
            raise _NoSweep
        self.access.add((name, o) + self.lhs)
        return f"{p}{k}[{o[0]} + n{k}_0 * ({o[1]} + n{k}_1 * {o[2]})]"

    def val(self, name, o):
        if name in self.temps:
            return super().val(name, o)
        if name not in self.aidx:
            raise ArgumentError(f"unknown array {name}")
        return self.load(name, o[:self.nd])

    def load(self, name, ix):
        if any(not isinstance(x, int) for x in ix):
            raise _NoSweep
        r = self.ref(name, ix)
        return f"__ldg(&{r})" if name in self.read_only else r

    def leaf(self, name, idx, key=None):
        if key is None or key[0] != "o":
            raise _NoSweep
        self.key(name, key)
        code = self.ahead(name, key[1]) if name in self.read_only else self.load(name, key[1])
        return self.node("load", code, [], aux=(name, key[1])) if name in self.dup else self.const(code)

    def ahead(self, name, o):
        """The register that holds a read-only array's value, loaded while the plane before was worked on."""
        self.ref(name, o)
        o = tuple(o) + (0,) * (3 - len(o))
        regs = self.regs.setdefault(self.lhs, {})
        return regs.setdefault((name, o), "L%d_%d" % (list(self.regs).index(self.lhs), len(regs)))

    def runs(self, lhs, point=("tx", "ty", "tz")):
        """Every thread of the grid stays for the shuffles and barriers: the columns outside the ranges (in_ false)
        execute no statement."""
        return "in_ && " + super().runs(lhs, point)

    def at_plane(self, z):
        """This thread's point in plane z of the sweep."""
        t3 = ["tx", "ty", "tz"]
        t3[self.nd - 1] = z
        return t3

    def plane_loads(self):
        """(declarations and the first plane's loads, loads of the next plane, their hand-over)"""
        zd = self.nd - 1
        first, nxt, hand = [], [], []
        for lhs, regs in self.regs.items():
            start, later = [], []
            for (name, o), r in regs.items():
                k = self.aidx[name]
                at = f"{o[0]} + n{k}_0 * ({o[1]} + n{k}_1 * {o[2]})"
                first.append(f"    E {r} = 0;")
                start.append(f"{r} = __ldg(&p{k}[{at}]);")
                up = regs.get((name, o[:zd] + (o[zd] + 1,) + o[zd + 1:]))
                nxt.append(f"    E N{r} = {up or '0'};")
                if not up:
                    later.append(f"N{r} = __ldg(&p{k}[st{k}_ + {at}]);")
                hand.append(f"    {r} = N{r};")
            if self.early and lhs == self.early[0]:
                k, at = self.early[1:]
                first.append("    E g_ = 0;")
                start.append(f"g_ = e{k}[{at}];")
                nxt.append("    E Ng_ = 0;")
                later.append(f"Ng_ = e{k}[st{k}_ + {at}];")
                hand.append("    g_ = Ng_;")
            first.append(f"    if ({self.runs(lhs, self.at_plane('z0_'))}) {{ {' '.join(start)} }}")
            nxt.append(f"    if ({self.runs(lhs, self.at_plane('zn_'))} && zn_ < z1_) {{ {' '.join(later)} }}")
        return first, nxt, hand

    def store(self, name, idx, rhs):
        o = self.lhs_offset
        self.emit(f"{self.ref(name, o)} = (E)({rhs.code});")
        self.written.add(name)
        return (name, o, rhs)

    def _stmt(self, s, ind):
        t = s.targets[0] if isinstance(s, ast.Assign) and len(s.targets) == 1 else None
        if isinstance(s, ast.Pass) or isinstance(s, ast.Return) and s.value is None and s is self.kd.body[-1]:
            return
        if not (isinstance(t, ast.Subscript) and isinstance(t.value, ast.Name) and t.value.id.startswith("__lhs_")):
            raise _NoSweep
        sel, name = t.value.id[6:], t.slice.id
        if sel in self.sels and name in self.aidx:
            li = self.sels[sel]
            self.lhs = (name, li)
            self.lhs_offset = tuple((li >> d) & 1 for d in range(self.nd))
        super()._stmt(s, ind)
        self.lhs = None

    # ---- reverse sweep
    def adjoint(self, op, out, ins, aux):
        if op == "load":
            name, o = aux
            k, b = self.aidx[name], f"b{out.code}"
            if self.is_shared(name):
                c = self.contribution(name, o)
                lines = [f"{c} += (E){b};"]
            else:
                self.lhs = self.lhs_of[out.code]
                lines = [f"{self.ref(name, o, 'e')} += (E){b};"]
                self.lhs = None
            return lines
        return super().adjoint(op, out, ins, aux)

    def contribution(self, name, o):
        o = tuple(o) + (0,) * (3 - len(o))
        if max(abs(x) for x in o) > 8:
            raise _NoSweep
        self.contrib.setdefault(name, set()).add(o)
        return "c%d_%d_%d_%d" % ((self.aidx[name],) + tuple(x + 8 for x in o))

    def reverse_lines(self):
        out = []
        self.contrib = {}
        for entry in reversed(range(len(self.tape))):
            f, nodes, store = self.tape[entry]
            if store is None:
                raise _NoSweep
            name, o, rhs = store
            if name not in self.dup:
                continue
            self.fresh = self.only_here(entry)
            li = sum(x << d for d, x in enumerate(o))
            self.lhs_of = {n[1].code: (name, li) for n in nodes}
            self.lhs = (name, li)
            r = self.ref(name, o, "e")
            self.lhs = None
            if len(self.tape) == 1 and self.regs:  # read with the loads of the plane
                self.early = ((name, li), self.aidx[name], r[r.index("[") + 1:-1])
                blk = [f"{r} = (E)0;"]
            else:
                blk = [f"g_ = {r}; {r} = (E)0;"]
            if rhs.var:
                blk.append(self.add(rhs.code, "(R)g_"))
            for op, out_, ins, aux in reversed(nodes):
                blk += self.adjoint(op, out_, ins, aux)
            out += [f"    if ({f}) {{"] + ["        " + x for x in blk] + ["    }"]
        return out

    def body_lines(self):
        fw = []
        for s in self.kd.body:
            fw += self.stmt(s, 1)
        self.check_races()
        rev = self.reverse_lines()
        # an offset that one value has needs no sum
        text = "\n".join(rev)
        for name, offs in self.contrib.items():
            for o in offs:
                c = self.contribution(name, o)
                if text.count(f"{c} += ") == 1:
                    text = text.replace(f"{c} += ", f"{c} = ")
        return fw + text.split("\n")

    # ---- sums over the threads of a block and the planes of a chunk
    def exchange(self, real):
        """(declarations before the sweep, code at the end of a plane, code after the sweep, buffers)"""
        es = {"double": 8, "float": 4}[real]
        pre, put, get, post, nb = [], [], [], [], 0
        zd = self.nd - 1
        for name in self.dup:
            if name not in self.contrib:
                continue
            k, offs = self.aidx[name], self.contrib[name]

            def at(dx, dy, dz):
                return f"e{k} + ({dx} + n{k}_0 * ({dy} + n{k}_1 * {dz}))"

            def off(dx, dy, w):
                return (dx, dy, w) if self.nd == 3 else (dx, w, 0)

            groups = {}  # sweep offset -> {dy -> [dx]} (dy = 0 in 2-D)
            for o in offs:
                groups.setdefault(o[zd], {}).setdefault(o[1] if self.nd == 3 else 0, []).append(o[0])
            mode_x = [o[0] for o in offs]
            x0 = max(sorted(set(mode_x)), key=mode_x.count)
            mode_y = [o[1] for o in offs] if self.nd == 3 else [0]
            y0 = max(sorted(set(mode_y)), key=mode_y.count)
            if max(abs(d - x0) for d in mode_x) > 8 or max(abs(d - y0) for d in mode_y) >= self.TY:
                raise _NoSweep
            wlo, whi = min(groups), max(groups)
            for w in range(wlo, whi + 1):
                q = f"q{k}_{w - wlo}"
                pre.append(f"    E {q} = 0;")
                for dy, dxs in sorted(groups.get(w, {}).items()):
                    h = f"h{k}_{w - wlo}_{dy + 8}"

                    def c(dx):
                        return self.contribution(name, off(dx, dy, w))
                    put.append(f"    E {h} = {c(x0) if x0 in dxs else '(E)0'};")
                    for dx in sorted(dxs):
                        s = dx - x0
                        if s == 0:
                            continue
                        up = "up" if s > 0 else "down"
                        put.append(f"    {{ const E r_ = __shfl_{up}_sync(0xFFFFFFFFu, {c(dx)}, {abs(s)}); "
                                   f"if (lane_ {'>= %d' % s if s > 0 else '< %d' % (32 + s)}) {h} += r_; }}")
                        if s > 0 and x0 - s in dxs:
                            continue  # with its mirror image
                        if x0 - s in dxs:  # both edges of the row in one addition
                            m = x0 - s
                            put.append(f"    if (lane_ < {-s} || lane_ >= {32 + s}) {{ const bool l_ = lane_ < {-s}; "
                                       f"const E v_ = l_ ? {c(dx)} : {c(m)}; "
                                       f"if (v_ != (E)0) ad_red(l_ ? {at(*off(dx, dy, w))} : {at(*off(m, dy, w))}, v_); }}")
                        else:
                            edge = f"lane_ >= {32 - s}" if s > 0 else f"lane_ < {-s}"
                            put.append(f"    if ({edge} && {c(dx)} != (E)0) ad_red({at(*off(dx, dy, w))}, {c(dx)});")
                    if dy == y0:
                        get.append(f"    {q} += {h};")
                        continue
                    t = dy - y0  # to the row t further on
                    put.append(f"    xs_[par_][{nb}][threadIdx.y][lane_] = {h};")
                    edge = f"threadIdx.y >= {self.TY - t}" if t > 0 else f"threadIdx.y < {-t}"
                    inside = f"threadIdx.y >= {t}" if t > 0 else f"threadIdx.y < {self.TY + t}"
                    put.append(f"    if ({edge} && {h} != (E)0) ad_red({at(*off(x0, dy, w))}, {h});")
                    get.append(f"    if ({inside}) {q} += xs_[par_][{nb}][threadIdx.y - ({t})][lane_];")
                    nb += 1
            first = at(*off(x0, y0, wlo))
            get.append(f"    if (q{k}_0 != (E)0) ad_red({first}, q{k}_0);")
            for j in range(whi - wlo):
                get.append(f"    q{k}_{j} = q{k}_{j + 1};")
                post.append(f"    if (q{k}_{j} != (E)0) ad_red(e{k} + (long long)({j}) * st{k}_ + "
                            f"({x0} + n{k}_0 * ({off(x0, y0, wlo)[1]} + n{k}_1 * {off(x0, y0, wlo)[2]})), q{k}_{j});")
            get.append(f"    q{k}_{whi - wlo} = 0;")
        if 2 * nb * self.TX * self.TY * es > self.SMEM:
            raise _NoSweep
        return pre, put, get, post, nb

    def source(self, real):
        kd, nd = self.kd, self.nd
        self.reg = "d" if real == "double" else "f"
        self.collect_temps()
        self.infer_locals(kd.body)
        if self.locals:
            raise _NoSweep
        body = self.body_lines()
        pre, put, get, post, nb = self.exchange(real)
        first, nxt, hand = self.plane_loads()
        zd = nd - 1
        decl, step = [], []
        t0 = ["tx", "ty", "0"] if nd == 3 else ["tx", "0", "0"]
        t0[zd] = "z0_"
        for name, k in self.aidx.items():
            decl.append(f"    const int n{k}_0 = (int)g.n[{k}][0], n{k}_1 = (int)g.n[{k}][1], n{k}_2 = (int)g.n[{k}][2];")
            decl.append(f"    const int st{k}_ = {f'n{k}_0 * n{k}_1' if nd == 3 else f'n{k}_0'};")
            decl.append(f"    E* p{k} = (E*)g.a[{k}] + ({t0[0]} + (long long)n{k}_0 * ({t0[1]} + (long long)n{k}_1 * {t0[2]}));")
            step.append(f"p{k} += st{k}_;")
        for name in self.dup:
            k = self.aidx[name]
            decl.append(f"    E* e{k} = (E*)g.a[{self.didx[name]}] + ({t0[0]} + (long long)n{k}_0 * ({t0[1]} + (long long)n{k}_1 * {t0[2]}));")
            step.append(f"e{k} += st{k}_;")
        for name, k in self.sidx.items():
            ty = "long long" if name in kd.int_scalars else "R"
            decl.append(f"    {ty} s{k} = ({ty})g.s[{k}];")
            if ty == "R":  # kept in a register: converted again on every plane it would cost an FP64 instruction each
                decl.append(f"    asm volatile(\"\" : \"+{self.reg}\"(s{k}));")
        regs = []
        init = {"R": "0", "long long": "0", "bool": "false"}
        for v, ctype in self.vars:
            regs.append(f"    {ctype} {v} = {init[ctype]};")
        for v in self.dvars:
            regs.append(f"    R b{v} = 0;")
        if not self.early:
            regs.append("    E g_ = 0;")
        for name, offs in self.contrib.items():
            for o in sorted(offs):
                regs.append(f"    E {self.contribution(name, o)} = 0;")
        xs = f"    __shared__ E xs_[2][{nb}][{self.TY}][{self.TX}];\n    int par_ = 0;" if nb else ""
        sync = ["    __syncthreads();"] if nb else []
        flip = ["    par_ ^= 1;"] if nb else []
        zblk = "z" if nd == 3 else "y"
        yb = "(int)(blockIdx.y * blockDim.y + threadIdx.y)" if nd == 3 else "0"
        tsweep = "tz" if nd == 3 else "ty"
        ypos = "\n    const int ty = (int)g.lo[1] + uy;" if nd == 3 else ""
        return f"""// reverse derivative of parallel {kd.name} ({nd}-D, {real}, sweep) -- generated by ps_gb300.ad
{self.types(real)}
struct ps_jit_args {{ void* a[{MAX_ARRAYS}]; long long n[{MAX_ARRAYS}][3]; double s[{MAX_SCALARS}]; long long lo[3]; long long cnt[3]; int* err; long long smem; long long loop; unsigned* ocnt; int ord[10]; }};
{VALUE_HELPERS}
__device__ __forceinline__ void ad_red(E* p, E v) {{ asm volatile("red.global.add.{'f64' if real == 'double' else 'f32'} [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "{self.reg}"(v) : "memory"); }}
extern "C" __global__ void __launch_bounds__({self.TX * self.TY if nd == 3 else 128}) ps_jit_entry(const ps_jit_args g) {{
{xs}
    const int lane_ = threadIdx.x & 31;
    const int ux = (int)(blockIdx.x * blockDim.x + threadIdx.x), uy = {yb};
    const bool in_ = ux < g.cnt[0]{" && uy < g.cnt[1]" if nd == 3 else ""};
    const int tx = (int)g.lo[0] + ux;{ypos}
    const int z0_ = (int)(g.lo[{zd}] + blockIdx.{zblk} * g.loop);
    const int z1_ = (int)(min((long long)z0_ + g.loop, g.lo[{zd}] + g.cnt[{zd}]));
{chr(10).join(decl + pre + first)}
    for (int {tsweep} = z0_; {tsweep} < z1_; ++{tsweep}) {{
    const int zn_ = {tsweep} + 1;
{chr(10).join(nxt + regs + body + put + sync + get + flip + hand)}
    {" ".join(step)}
    }}
{chr(10).join(post)}
}}
"""

    def types(self, real):
        return _Gen.types(self, real)


def sweep_fits(spans, dims, lo, cnt, nd):
    """Whether every access of a sweep kernel lies in its array, for all points of the box (lo, cnt) at which
    its statement runs, and 32-bit indices reach every element. spans: (array, left-hand array, its mask,
    least and largest offsets); dims: array -> extents."""
    big = 2 ** 31 - 2 ** 20
    if any(n[0] * n[1] * n[2] >= big for n in dims.values()) or max(lo[d] + cnt[d] for d in range(3)) >= big:
        return False
    for name, lhs, li, omin, omax in spans:
        n, m = dims[name], dims[lhs]
        for d in range(nd):
            end = min(lo[d] + cnt[d], m[d] - 2 * ((li >> d) & 1))
            if end > lo[d] and (lo[d] + omin[d] < 0 or end - 1 + omax[d] >= n[d]):
                return False
    return all(lo[d] == 0 for d in range(nd, 3))


def generate(kd, ndims, dtype, dup, mode="reverse"):
    """CUDA C of the derivative kernel of `kd` (arrays `dup` duplicated; their shadows follow the
    primal arrays in the argument list)."""
    return _AdGen(kd, ndims, set(dup), mode).source(dtype)


def _pairs(kernel: JitKernel, args, grad):
    """`grad` = ((primal, shadow), ...), as ∇=(A->Ā, B->B̄): primals matched to the call's array
    arguments by identity. Returns the duplicated argument names and their shadows in order."""
    names = {}
    for (kind, name), a in zip(kernel.kd.args, args):
        if kind == "array":
            names.setdefault(id(a), name)
    dup = {}
    for pair in grad:
        if len(pair) != 2:
            raise ArgumentError("∇ pairs are (primal, shadow)")
        p, s = pair
        if id(p) not in names:
            raise ArgumentError("∇: a primal is not an array argument of the kernel call")
        n = names[id(p)]
        if n in dup:
            raise ArgumentError(f"∇: {n} appears twice")
        dup[n] = s
    return dup


def _handle(kernel, key, source):
    if key not in kernel._handles:
        h = ctypes.c_void_p()
        _lib.call("ps_jit_compile", source().encode(), b"ps_jit_entry", ctypes.byref(h))
        kernel._handles[key] = h
    return kernel._handles[key]


def generate_sweep(kd, ndims, dtype, dup):
    """(CUDA C, accesses) of the reverse kernel's sweep form, or None where it does not apply."""
    try:
        gen = _AdSweepGen(kd, ndims, set(dup))
        src = gen.source(dtype)
    except _NoSweep:
        return None
    spans = {}  # (array, left-hand array, its mask) -> least and largest offset per dimension
    for name, o, lhs, li in gen.access:
        lo, hi = spans.setdefault((name, lhs, li), (list(o), list(o)))
        for d in range(3):
            lo[d], hi[d] = min(lo[d], o[d]), max(hi[d], o[d])
    return src, [k + v for k, v in sorted(spans.items())]


def _sweep_handle(kernel, ndims, dt, order, descs, lo, cnt):
    """(handle, blocks per SM) of the sweep form for a launch over the box (lo, cnt), or None."""
    key = ("ad_sweep", tuple(order), ndims, dt)
    if key not in kernel._sweeps:
        kernel._sweeps[key] = generate_sweep(kernel.kd, ndims, dt, order)
    if kernel._sweeps[key] is None:
        return None
    src, spans = kernel._sweeps[key][:2]
    dims = {n: d[1] for n, d in zip(kernel.kd.arrays, descs)}
    if not sweep_fits(spans, dims, lo, cnt, ndims):
        return None
    h = _handle(kernel, key, lambda: src)
    if len(kernel._sweeps[key]) == 2:
        kernel._sweeps[key] += (blocks_per_sm(h, _AdSweepGen.TX * _AdSweepGen.TY if ndims == 3 else 128),)
    return h, kernel._sweeps[key][2]


def parallel_grad(kernel: JitKernel, args, grad, ad_mode="reverse", ranges=None, stream=None, sync=True,
                  nblocks=None, nthreads=None):
    """`@parallel ∇=(A->Ā, ...) [ad_mode=...] kernel!(args...)` for a run-time compiled kernel:
    launches the derivative kernel over the kernel's own grid (or `ranges` / nblocks .* nthreads), one
    point per thread, or as a sweep (_AdSweepGen) in FP32 reverse mode. Shadows are arrays of the primals' shapes and number type."""
    require_initialized()
    if not isinstance(kernel, JitKernel):
        raise ArgumentError("∇ applies to run-time compiled kernels (ps_gb300.parallel_kernel)")
    if ad_mode not in MODES:
        raise ArgumentError(f"ad_mode must be one of {MODES}")
    if len(args) != kernel.nargs:
        raise ArgumentError(f"{kernel.name} takes {kernel.nargs} arguments (obtained {len(args)})")
    dup = _pairs(kernel, args, grad)
    arrs, scal = [], []
    for (kind, name), a in zip(kernel.kd.args, args):
        if kind == "array":
            arrs.append(a)
        elif type(a) is float or type(a) is int or isinstance(a, numbers.Real):
            scal.append(float(a))
        else:
            raise ArgumentError(f"{kernel.name}: argument {name} is a scalar (obtained {type(a).__name__})")
    descs = [describe(a) for a in arrs]
    order = [n for n in kernel.kd.arrays if n in dup]
    sdescs = [describe(dup[n]) for n in order]
    primal = dict(zip(kernel.kd.arrays, descs))
    for n, sd in zip(order, sdescs):
        pd = primal[n]
        if sd[1:] != pd[1:]:
            raise ArgumentError(f"∇: the shadow of {n} must have its shape and number type")
    dt = _REALS.get(descs[0][2]) if descs else "double"
    if dt is None or any(d[2] != descs[0][2] for d in descs):
        raise ArgumentError("the array arguments must share one FP64 or FP32 type")
    if len(descs) + len(sdescs) > 32:
        raise ArgumentError("∇: at most 32 arrays and shadows")
    ndims = kernel.ndims or array_ndims(descs)
    lo, cnt = [0, 0, 0], JitKernel._extent(descs, ndims)
    threads = [32, 8, 1]
    if nthreads is not None:
        nt = tuple(int(x) for x in (nthreads if isinstance(nthreads, (tuple, list)) else (nthreads,)))
        threads = list(nt) + [1] * (3 - len(nt))
    if nblocks is not None:
        if nthreads is None:
            raise ArgumentError("nblocks needs nthreads")
        nb = tuple(int(x) for x in (nblocks if isinstance(nblocks, (tuple, list)) else (nblocks,)))
        nb = nb + (1,) * (3 - len(nb))
        cnt = [nb[d] * threads[d] for d in range(3)]
    if ranges is not None:
        lo, hi = ranges_to_box(ranges)
        if min(lo) < 0:
            raise ArgumentError("ranges must start at index 1 or above")
        cnt = [max(0, hi[d] - lo[d]) for d in range(3)]
    loop = [1, 1, 1]
    # FP32 sweeps: 192^3 477 us per launch with one point per thread, 100 so; 2-D 4096^2 994, 111. In FP64 both
    # forms are bound by the FP64 pipe, where the sweep's own sums cost more than the additions they save
    # (200^3: 1.90 ms against 1.41). Below SWEEP_MIN points a launch is shorter than its way through the
    # host, which the sweep's checks make longer (24 x 30 x 26: 58 us without them, 68 with).
    h, points = None, ("ad", ad_mode, tuple(order), ndims, dt)
    if ad_mode == "reverse" and dt == "float" and nthreads is None and nblocks is None and ndims in (2, 3) and \
            cnt[0] * cnt[1] * cnt[2] >= SWEEP_MIN:
        if ("ad_sweep",) + points[2:] not in kernel._handles:
            # The form of one point per thread is compiled before the sweep: a launch under capture, where nothing
            # can be compiled, takes it where the sweep has not run yet.
            h = _handle(kernel, points, lambda: generate(kernel.kd, ndims, dt, order, ad_mode))
        sweep = _sweep_handle(kernel, ndims, dt, order, descs, lo, cnt) if h is None or not capturing(stream) else None
        if sweep is not None:
            h, resident = sweep
            threads = [_AdSweepGen.TX, _AdSweepGen.TY, 1] if ndims == 3 else [128, 1, 1]
            cols = -(-cnt[0] // threads[0]) * (-(-cnt[1] // threads[1]) if ndims == 3 else 1)
            loop[ndims - 1] = sweep_chunk(cnt[ndims - 1], max(1, cols), resident, 3)
    if h is None:
        h = _handle(kernel, points, lambda: generate(kernel.kd, ndims, dt, order, ad_mode))
    alld = descs + sdescs
    A = (PSArray * len(alld))(*alld)
    S = (ctypes.c_double * max(1, len(scal)))(*scal)
    _lib.call("ps_jit_launch_ex", h, A, len(alld), S, len(scal), _I64x3(*lo),
              _I64x3(*cnt), _I32x3(*threads), 0, _I32x3(*loop),
              stream_handle(stream), int(bool(sync)))
