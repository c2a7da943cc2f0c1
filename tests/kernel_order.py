"""Order of the memory accesses of a warp-specialised kernel, from its own source, without a GPU.

`Source` reads the C++ that a kernel is made of; `Run` walks the kernel's body once for every warp, with addresses,
control flow and lane masks exact and all floating-point values unknown, down to the one-instruction helpers (mbarriers,
bulk copies, tensor-core products, tensor-memory loads), which record what they touch and what they order.  The warps,
copies and products are then put together (a wait comes after everything that completes its barrier's phase) and asked:

  problems      does every phase that is waited for complete, with the bytes that its loads bring, and without a circle of waits?
  phases()      does no phase complete before everyone who waits for the one before has seen it (a parity tells only two
                apart), and does no arrival count for an earlier phase?
  races()       of two accesses to the same 16 bytes of shared memory (or place in tensor memory, or in the scratch), one of
                them a write, is one ordered before the other?
  provenance()  did one bulk store of the same place and size leave what a bulk load brings from the scratch?

What is not modelled: proxy fences, the abort path, values.
"""
import re

import numpy as np

LANES = np.arange(32)
SIZES = {"uint8_t": 1, "char": 1, "__nv_bfloat16": 2, "float": 4, "uint32_t": 4, "int": 4, "f32x2": 8, "float2": 8, "uint64_t": 8,
         "float4": 16, "uint4": 16}
TYPES = set(SIZES) | {"bool", "long", "auto", "uint16_t", "TokFrag", "Frag16", "CopyOp", "MmaOp", "Product", "Lane", "unsigned", "void"}
TEMPLATES = {"static_cast", "const_cast", "reinterpret_cast", "tma_wait_group_read", "tma_wait_group", "frag_allreduce2",
             "reg_take", "reg_give", "send_impl", "run_impl", "tok_row_allreduce", "mma_hid64", "mma_64_lead", "mma_hidden_lead", "mma_hidden_ta", "mma_lead", "mma_lead_ta"}
# arithmetic on values, shuffles and fences: no access, no order
PURE = set("""pk pk1 upk hsum add2 mul2 fma2 fmaf rsqrtf gelu_pair2 gelu_grad_h2 f32x2_to_f16x2 f16x2_to_f32x2 f32x2_to_bf16x2
bf16x2_to_f32x2 bf16_lo bf16_hi pack_bf16 make_uint4 make_float2 make_float4 __float_as_uint __uint_as_float __bfloat162float
__float2bfloat16 __shfl_xor_sync __syncwarp __threadfence fence_proxy_async_smem fence_proxy_async_all fence_mbar_init
tc_fence_before_sync tc_fence_after_sync tmem_wait_ld tmem_wait_st tmem_alloc tmem_relinquish tmem_dealloc prefetch_tmap
prefetch_l2 tma_commit_group globaltimer_ns atomicExch reg_take reg_give f16_pack
gelu_half2 atomicXor atomicOr __shfl_down_sync RS_row_layernorm RS_row_sums griddep_launch griddep_wait""".split())


class Unknown:
    """A value that nothing here depends on."""
    def _same(self, *_, **__):
        return self
    __add__ = __radd__ = __sub__ = __rsub__ = __mul__ = __rmul__ = __truediv__ = __rtruediv__ = __neg__ = __xor__ = __rxor__ = \
        __and__ = __rand__ = __or__ = __ror__ = __lshift__ = __rshift__ = __getitem__ = __setitem__ = _same
    __array_ufunc__ = None

    def __bool__(self):
        raise TypeError("control flow on an unmodelled value")


U = Unknown()


class Ptr:
    """space: s (shared memory of CTA `cta`), g (scratch), x (other global memory, not followed)"""
    __array_ufunc__ = None

    def __init__(self, space, addr, size, cta=None):
        self.space, self.addr, self.size, self.cta = space, addr, size, cta

    def __add__(self, n):
        return Ptr(self.space, self.addr + n * self.size, self.size, self.cta)
    __radd__ = __add__


class Struct:
    def __init__(self, **kw):
        self.__dict__.update(kw)

    def copy(self):
        return Struct(**self.__dict__)


class Object:
    """Of a class template that Source.template has read: members and methods share a scope."""

    def __init__(self, walker, constants, methods):
        scope = Scope()
        scope.v.update(constants, n=0, nx=0)
        scope.v.update({name: (scope, prm, body) for name, (prm, body) in methods.items()})
        self.__dict__.update(off=None, scope=scope, walker=walker)

    def __getattr__(self, name):
        v = self.scope.v[name]
        return (lambda *a: self.walker.run(v[1], v[2], list(a), Scope(v[0], self.walker.mask))) if isinstance(v, tuple) else v

    def __setattr__(self, name, v):
        self.scope.v[name] = v


# ------------------------------------------------------------------------------------------------ expressions
TOKEN = re.compile(r"""\s*(?:(?P<num>0x[0-9a-fA-F]+[uUlL]*|\d+\.?\d*(?:e[-+]?\d+)?[fuUlL]*)|(?P<id>[A-Za-z_][\w]*(?:::\w+)*)
|(?P<op><<=|>>=|<<|>>|<=|>=|==|!=|&&|\|\||\+\+|--|->|[-+*/|&^]=|[-+*/%&|^~!<>=?:,.()\[\]{}]))""", re.X)
BINARY = [["||"], ["&&"], ["|"], ["^"], ["&"], ["==", "!="], ["<", ">", "<=", ">="], ["<<", ">>"], ["+", "-"], ["*", "/", "%"]]
LEVEL = {op: i for i, ops in enumerate(BINARY) for op in ops}
ASSIGN = {"=", "+=", "-=", "*=", "/=", "|=", "&=", "^=", "<<=", ">>="}


def tokens(text):
    out, i = [], 0
    text = text.strip()
    while i < len(text):
        m = TOKEN.match(text, i)
        assert m, f"cannot read {text[i:i + 60]!r}"
        out.append(m.group("num") or m.group("id") or m.group("op"))
        i = m.end()
        while i < len(text) and text[i].isspace():
            i += 1
    return out


class Parser:
    def __init__(self, text):
        self.t, self.i = tokens(re.sub(r"decltype\((\w+)\)::value", r"\1", text)), 0

    def peek(self):
        return self.t[self.i] if self.i < len(self.t) else None

    def next(self):
        self.i += 1
        return self.t[self.i - 1]

    def expect(self, x):
        assert self.next() == x, (x, self.t, self.i)

    def expr(self):
        left = self.binary(0)
        if self.peek() == "?":
            self.next()
            a = self.expr()
            self.expect(":")
            return ("tern", left, a, self.expr())
        if self.peek() in ASSIGN:
            op = self.next()
            return ("asg", op, left, self.expr())
        return left

    def binary(self, level):
        left = self.unary()
        while self.peek() in LEVEL and LEVEL[self.peek()] >= level:
            op = self.next()
            left = ("bin", op, left, self.binary(LEVEL[op] + 1))
        return left

    def unary(self):
        p = self.peek()
        if p in ("!", "-", "+", "~", "*", "&", "++", "--"):
            self.next()
            return ("un", p, self.unary())
        return self.postfix()

    def args(self, close):
        out = []
        while self.peek() != close:
            out.append(self.expr())
            if self.peek() == ",":
                self.next()
        self.next()
        return out

    def postfix(self):
        p = self.next()
        if p == "(":
            e = self.expr()
            self.expect(")")
        elif p == "{":
            e = ("init", self.args("}"))
        elif p[0].isdigit():
            e = ("num", int(p.rstrip("uUlL"), 0) if re.fullmatch(r"(0x[\da-fA-F]+|\d+)[uUlL]*", p) else float(p.rstrip("f")))
        else:
            e = ("id", p)
            if p in TEMPLATES and self.peek() == "<":
                self.next()
                targs = []
                while self.peek() != ">":
                    targs.append(self.next())
                self.next()
                e = ("tid", p, [a for a in targs if a != ","])
            elif self.peek() == "{":
                self.next()
                e = ("make", p, self.args("}"))
        while self.peek() in ("(", "[", ".", "->"):
            op = self.next()
            if op == "(":
                e = ("call", e, self.args(")"))
            elif op == "[":
                e = ("idx", e, self.expr())
                self.expect("]")
            else:
                e = ("mem", e, self.next())
        return e


_cache = {}


def parse(text):
    if text not in _cache:
        p = Parser(text)
        _cache[text] = p.expr()
        assert p.peek() is None, f"left over in {text!r}: {p.t[p.i:]}"
    return _cache[text]


# ------------------------------------------------------------------------------------------------ statements
def closing(s, i):
    """Index of the bracket that closes the one at s[i]."""
    depth = 0
    for k in range(i, len(s)):
        if s[k] in "([{":
            depth += 1
        elif s[k] in ")]}":
            depth -= 1
            if depth == 0:
                return k
    raise ValueError(s[i:i + 80])


def split(s, sep=","):
    out, depth, start = [], 0, 0
    for k, c in enumerate(s):
        depth += c in "([{"
        depth -= c in ")]}"
        if c == sep and depth == 0:
            out.append(s[start:k])
            start = k + 1
    return [x.strip() for x in out + [s[start:]] if x.strip()]


DECL = re.compile(r"(?:static |constexpr |const |volatile )*((?:unsigned |long )?[A-Za-z_]\w*)((?:\s|\*|&|const\b)+)(?=[A-Za-z_])")


class Block:
    """Statements of `s`: ("block", [...]), ("if", cond, a, b), ("for", init, cond, inc, body), ("while", cond, body),
    ("lambda", name, params, body), ("decl", type, [(name, how, init)]), ("return", e), ("break",), ("expr", e)"""

    def __init__(self, s):
        self.s, self.i = s, 0

    def ws(self):
        while self.i < len(self.s) and self.s[self.i].isspace():
            self.i += 1

    def all(self):
        out = []
        self.ws()
        while self.i < len(self.s):
            out.append(self.one())
            self.ws()
        return ("block", out)

    def paren(self):
        self.ws()
        e = closing(self.s, self.i)
        inner, self.i = self.s[self.i + 1:e], e + 1
        return inner

    def one(self):
        self.ws()
        s = self.s
        if s[self.i] == "{":
            e = closing(s, self.i)
            inner, self.i = s[self.i + 1:e], e + 1
            return Block(inner).all()
        word = re.match(r"\w+", s[self.i:])
        word = word.group(0) if word else ""
        if word == "if":
            self.i += re.match(r"if(\s+constexpr)?", s[self.i:]).end()
            c = parse(self.paren())
            a = self.one()
            self.ws()
            b = None
            if re.match(r"else\b", s[self.i:]):
                self.i += 4
                b = self.one()
            return ("if", c, a, b)
        if word == "for":
            self.i += 3
            init, cond, inc = (x.strip() for x in self.paren().split(";"))
            return ("for", Block(init + ";").one(), parse(cond), [parse(x) for x in split(inc)], self.one())
        if word == "while":
            self.i += 5
            return ("while", self.paren(), self.one())
        e, depth = self.i, 0
        while s[e] != ";" or depth:
            depth += s[e] in "([{"
            depth -= s[e] in ")]}"
            e += 1
        text, self.i = s[self.i:e].strip(), e + 1
        m = re.match(r"auto (\w+) = \[&\]\(", text)
        if m:
            p = m.end() - 1
            q = closing(text, p)
            body = text[text.index("{", q) + 1:closing(text, text.index("{", q))]
            return ("lambda", m.group(1), params(text[p + 1:q]), Block(body).all())
        if not text or word in ("using", "struct", "static_assert", "extern", "asm"):
            return ("block", [])
        if word == "return":
            return ("return", parse(text[6:]) if text[6:].strip() else None)
        if word == "break":
            return ("break",)
        m = DECL.match(text)
        if m and (m.group(1).split()[-1] in TYPES | {"TokMap", "TokMap16"} or m.group(1).endswith("_object")):
            names = []
            for d in split(text[m.end():]):
                n = re.match(r"[*&\s]*(\w+)", d)
                rest = d[n.end():].strip()
                if rest.startswith("("):
                    names.append((n.group(1), "make", [parse(x) for x in split(rest[1:-1])]))
                else:
                    array = rest.startswith("[")
                    while rest.startswith("["):
                        rest = rest[closing(rest, 0) + 1:].strip()
                    names.append((n.group(1), "array" if array else "plain", parse(rest[1:]) if rest.startswith("=") else None))
            return ("decl", m.group(1), names)
        return ("expr", parse(text))


class Name(str):
    default = None


def params(text):
    """(name, by reference) of each, the name with its default."""
    out = []
    for p in split(text):
        head, _, default = p.partition("=")
        name = Name(re.search(r"(\w+)(?:\)?(?:\[\w*\])*)?$", head.strip()).group(1))
        name.default = default.strip()
        out.append((name, "&" in head or "*" in head))
    return out


def expand(text):
    """Function-like macros, written out."""
    for m in re.finditer(r"^#define (\w+)\(([^)]*)\)((?:.*\\\n)+.*\n)", text, re.M):
        text = text.replace(m.group(0), "")
        while True:
            use = re.search(r"\b%s\(" % m.group(1), text)
            if not use:
                break
            e, body, depth, args, start = closing(text, use.end() - 1), m.group(3).replace("\\\n", "\n"), 0, [], use.end()
            for k in range(use.end(), e + 1):
                depth += text[k] in "([{"
                depth -= text[k] in ")]}"
                if k == e or text[k] == "," and depth == 0:
                    args.append(text[start:k])
                    start = k + 1
            for name, a in zip(split(m.group(2)), args):
                body = re.sub(r"\b%s\b" % name, lambda _: a, body)
            text = text[:use.start()] + body + text[e + 1:]
    return text


class Source:
    """Constants, enums, tables, helper functions and fragment maps of some files; and a kernel's body."""

    def __init__(self, *paths, edit=lambda text: text):
        text = "\n".join(edit(open(p).read()) for p in paths)
        text = expand(re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", text), flags=re.S))
        self.text = re.sub(r"^\s*#.*$", "", text, flags=re.M)
        self.barriers, self.classes = {}, {}
        self.names, self.functions, self.maps = {"true": True, "false": False, "nullptr": 0, "T": True, "F": False}, {}, {}
        ev = lambda e: Walker.constant(self, e)                                                   # noqa: E731
        for m in re.finditer(r"\benum\b[^{;]*\{([^}]*)\}|constexpr (?:int|uint32_t|uint8_t|float) ([^;{}()]*=[^;]*);", self.text):
            if m.group(1) is not None:
                v = -1
                for item in split(m.group(1)):
                    name, _, e = item.partition("=")
                    v = ev(e) if e else v + 1
                    self.names[name.strip()] = v
                if "kBars" in m.group(1):
                    self.barriers = {self.names[n]: n for n in re.findall(r"\w+", m.group(1)) if n in self.names and n[0] != "k"}
            else:
                for item in split(m.group(2)):
                    name, _, e = item.partition("=")
                    try:
                        self.names[name.strip()] = ev(e)
                    except KeyError:
                        pass                                             # a constant of a function's own
        fields = {}
        for m in re.finditer(r"struct (\w+) \{([^}]*)\};", self.text):
            fields[m.group(1)] = [n for d in m.group(2).split(";") if d.strip() for n in split(d.strip().split(None, 1)[1])]
        for m in re.finditer(r"__constant__ const (\w+) (\w+)\[\w+\] = (\{.*?\});", self.text, re.S):
            rows = [[ev(x) for x in split(r[1:-1])] if r[0] == "{" else ev(r) for r in split(m.group(3)[1:-1])]
            self.names[m.group(2)] = Table(fields.get(m.group(1)), rows)
        fn = r"(?:template <([^>]*)>\s*)?(?:static )?(?:__host__ )?__device__ (?:__forceinline__ )?(?:constexpr )?[\w ]+?[\s&*]+(\w+)\("
        for m in re.finditer(fn, self.text):
            q = closing(self.text, m.end() - 1)
            if not re.match(r"\s*\{", self.text[q + 1:q + 5]):
                continue
            b = self.text.index("{", q)
            body = self.text[b + 1:closing(self.text, b)]
            if "asm" not in body and m.group(2) not in PURE:
                tp = [(Name(x.split()[-1]), False) for x in split(m.group(1) or "")]
                self.functions[m.group(2)] = (tp + params(self.text[m.end():q]), body)
        for m in re.finditer(r"struct (TokMap\w*) \{", self.text):
            body = self.text[m.end():closing(self.text, m.end() - 1)]
            init = re.search(r":\s*(quad.*?)\s*\{\}", body, re.S).group(1)
            members = [(x[:x.index("(")], x[x.index("(") + 1:-1]) for x in split(init)]
            methods = re.findall(r"(\w+)\(([^)]*)\) const \{ return (.*?); \}", body)
            self.maps[m.group(1)] = (members, [(n, params(p), e) for n, p, e in methods])

    def template(self, name, prefix, **args):
        """A class template's constants and methods for these arguments; its static ones are also entered as <prefix>name."""
        i = self.text.index("{", re.search(r"struct %s \{" % name, self.text).start())
        body, consts, methods = self.text[i + 1:closing(self.text, i)], dict(args), {}
        for m in re.finditer(r"static constexpr (?:int|uint32_t|bool) (\w+) = ([^;]*);", body):
            sc = Scope()
            sc.v.update(consts)
            consts[m.group(1)] = Walker(self, None).ev(parse(m.group(2)), sc)
        for m in re.finditer(r"(?:template <([^>]*)>\s*)?(?:static )?__device__ __forceinline__ [\w ]+?[\s&*]+(\w+)\(", body):
            q = closing(body, m.end() - 1)
            b = body.index("{", q)
            code = Block(body[b + 1:closing(body, b)]).all()
            methods[m.group(2)] = ([(x.split()[-1], False) for x in split(m.group(1) or "")] + params(body[m.end():q]), code)
        self.names.update({prefix + k: v for k, v in consts.items()})
        self.functions.update({prefix + k: v for k, v in methods.items()})
        self.classes[prefix + "object"] = (consts, methods)
        return consts

    def body(self, kernel):
        i = self.text.index("(", self.text.index(kernel))
        b = self.text.index("{", closing(self.text, i))
        return Block(self.text[b + 1:closing(self.text, b)]).all()


class Table:
    def __init__(self, fields, rows):
        self.fields, self.rows = fields, rows

    def __getitem__(self, i):
        if self.fields is None:
            return self.rows[int(i)]
        if isinstance(i, np.ndarray):
            return Struct(**{f: np.array([self.rows[k][n] for k in i]) for n, f in enumerate(self.fields)})
        return Struct(**dict(zip(self.fields, self.rows[int(i)])))


class Scope:
    def __init__(self, parent=None, mask=None):
        self.v, self.parent, self.mask = {}, parent, mask      # mask: the lanes that its variables exist for

    def find(self, name):
        s = self
        while s is not None:
            if name in s.v:
                return s
            s = s.parent
        return None


class Break(Exception):
    pass


class Return(Exception):
    def __init__(self, value):
        self.value = value


# ------------------------------------------------------------------------------------------------ one warp
class Walker:
    """Walks statements for one warp; `lane`-dependent values are arrays of 32, partial branches narrow `mask`."""

    def __init__(self, source, leaf):
        self.src, self.leaf = source, leaf
        self.mask, self.gone, self.entry = np.ones(32, bool), np.zeros(32, bool), np.ones(32, bool)

    @staticmethod
    def constant(source, text):
        w = Walker(source, None)
        return w.ev(parse(text), Scope())

    # -- values
    def full(self):
        return bool(self.mask.all())

    def merge(self, new, old):
        """A value assigned under the mask."""
        if self.full() or old is U or isinstance(new, (Unknown, Struct)):
            return new
        if isinstance(new, Ptr):
            if not isinstance(old, Ptr):
                old = Ptr(new.space, 0, new.size, new.cta)
            return Ptr(new.space, np.where(self.mask, new.addr, old.addr), new.size, new.cta)
        return np.where(self.mask, new, old)

    def truth(self, c):
        """A condition over the active lanes: True, False, or the array."""
        if isinstance(c, np.ndarray):
            act = c[self.mask].astype(bool)
            return True if act.all() else False if not act.any() else c.astype(bool)
        return bool(c)

    def load(self, p):
        if not isinstance(p, Ptr):
            return U
        return self.leaf.touch(self, p, p.size, False) if p.space != "x" else U

    def ev(self, e, sc):
        k = e[0]
        if k in ("num", "const"):
            return e[1]
        if k == "id":
            s = sc.find(e[1])
            if s is not None:
                return s.v[e[1]]
            if e[1] in self.src.names:
                return self.src.names[e[1]]
            raise KeyError(e[1])
        if k == "bin":
            return self.binary(e[1], e[2], e[3], sc)
        if k == "un":
            return self.unary(e[1], e[2], sc)
        if k == "call":
            return self.call(e, sc)
        if k == "idx":
            a = self.ev(e[1], sc)
            i = self.ev(e[2], sc)
            if isinstance(a, Ptr):
                return self.load(a + i)
            return a[i] if isinstance(a, (list, Table)) and (isinstance(a, Table) or isinstance(i, int)) else U
        if k == "mem":
            a = self.ev(e[1], sc)
            return U if isinstance(a, Unknown) or e[2] in "xyzw" and not hasattr(a, e[2]) else getattr(a, e[2])
        if k == "tern":
            c = self.ev(e[1], sc)
            c = c if isinstance(c, Unknown) else self.truth(c)
            if c is U:
                self.ev(e[2], sc), self.ev(e[3], sc)
                return U
            if c is True or c is False:
                return self.ev(e[2] if c else e[3], sc)
            a, b = self.ev(e[2], sc), self.ev(e[3], sc)
            if isinstance(a, Unknown) or isinstance(b, Unknown):
                return U
            if isinstance(a, Ptr):
                return Ptr(a.space, np.where(c, a.addr, b.addr), a.size, a.cta)
            return np.where(c, a, b)
        if k == "asg":
            return self.assign(e[1], e[2], e[3], sc)
        if k == "init":
            return [self.ev(x, sc) for x in e[1]]
        if k == "make":
            return self.src.names[e[1]] if not e[2] else self.ev(e[2][0], sc)
        raise ValueError(e)

    def binary(self, op, a, b, sc):
        x = self.ev(a, sc)
        if op in ("&&", "||"):
            c = self.truth(x)
            if c is True or c is False:
                return self.ev(b, sc) if c == (op == "&&") else c
            y = self.ev(b, sc)
            return np.logical_and(c, y) if op == "&&" else np.logical_or(c, y)
        y = self.ev(b, sc)
        if isinstance(x, Unknown) or isinstance(y, Unknown):
            return U
        if op == "+":
            return x + y
        if op == "-":
            return x - y
        if op == "*":
            return x * y
        if op == "/":
            return x / y if isinstance(x, float) or isinstance(y, float) else x // y
        if op == "%":
            return x % y
        if op in ("<<", ">>", "&", "|", "^"):
            x, y = (int(v) if isinstance(v, (bool, np.bool_)) else v for v in (x, y))
            return {"<<": lambda: x << y, ">>": lambda: x >> y, "&": lambda: x & y, "|": lambda: x | y, "^": lambda: x ^ y}[op]()
        return {"==": lambda: x == y, "!=": lambda: x != y, "<": lambda: x < y, ">": lambda: x > y, "<=": lambda: x <= y,
                ">=": lambda: x >= y}[op]()

    def unary(self, op, a, sc):
        if op == "&":
            return self.place(a, sc)
        if op in ("++", "--"):
            self.put(a, self.ev(a, sc) + (1 if op == "++" else -1), sc)
            return self.ev(a, sc)
        x = self.ev(a, sc)
        if op == "*":
            return self.load(x)
        if isinstance(x, Unknown):
            return U
        if op == "!":
            return np.logical_not(x) if isinstance(x, np.ndarray) else not x
        return -x if op == "-" else ~x if op == "~" else x

    def place(self, e, sc):
        """An operand's address: pointers into followed memory, else a plain value."""
        if e[0] == "idx":
            a = self.ev(e[1], sc)
            if isinstance(a, Ptr):
                return a + self.ev(e[2], sc)
            return U
        if e[0] == "un" and e[1] == "*":
            return self.ev(e[2], sc)
        return self.ev(e, sc)

    def put(self, e, value, sc):
        if e[0] == "id":
            s = sc.find(e[1])
            same = s.mask is not None and (s.mask == self.mask).all()
            s.v[e[1]] = value if same else self.merge(value, s.v[e[1]])
        elif e[0] == "mem":
            a = self.ev(e[1], sc)
            if isinstance(a, Object):
                setattr(a, e[2], value)
            elif isinstance(a, Struct):
                setattr(a, e[2], self.merge(value, getattr(a, e[2], U)))
        else:
            if e[0] == "idx" and isinstance(self.ev(e[1], sc), (Unknown, list)):
                a, i = self.ev(e[1], sc), self.ev(e[2], sc)
                if isinstance(a, list) and isinstance(i, int):
                    a[i] = value
                return
            p = self.place(e, sc)
            if isinstance(p, Ptr) and p.space != "x":
                self.leaf.touch(self, p, p.size, True)

    def assign(self, op, lhs, rhs, sc):
        v = self.ev(rhs, sc)
        if op != "=":
            v = self.binary(op[:-1], lhs, ("const", v), sc)
        self.put(lhs, v, sc)
        return v

    def call(self, e, sc):
        f, targs = e[1], []
        if f[0] == "tid":
            name, targs = f[1], f[2]
            if name in ("static_cast", "const_cast", "reinterpret_cast"):
                v = self.ev(e[2][0], sc)
                t = [x for x in targs if x not in ("const", "volatile")]
                return Ptr(v.space, v.addr, SIZES[t[0]], v.cta) if isinstance(v, Ptr) and t[-1] == "*" else v
            targs = [self.ev(parse(x), sc) for x in targs]
        elif f[0] == "mem":
            return getattr(self.ev(f[1], sc), f[2])(*[self.ev(x, sc) for x in e[2]])
        else:
            name = f[1]
        s = sc.find(name)
        if s is not None and isinstance(s.v[name], tuple):
            scope, prm, body = s.v[name]
            return self.run(prm, body, targs + [self.ev(x, sc) for x in e[2]], Scope(scope, self.mask))
        if name in PURE:
            for x in e[2]:
                self.ev(x, sc)
            return U
        leaf = getattr(self.leaf, "f_" + name, None)
        if leaf is not None:
            return leaf(self, *targs, *[self.ev(x, sc) for x in e[2]])
        if name not in self.src.functions:
            raise KeyError(f"{name}: neither here nor in the sources")
        prm, body = self.src.functions[name]
        if isinstance(body, str):
            body = Block(body).all()
            self.src.functions[name] = (prm, body)
        return self.run(prm, body, targs + [self.ev(x, sc) for x in e[2]], Scope(None, self.mask))

    def run(self, prm, body, args, scope):
        args = args + [self.ev(parse(n.default), scope) for n, _ in prm[len(args):]]
        for (n, ref), a in zip(prm, args):
            scope.v[n] = a.copy() if isinstance(a, Struct) and not ref and not hasattr(a, "off") else a
        mask, gone, entry = self.mask, self.gone, self.entry
        self.gone, self.entry = np.zeros(32, bool), self.mask
        try:
            self.do(body, scope)
        except Return as r:
            return r.value
        finally:
            self.mask, self.gone, self.entry = mask, gone, entry
        return U

    # -- statements
    def do(self, st, sc):
        k = st[0]
        if k == "block":
            inner = Scope(sc, self.mask)
            for s in st[1]:
                self.do(s, inner)
                if self.gone.any():
                    self.mask = self.mask & ~self.gone
        elif k == "expr":
            self.ev(st[1], sc)
        elif k == "decl":
            for name, how, init in st[2]:
                if how == "make":
                    sc.v[name] = self.make_map(st[1], [self.ev(x, sc) for x in init])
                elif init is not None:
                    v = self.ev(init, sc)
                    sc.v[name] = v.copy() if isinstance(v, Struct) and not hasattr(v, "off") else v
                else:
                    sc.v[name] = Struct() if st[1] in ("Lane", "Product") else \
                        Object(self, *self.src.classes[st[1]]) if st[1].endswith("_object") else U
        elif k == "if":
            c = self.truth(self.ev(st[1], sc))
            if c is True or c is False:
                body = st[2] if c else st[3]
                if body is not None:
                    self.do(body, sc)
                return
            mask = self.mask
            for body, m in ((st[2], mask & c), (st[3], mask & ~c)):
                if body is not None:
                    self.mask = m
                    self.do(body, sc)
            self.mask = mask & ~self.gone
        elif k == "for":
            inner = Scope(sc, self.mask)
            self.do(st[1], inner)
            while self.truth(self.ev(st[2], inner)) is True:
                try:
                    self.do(st[4], inner)
                except Break:
                    break
                for x in st[3]:
                    self.ev(x, inner)
        elif k == "while":
            m = re.fullmatch(r"ok && ld_acquire_cluster\(freed\) < (.*)", st[1])
            assert m, f"loop not modelled: {st[1]}"
            self.leaf.acquire(self, self.ev(parse(m.group(1)), sc))
        elif k == "lambda":
            sc.v[st[1]] = (sc, st[2], st[3])
        elif k == "return":
            v = self.ev(st[1], sc) if st[1] is not None else U
            self.gone = self.gone | self.mask            # these lanes are through
            if not (self.entry & ~self.gone).any():
                raise Return(v)
        elif k == "break":
            raise Break

    def make_map(self, name, args):
        members, methods = self.src.maps[name]
        sc = Scope()
        sc.v.update(warp=args[0], lane=args[1])
        own = Scope(sc)
        for n, x in members:
            own.v[n] = self.ev(parse(x), own)
        m = Struct(**own.v)

        def method(prm, text):
            def f(*a):
                s = Scope(own)
                s.v.update({n: x for (n, _), x in zip(prm, a)})
                return self.ev(parse(text), s)
            return f
        for n, prm, text in methods:
            setattr(m, n, method(prm, text))
        return m


# ------------------------------------------------------------------------------------------------ all warps
class Node:
    __slots__ = ("what", "pred", "reads", "writes", "seen")

    def __init__(self, what, pred):
        self.what, self.pred, self.reads, self.writes = what, list(pred), set(), set()


class Agent:
    """One warp of one CTA: its walker's leaves."""

    def __init__(self, run, cta, warp):
        self.r, self.cta, self.warp = run, cta, warp
        self.name = f"cta {cta} warp {warp}"
        self.at = run.node(f"{self.name} start", [])
        self.tensor = None                              # last product issued
        self.stores = {}                                # lane -> bulk stores not known to be read: [read node, write node]
        self.waits, self.bars = {}, {}

    def sync(self, what, pred=()):
        n = self.r.node(f"{self.name} {what}", [self.at, *pred])
        self.at = self.r.node(f"{self.name} after {what}", [n])
        return n

    def issue(self, what, pred=()):
        """Something that runs on by itself from here."""
        n = self.r.node(f"{self.name} {what}", [self.at, *pred])
        self.at = self.r.node(f"{self.name} after {what}", [self.at])
        return n

    def bar(self, p):
        i = (p.addr - self.r.off_bar) // 8
        return (self.cta if p.cta is None else p.cta, i)

    # -- accesses
    def span(self, cta, addr, nbytes):
        """The places of some bytes of shared memory: of 16, in the vectors of 4."""
        grain = 16 if addr < self.r.vectors else 4
        return {("s", cta, k * grain) for k in range(addr // grain, (addr + nbytes - 1) // grain + 1)}

    def keys(self, w, p, size):
        addr = np.broadcast_to(p.addr, 32)[w.mask]
        return set().union(*[self.span(self.cta if p.cta is None else p.cta, a, size) for a in np.unique(addr).tolist()])

    def touch(self, w, p, size, write):
        if p.space == "s":
            a = np.broadcast_to(p.addr, 32)[w.mask]
            assert (a >= 0).all() and (a + size <= self.r.smem_bytes).all(), "shared memory access out of range"
            if self.r.off_misc <= a[0] < self.r.off_misc + 64:
                return 0                                # flags
            (self.at.writes if write else self.at.reads).update(self.keys(w, p, size))
        return U

    def tmem(self, addr, columns, write):
        lane, col = int(addr) >> 16, int(addr) & 0xffff
        assert col + columns <= 512
        keys = {("t", self.cta, lane // 32, c) for c in range(col // 8, (col + columns + 7) // 8)}
        (self.at.writes if write else self.at.reads).update(keys)
        return U

    def f_tmem_ld8(self, w, addr, v): return self.tmem(addr, 8, False)
    def f_tmem_ld16(self, w, addr, v): return self.tmem(addr, 16, False)
    def f_tmem_ld32(self, w, addr, v): return self.tmem(addr, 32, False)
    def f_tmem_st16(self, w, addr, v): return self.tmem(addr, 16, True)
    def f_tmem_st32(self, w, addr, v): return self.tmem(addr, 32, True)
    def f_tmem_ld_16x256b_x2(self, w, addr, v): return self.tmem(addr, 16, False)
    def f_tmem_ld_16x256b_x4(self, w, addr, v): return self.tmem(addr, 32, False)
    def f_tmem_st_16x256b_x4(self, w, addr, v): return self.tmem(addr, 32, True)

    # -- plain helpers
    def f_smem_u32(self, w, p): return p.addr if p.cta is None else p
    def f_cluster_ctarank(self, w): return self.cta
    def f_elect_one(self, w): return True
    def f___shfl_sync(self, w, m, v, src): return int(np.broadcast_to(v, 32)[0]) if not isinstance(v, Unknown) else U
    def f___all_sync(self, w, m, v): return bool(np.all(v))
    def f_mapa(self, w, addr, rank): return Ptr("s", addr, 1, cta=rank)
    def f_uniform(self, w, v): return v
    def f_long(self, w, v): return v
    def f_min(self, w, a, b): return min(a, b)
    def f_smem_align_1024(self, w, p): return p

    # -- barriers
    def f_mbar_init(self, w, p, count): self.r.count[self.bar(p)] = int(count)

    def arrive(self, b, what, pred=(), times=1):
        n = self.sync(f"arrives at {self.r.label(b)} ({what})", pred)
        self.r.arrivals.setdefault(b, {}).setdefault(self, []).append((n, times))
        return n

    def f_mbar_arrive(self, w, p): self.arrive(self.bar(p), "warp", times=int(w.mask.sum()))
    def f_mbar_arrive_remote(self, w, p, rank): self.arrive((rank, self.bar(p)[1]), "remote", times=int(w.mask.sum()))

    def wait(self, b, phase=None):
        if phase is None:
            phase = self.waits.get(b, 0)
            self.waits[b] = phase + 1
        n = self.sync(f"waits for phase {phase} of {self.r.label(b)}")
        self.r.waiters.append((b, phase, n, self))
        return True

    def f_wait(self, w, b):
        b = np.unique(np.broadcast_to(b, 32)[w.mask])
        assert len(b) == 1
        return self.wait((self.cta, int(b[0])))

    def f_wait_bar(self, w, b, parity=None):
        b = np.unique(np.broadcast_to(b, 32)[w.mask])
        at = (self.cta, int(b[0]))
        assert len(b) == 1 and (parity is None or self.waits.get(at, 0) & 1 == parity & 1), f"{self.name}: not {self.r.label(at)}'s next use"
        return self.wait(at)

    def f_mbar_wait_cl(self, w, p, parity, *_):
        b = self.bar(Ptr("s", int(np.unique(np.broadcast_to(p.addr, 32)[w.mask])[0]), 8))
        assert self.waits.get(b, 0) & 1 == parity, f"{self.name}: the use of {self.r.label(b)} that it waits for is not the next"
        return self.wait(b)

    f_mbar_wait_bounded = f_mbar_wait_cl

    def st_async(self, w, addr, bar, size):
        addr, peer, bar = (np.broadcast_to(v, 32)[w.mask].tolist() for v in (addr.addr, addr.cta, bar.addr))
        for c in sorted(set(peer)):
            to = [(a, b) for a, b, q in zip(addr, bar, peer) if q == c]
            n = self.issue(f"stores into cta {c}")
            n.writes |= set().union(*[self.span(c, a, size) for a, _ in to])
            # (a warp waits for every use of its own CTA's barrier, and sends for a use before it waits for it)
            i = (to[0][1] - self.r.off_bar) // 8
            self.r.loads.append(((c, i), size * len(to), n, self.waits.get((self.cta, i), 0)))

    def f_st_async_f1(self, w, addr, bar, *v): self.st_async(w, addr, bar, 4)
    def f_st_async_f2(self, w, addr, bar, *v): self.st_async(w, addr, bar, 8)
    def f_st_async_f4(self, w, addr, bar, *v): self.st_async(w, addr, bar, 16)

    def f_skip_bar(self, w, b):
        self.waits[self.cta, int(b)] = self.waits.get((self.cta, int(b)), 0) + 1

    def f_bounded(self, w, b, parity):                  # with a parity of the caller's own: the last such phase of its kernel
        phase = self.r.bounded_phase
        assert phase & 1 == parity
        return self.wait((self.cta, int(b)), phase)

    def f_named_bar_sync(self, w, i, threads): self.meet(("named", self.cta, int(i)), threads // 32)

    def f_named_bar_or(self, w, i, threads, v):
        self.f_named_bar_sync(w, i, threads)
        return False

    def f___syncthreads(self, w): self.meet(("cta", self.cta), self.r.warps)

    def f___syncthreads_or(self, w, v):
        self.f___syncthreads(w)
        return False

    def f_cluster_arrive(self, w): self.cluster = self.sync("arrives at the cluster")
    def f_cluster_wait(self, w): self.meet(("cluster",), self.r.warps * self.r.ctas, [self.cluster])

    def meet(self, key, n, pred=()):
        i = self.bars[key] = self.bars.get(key, -1) + 1
        if (key, i) not in self.r.meets:
            self.r.meets[key, i] = (n, self.r.node(f"{key} {i}", []), [])
        m = self.r.meets[key, i]
        before = self.sync(f"reaches {key}", pred)
        m[1].pred.append(before)
        m[2].append(self)
        self.at.pred.append(m[1])

    def f_st_release_cluster(self, w, p, value): self.r.released.append((p.cta, int(value), self.sync("frees")))

    def acquire(self, w, need):
        if need > 0:
            self.r.acquired.append((self.cta, int(need), self.sync(f"sees {need} freed")))

    # -- bulk copies (of the active lanes)
    def f_mbar_expect_tx(self, w, p, nbytes):
        for lane in LANES[w.mask]:
            b = self.bar(Ptr("s", int(np.broadcast_to(p.addr, 32)[lane]), 8))
            self.arrive(b, "expects bytes")
            self.r.expected.setdefault(b, []).append(int(np.broadcast_to(nbytes, 32)[lane]))

    def f_arm(self, w, b, nbytes): self.f_mbar_expect_tx(w, Ptr("s", self.r.off_bar + b * 8, 8), nbytes)

    def load_one(self, dst, nbytes, bar, reads):
        b = self.bar(Ptr("s", bar, 8))
        n = self.issue(f"load for {self.r.label(b)}")
        assert dst % 16 == 0 and 0 <= dst and dst + nbytes <= self.r.smem_bytes
        n.writes |= self.span(self.cta, dst, nbytes)
        n.reads |= reads
        self.r.loads.append((b, nbytes, n, None))

    def each(self, w, *vals):
        return zip(*[np.broadcast_to(v.addr if isinstance(v, Ptr) else v, 32)[w.mask].tolist() for v in vals])

    def f_tma_load_2d(self, w, dst, tmap, bar, x, y):
        for d, b in self.each(w, dst, bar):
            self.load_one(d, 8192, b, set())

    def scratch(self, addr, nbytes):
        base = addr >> 40
        if base not in self.r.scratch:
            return set()
        assert (addr & (1 << 40) - 1) + nbytes <= self.r.scratch[base] and nbytes % 256 == 0
        return {("g", (addr + k) >> 8) for k in range(0, nbytes, 256)}

    def f_bulk_load_1d(self, w, dst, src, nbytes, bar):
        for d, s, n, b in self.each(w, dst, src, nbytes, bar):
            self.load_one(d, n, b, self.scratch(s, n))

    def store(self, lane, src, nbytes, writes):
        read = self.issue(f"store from {src}")
        read.reads |= self.span(self.cta, src, nbytes)
        done = self.r.node(f"{self.name} store's end", [read])
        done.writes |= writes
        self.stores.setdefault(lane, []).append([read, done])

    def f_bulk_store_1d(self, w, dst, src, nbytes):
        for lane, d, s, n in self.each(w, LANES, dst, src, nbytes):
            self.store(lane, s, n, self.scratch(d, n))

    def f_tma_store_2d(self, w, tmap, src, x, y):
        for lane, s in self.each(w, LANES, src):
            self.store(lane, s, 8192, set())

    def f_tma_wait_group_read(self, w, left, end=0):
        done = []
        for lane in LANES[w.mask].tolist():
            q = self.stores.get(lane, [])
            for x in q[:len(q) - left]:
                done += [x[end]] if x[end] is not None else []
                x[0] = x[end] = None
        self.sync("waits for its stores", done)

    def f_tma_wait_group(self, w, left): self.f_tma_wait_group_read(w, left, 1)

    # -- products
    def rows(self, desc, first, n):
        """The 16-byte chunks that an operand's K step reads."""
        a = (desc & 0x3fff) << 4
        if first:                                       # K-major: n rows of 32 bytes
            r = np.arange(n)
            c = (a >> 4) & 7
            base = (a & ~127) // 16 + (r // 8) * 64 + (r % 8) * 8
            return np.concatenate([base + ((c + h) ^ (r & 7)) for h in (0, 1)])
        blocks = range(max(1, n // 64))                 # MN-major: 16 rows of 128 bytes per block of 64
        return np.concatenate([a // 16 + blk * ((desc >> 16) & 0x3fff) + np.arange(128) for blk in blocks])

    def product(self, d, a, b, idesc, a_tmem=False):
        n, m = (idesc >> 17 & 63) * 8, (idesc >> 24 & 31) * 16
        if self.tensor is None or self.tensor[1] is not self.at:
            self.tensor = (self.issue("product", [self.tensor[0]] if self.tensor else []), None)
            self.tensor = (self.tensor[0], self.at)
        t = self.tensor[0]
        if a_tmem:
            t.reads |= {("t", self.cta, q, (a & 0xffff) // 8) for q in range(4)}
        else:
            t.reads |= {("s", self.cta, int(k) * 16) for k in self.rows(a, not idesc >> 15 & 1, m)}
        # (a product of 16 columns is a row sum: only its first column is used, the others multiply what happens to lie there)
        t.reads |= {("s", self.cta, int(k) * 16) for k in self.rows(b, not idesc >> 16 & 1, 1 if n == 16 else n)}
        t.writes |= {("t", self.cta, q, c) for q in range(4) for c in range((d & 0xffff) // 8, ((d & 0xffff) + n) // 8)}
        assert (d & 0xffff) + n <= 512

    def f_mma_lead(self, w, acc, d, a, b, idesc, lead): self.product(d, a, b, idesc)
    def f_mma_lead_rt(self, w, d, a, b, idesc, acc, lead): self.product(d, a, b, idesc)
    def f_mma_issue_rt(self, w, d, a, b, idesc, acc): self.product(d, a, b, idesc)
    def f_mma_lead_ta(self, w, acc, d, a, b, idesc, lead): self.product(d, a, b, idesc, True)
    def f_umma_commit(self, w, p): self.arrive(self.bar(p), "products", [self.tensor[0]] if self.tensor else [])

    def f_ld_cluster_f32(self, w, p):
        self.at.reads.update(self.keys(w, p, 4))
        return U


class Run:
    """All warps of one cluster.  `params`: the kernel's argument struct and constants; `scratch`: allocations behind the
    scratch pointers (their addresses are (index << 40) + offset) and their sizes."""

    def __init__(self, source, kernel, params, scratch, ctas, warps, skip=("bounded", "wait", "arm", "uniform"), prefix="",
                 vectors=None):
        self.src, self.ctas, self.warps, self.scratch = source, ctas, warps, scratch
        self.off_bar, self.off_misc, self.smem_bytes = (source.names[prefix + k] for k in ("OFF_BAR", "OFF_MISC", "SMEM_BYTES"))
        self.vectors = self.smem_bytes if vectors is None else vectors      # where accesses are told apart by 4 bytes
        self.nodes, self.count, self.meets = [], {}, {}
        self.arrivals, self.expected, self.waiters, self.loads = {}, {}, [], []
        self.released, self.acquired = [], []
        body = source.body(kernel)
        body = ("block", [s for s in body[1] if not (s[0] == "lambda" and s[1] in skip)])
        for cta in range(ctas):
            for warp in range(warps):
                a = Agent(self, cta, warp)
                w = Walker(source, a)
                sc = Scope()
                sc.v.update(params, smem=Ptr("s", 0, 1), smem_raw=Ptr("s", 0, 1), threadIdx=Struct(x=warp * 32 + LANES), blockIdx=Struct(x=cta))
                inner = Scope(sc)
                self.agent_scope = inner
                try:
                    for s in body[1]:
                        if s[0] != "block" or s[1]:
                            w.do(s, inner)
                except Return:
                    pass
        self.link()

    def node(self, what, pred):
        n = Node(what, pred)
        self.nodes.append(n)
        return n

    @property
    def bounded_phase(self):
        return self.agent_scope.v["nrec"] - 1

    def label(self, b):
        return f"{self.src.barriers.get(b[1], b[1])} of cta {b[0]}"

    # -- what orders what
    def link(self):
        self.problems = []
        # a phase takes the same share of every agent's arrivals; but one agent may complete the first by itself
        self.phase, arrived = {}, {}
        for b, by in self.arrivals.items():
            count, ph = self.count[b], self.phase.setdefault(b, {})
            whole = [n for x in by.values() for n, times in x[:1] if times == count > 1]
            lists = [[n for n, times in x for _ in range(times) if n not in whole] for x in by.values()]
            phases, rest = divmod(sum(map(len, lists)), count)
            if rest or len(whole) > 1 or any(len(x) % max(phases, 1) for x in lists):
                self.problems.append(f"{self.label(b)}: {[len(x) for x in lists]} arrivals, {count} to a phase")
                continue
            for x in lists:
                for k, n in enumerate(x):
                    ph.setdefault(k * phases // len(x) + len(whole), []).append(n)
            arrived[b] = {k: len(v) for k, v in ph.items()}
            if whole:
                ph[0], arrived[b][0] = whole, count
        brought = {}
        for b, nbytes, n, k in self.loads:              # k: the phase, of a CTA's own loads the first that is not complete
            got, want = brought.setdefault(b, [0] * len(self.expected[b])), self.expected[b]
            if k is None:
                k = next((i for i, x in enumerate(got) if x < want[i]), len(got) - 1)
            got[k] += nbytes
            self.phase[b].setdefault(k, []).append(n)
        for b, got in brought.items():
            if got != self.expected[b]:
                self.problems.append(f"{self.label(b)}: {got} bytes, expected {self.expected[b]}")
        for b, phase, n, a in self.waiters:
            by = self.phase.get(b, {}).get(phase, [])
            if arrived.get(b, {}).get(phase) != self.count[b]:
                self.problems.append(f"{n.what}: never completes")
            n.pred += by
        for cta, need, n in self.acquired:               # (released in rising order by one warp)
            first = next((r for c, v, r in self.released if c == cta and v >= need), None)
            if first is None:
                self.problems.append(f"{n.what}: never freed")
            else:
                n.pred.append(first)
        for (key, i), (n, _, who) in self.meets.items():
            if len(who) != n:
                self.problems.append(f"{key} {i}: {len(who)} of {n} warps")
        # a linear order
        left = {id(n): len(n.pred) for n in self.nodes}
        succ = {}
        for n in self.nodes:
            for p in n.pred:
                succ.setdefault(id(p), []).append(n)
        ready, self.order = [n for n in self.nodes if not n.pred], []
        while ready:
            n = ready.pop()
            self.order.append(n)
            for s in succ.get(id(n), ()):
                left[id(s)] -= 1
                if not left[id(s)]:
                    ready.append(s)
        if len(self.order) != len(self.nodes):
            stuck = [n.what for n in self.nodes if left[id(n)]]
            self.problems.append(f"waits in a circle, among them {stuck[:4]}")
            return
        index = {id(n): i for i, n in enumerate(self.order)}
        for i, n in enumerate(self.order):
            seen = 1 << i
            for p in n.pred:
                seen |= p.seen
            n.seen = seen
        for n in self.order:
            n.seen = n.seen.to_bytes(len(self.order) // 8 + 1, "little")
        self.index = index

    def before(self, a, b):
        """a is ordered before b (or is b)."""
        i = self.index[id(a)]
        return b.seen[i >> 3] >> (i & 7) & 1

    def phases(self):
        """Phases that complete before the one before has been seen, arrivals that could count too early."""
        bad = set()
        for b, phase, n, a in self.waiters:
            later = self.phase[b].get(phase + 1)
            if later and not any(self.before(n, x) for x in later):
                bad.add((self.label(b), "completes again before a waiter has seen it", a.name))
        for b, ph in self.phase.items():
            for k in ph:
                for x in ph.get(k + 1, ()):
                    if not all(self.before(y, x) for y in ph[k]):
                        bad.add((self.label(b), "takes an arrival for the phase before", x.what))
        return bad

    def races(self):
        """Unordered accesses: (place, access, access)."""
        bad, last = {}, {}                               # place -> last write, reads since
        for n in self.order:
            fine = {}

            def after(x, key):
                if x is not None and x is not n:
                    if id(x) not in fine:
                        fine[id(x)] = self.before(x, n)
                    if not fine[id(x)]:
                        bad.setdefault((x.what, n.what), key)
            for key in n.reads:
                w, rs = last.setdefault(key, (None, []))
                after(w, key)
                rs.append(n)
            for key in n.writes:
                w, rs = last.get(key, (None, ()))
                after(w, key)
                for r in rs:
                    after(r, key)
                last[key] = (n, [])
        return [(key, a, b) for (a, b), key in bad.items()]

    def provenance(self):
        """Loads from the scratch that are not of one store's place and size."""
        bad, last = [], {}
        for n in self.order:
            if any(k[0] == "g" for k in n.reads):
                keys = {k for k in n.reads if k[0] == "g"}
                if len({id(last.get(k)) for k in keys}) != 1 or last.get(next(iter(keys))) is None or \
                        last[next(iter(keys))].writes != keys:
                    bad.append(n.what)
            for k in n.writes:
                if k[0] == "g":
                    last[k] = n
        return bad
