"""
Discrete adjoint of the fused tissue step.

For a loss on logged membrane potentials,
``L = sum over probes p and log points j of (V_p(t_j) - target_pj)^2``,
the gradients with respect to per-cell scalar fields (for example GKr and
GNa scale fields) and to the diffusion conductances gx, gy are computed by
reverse-mode differentiation of the discrete forward map (forward Euler or
Rush-Larsen, plus the diffusion stencil), not of the ODEs: they are the
exact gradients of what the forward kernel computes, up to rounding.

- :func:`local_partial` differentiates one equation's right-hand side with
  respect to one referenced variable, all other references held fixed (the
  reference's ``Expression.diff``, ``myokit/_expressions.py:243``, expands
  intermediate variables instead; here every equation is differentiated
  locally and the chain rule runs through the generated reverse sweep).
- :class:`AdjointKernel` emits, from the forward :class:`TissueKernel`'s
  equation list, a CUDA kernel that re-evaluates the model at step k from a
  recorded trajectory and sweeps the equations in reverse.
  For small grids two kernels instead: the sparse matrix of every cell and
  step at once, and a sweep that multiplies through them.
- :class:`TissueAdjoint` runs forward with checkpoints every K steps, then
  per segment (last first) recomputes the trajectory and runs the adjoint
  kernels; :class:`TissueLossFunction` wraps this as a
  ``torch.autograd.Function``.
"""
import math

import numpy as np

from ._deps import myokit
from . import exporter as _exp
from . import _lib
from . import autotune

_N = myokit.Number
# Tiles per SM up to which the reverse goes by tape and sweep, where the
# sweep's registers allow it. ms forward and backward, general and so: 8
# states, double precision, 200 steps: 2 tiles in all 9.9, 2.0; 100 steps: one
# tile per SM 6.0, 2.7; four 6.6, 4.4; eight 8.9, 8.1. Single precision, 100
# steps: four 1.45, 1.25; eight 1.78, 1.61; ten 1.90, 1.91. 48 states, single
# precision, 100 steps: one 2.42, 1.94; three (all that fit) 3.15, 2.89.
_MAP_TILES = 8


def _mul(a, b):
    if a is None or b is None:
        return None
    return myokit.Multiply(a, b)


def _add(a, b):
    if a is None:
        return b
    if b is None:
        return a
    return myokit.Plus(a, b)


def _sub(a, b):
    if b is None:
        return a
    if a is None:
        return myokit.PrefixMinus(b)
    return myokit.Minus(a, b)


def local_partial(e, ref):
    """
    Partial derivative of expression ``e`` with respect to the
    :class:`myokit.Name` (or ``Derivative``) ``ref``, treating every other
    reference as a constant. Returns an expression or ``None`` for zero.
    Conditionals differentiate their branches (right derivatives at the
    switching points), as ``Expression.diff`` does.
    """
    d = lambda x: local_partial(x, ref)  # noqa: E731
    if isinstance(e, (myokit.Name, myokit.Derivative)):
        return _N(1) if e == ref else None
    if isinstance(e, myokit.Number):
        return None
    if isinstance(e, myokit.PrefixPlus):
        return d(e[0])
    if isinstance(e, myokit.PrefixMinus):
        x = d(e[0])
        return None if x is None else myokit.PrefixMinus(x)
    if isinstance(e, myokit.Plus):
        return _add(d(e[0]), d(e[1]))
    if isinstance(e, myokit.Minus):
        return _sub(d(e[0]), d(e[1]))
    if isinstance(e, myokit.Multiply):
        return _add(_mul(d(e[0]), e[1]), _mul(e[0], d(e[1])))
    if isinstance(e, myokit.Divide):
        a, b = e[0], e[1]
        da, db = d(a), d(b)
        out = None if da is None else myokit.Divide(da, b)
        if db is not None:
            out = _sub(out, myokit.Divide(myokit.Multiply(a, db),
                                          myokit.Power(b, _N(2))))
        return out
    if isinstance(e, myokit.Power):
        a, b = e[0], e[1]
        da, db = d(a), d(b)
        out = None
        if da is not None:
            if isinstance(b, myokit.Number):
                p = b.eval()
                out = myokit.Multiply(
                    myokit.Multiply(_N(p), myokit.Power(a, _N(p - 1))), da)
            else:
                out = myokit.Multiply(
                    myokit.Multiply(b, myokit.Power(a, myokit.Minus(b, _N(1)))),
                    da)
        if db is not None:
            out = _add(out, myokit.Multiply(
                myokit.Multiply(e, myokit.Log(a)), db))
        return out
    if isinstance(e, myokit.Exp):
        x = d(e[0])
        return None if x is None else myokit.Multiply(e, x)
    if isinstance(e, myokit.Log):
        if len(e) == 1:
            x = d(e[0])
            return None if x is None else myokit.Divide(x, e[0])
        # log_b(a) = ln a / ln b
        return d(myokit.Divide(myokit.Log(e[0]), myokit.Log(e[1])))
    if isinstance(e, myokit.Log10):
        x = d(e[0])
        return None if x is None else myokit.Divide(
            x, myokit.Multiply(e[0], _N(math.log(10))))
    if isinstance(e, myokit.Sqrt):
        x = d(e[0])
        return None if x is None else myokit.Divide(
            x, myokit.Multiply(_N(2), e))
    if isinstance(e, myokit.Sin):
        x = d(e[0])
        return None if x is None else myokit.Multiply(myokit.Cos(e[0]), x)
    if isinstance(e, myokit.Cos):
        x = d(e[0])
        return None if x is None else myokit.PrefixMinus(
            myokit.Multiply(myokit.Sin(e[0]), x))
    if isinstance(e, myokit.Tan):
        x = d(e[0])
        return None if x is None else myokit.Divide(
            x, myokit.Power(myokit.Cos(e[0]), _N(2)))
    if isinstance(e, myokit.ASin):
        x = d(e[0])
        return None if x is None else myokit.Divide(x, myokit.Sqrt(
            myokit.Minus(_N(1), myokit.Power(e[0], _N(2)))))
    if isinstance(e, myokit.ACos):
        x = d(e[0])
        return None if x is None else myokit.PrefixMinus(myokit.Divide(
            x, myokit.Sqrt(myokit.Minus(_N(1), myokit.Power(e[0], _N(2))))))
    if isinstance(e, myokit.ATan):
        x = d(e[0])
        return None if x is None else myokit.Divide(x, myokit.Plus(
            _N(1), myokit.Power(e[0], _N(2))))
    if isinstance(e, (myokit.Floor, myokit.Ceil, myokit.Quotient)):
        return None
    if isinstance(e, myokit.Remainder):
        return _sub(d(e[0]), _mul(d(e[1]), myokit.Floor(
            myokit.Divide(e[0], e[1]))))
    if isinstance(e, myokit.Abs):
        x = d(e[0])
        return None if x is None else myokit.If(
            myokit.MoreEqual(e[0], _N(0)), x, myokit.PrefixMinus(x))
    if isinstance(e, myokit.If):
        t, f = d(e._t), d(e._e)
        if t is None and f is None:
            return None
        return myokit.If(e._i, t or _N(0), f or _N(0))
    if isinstance(e, myokit.Piecewise):
        parts = [d(x) for x in e._e]
        if all(p is None for p in parts):
            return None
        args = []
        for c, p in zip(e._i, parts[:-1]):
            args.extend([c, p or _N(0)])
        args.append(parts[-1] or _N(0))
        return myokit.Piecewise(*args)
    if isinstance(e, (myokit.Condition,)):
        return None
    raise NotImplementedError(
        'No local derivative for ' + type(e).__name__)


def _references(e):
    """Names and derivatives referenced in e (unique, stable order)."""
    seen = []
    for x in e.walk():
        if isinstance(x, (myokit.Name, myokit.Derivative)) and x not in seen:
            seen.append(x)
    return seen


class AdjointKernel(object):
    """
    CUDA source for the adjoint of a forward :class:`TissueKernel`: the
    trajectory-writing forward kernel and the reverse kernel, in one module.
    Supports forward-Euler and Rush-Larsen updates, every diffusion mode
    (homogeneous or per-edge conductances on a 1D or 2D grid, arbitrary
    connections, none) and scalar fields.
    """
    def __init__(self, fwd, min_blocks=1, threads=None, guards=True,
                 tiles_per_sm=0):
        self.fwd = fwd
        self.single = fwd.single
        self.min_blocks = int(min_blocks)
        self.threads = int(threads or fwd.block[0])
        if self.threads % 32 or not 32 <= self.threads <= 1024:
            raise ValueError('threads must be a multiple of 32 up to 1024')
        self.guards = bool(guards)
        self._key = None
        # Numbers per cell and step on the tape, and warps per tile of the
        # sweep (0: the general reverse kernel)
        self.slots = self.parts = 0
        self._source = self._generate_map(tiles_per_sm) \
            if tiles_per_sm else None
        if self._source is None:
            self._source = self._generate()

    def _forward_values(self, tab):
        """The model's variables at step k, from the trajectory."""
        fwd = self.fwd
        name = fwd._name
        fw = []
        for i, s in enumerate(fwd.states):
            fw.append(f'{tab}const Real {name(s)} = xk[(long long){i}'
                      f' * pitch + cid];')
        for k, var in enumerate(fwd.fields):
            fw.append(f'{tab}const Real {name(var)} = '
                      f'field[(long long){k} * pitch + cid];')
        for lhs, rhs in fwd.cell_const_eqs:
            fw.append(f'{tab}const Real {name(lhs)} = {fwd.writer.ex(rhs)};')
        for lhs, rhs in fwd.rhs_eqs:
            fw.append(f'{tab}const Real {name(lhs)} = '
                      f'{fwd.rhs_code(lhs, rhs)};')
        return fw

    def _generate(self):
        fwd = self.fwd
        w = fwd.writer
        name = fwd._name
        tab = '            '
        states = fwd.states
        fw = self._forward_values(tab)

        # Adjoint accumulators: every state, field, per-cell constant,
        # equation left-hand side and the diffusion current
        acc = []

        def A(n):
            return 'A' + n

        accs = [name(s) for s in states] + [name(v) for v in fwd.fields]
        accs += [name(lhs) for lhs, _ in fwd.cell_const_eqs]
        accs += [name(lhs) for lhs, _ in fwd.rhs_eqs]
        accs.append(_exp._IDIFF)
        seen = set()
        for n in accs:
            if n not in seen:
                acc.append(f'{tab}Real {A(n)} = 0;')
                seen.add(n)

        def ref(var):
            x = fwd.literal_subst.get(myokit.Name(var))
            return w.ex(x) if x is not None else name(var)

        # Seeds: lambda_{k+1} through the update of each state
        seeds = list(acc)
        for i, s in enumerate(states):
            lam = f'lam[(long long){i} * pitch + cid]'
            if i == fwd.i_vm:
                lam = f'({lam} + gather)'
            n = name(s)
            seeds.append(f'{tab}{{ const Real l_ = {lam};')
            if s in fwd.rl_states:
                inf, tau = fwd.rl_states[s]
                ri, rt = ref(inf), ref(tau)
                seeds.append(f'{tab}  const Real E_ = '
                             f'{fwd.decay(tau, rt, fwd.rates)};')
                seeds.append(f'{tab}  {A(n)} = {w.fma("l_", "E_", A(n))};')
                if myokit.Name(inf) not in fwd.literal_subst:
                    a = A(name(inf))
                    seeds.append(f'{tab}  {a} = {w.fma("l_", "1 - E_", a)};')
                if myokit.Name(tau) not in fwd.literal_subst:
                    num = f'-l_ * ({ri} - {n}) * E_ * dt_'
                    den = f'{rt} * {rt}'
                    q = f'{num} / ({den})' if self.single else \
                        f'mkg_div({num}, {den})'
                    seeds.append(f'{tab}  {A(name(tau))} += {q};')
            else:
                seeds.append(f'{tab}  {A(n)} += l_;')
                a = A(name(s.lhs()))
                seeds.append(f'{tab}  {a} = {w.fma("l_", "dt_", a)};')
            seeds.append(f'{tab}}}')

        # Reverse sweep: equations in reverse evaluation order
        rev = []
        valid = set(seen)
        for lhs, rhs in reversed(fwd.rhs_eqs + []):
            a = A(name(lhs))
            terms = []
            bcd = fwd.cubic.get(name(lhs))
            if bcd is not None:
                # A refined root x of x^3 + b x^2 + c x + d: by the implicit
                # function theorem dx/db = -x^2/g, dx/dc = -x/g, dx/dd = -1/g
                # with g = 3x^2 + 2bx + c
                x = name(lhs)
                b, c, d = bcd
                g = w.fma(w.fma('2', b, f'3 * {x}'), x, c)
                terms.append(f'{tab}    const Real g_ = {g};')
                terms.append(f'{tab}    const Real r_ = (g_ != 0) ? a_ / g_'
                             ' : (Real)0;')
                for rn, dx in ((b, f'{x} * {x}'), (c, x), (d, '1')):
                    if rn in valid:
                        a = A(rn)
                        terms.append(
                            f'{tab}    {a} = {w.fma("-r_", dx, a)};')
                rhs = myokit.Number(0)   # no further terms
            for r in _references(rhs):
                rn = name(r)
                if rn in (_exp._T, _exp._PACE):
                    continue
                if rn not in valid:
                    continue
                dp = local_partial(rhs, r)
                if dp is None:
                    continue
                terms.append(f'{tab}    {A(rn)} = '
                             f'{w.fma("a_", w.ex(dp), A(rn))};')
            if terms:
                # With guards an equation whose adjoint is still zero is
                # skipped; without, the sweep is straight-line code
                if self.guards:
                    rev.append(f'{tab}if ({a} != 0) {{ const Real a_ = {a};')
                else:
                    rev.append(f'{tab}{{ const Real a_ = {a};')
                rev.extend(terms)
                rev.append(f'{tab}}}')
        for lhs, rhs in reversed(fwd.cell_const_eqs):
            a = A(name(lhs))
            for r in _references(rhs):
                rn = name(r)
                if rn not in valid:
                    continue
                dp = local_partial(rhs, r)
                if dp is None:
                    continue
                rev.append(f'{tab}{A(rn)} = {w.fma(a, w.ex(dp), A(rn))};')

        # Outputs
        out = []
        for i, s in enumerate(states):
            n = name(s)
            extra = ''
            if i == fwd.i_vm and fwd.diffusion != _exp.DIFF_NONE:
                extra = f' + {A(_exp._IDIFF)} * cdiag'
            out.append(f'{tab}lam[(long long){i} * pitch + cid] = '
                       f'{A(n)}{extra};')
        for k, var in enumerate(fwd.fields):
            out.append(f'{tab}gfield[(long long){k} * pitch + cid] += '
                       f'{A(name(var))};')
        if fwd.diffusion != _exp.DIFF_NONE:
            out.append(f'{tab}mu_out[cid] = {A(_exp._IDIFF)};')
            out.append(f'{tab}gg[cid] += {A(_exp._IDIFF)} * xterm;')
            out.append(f'{tab}gg[pitch + cid] += {A(_exp._IDIFF)} * yterm;')

        loss_target = A(name(states[fwd.i_vm])) if fwd.i_vm >= 0 else \
            A(name(fwd.vm))
        subs = {
            '@ADJ_MINB@': str(self.min_blocks),
            '@ADJ_BX@': str(self.threads),
            '@FORWARD@': '\n'.join(fw),
            '@SEEDS@': '\n'.join(seeds),
            '@LOSS_TARGET@': loss_target,
            '@REVERSE@': '\n'.join(rev),
            '@OUTPUTS@': '\n'.join(out),
            '@IDIFF_ADJ@': A(_exp._IDIFF),
        }
        text = _exp._read('tissue_adjoint.cu.in')
        for k, v in subs.items():
            text = text.replace(k, v)
        # The forward kernel with trajectory output, in the same module
        return self._join(fwd.source(), text)

    def _step_matrix(self, tab):
        """
        ``(partials, rows, entries)``: the code of the local partial
        derivatives and of the rows of the matrix of one step, and per
        column name the ``(state, slot)`` of its entries. A forward Euler
        state's row is the identity plus its entries.
        """
        fwd = self.fwd
        w = fwd.writer
        name = fwd._name
        states = fwd.states
        equations = fwd.cell_const_eqs + fwd.rhs_eqs
        leaves = [name(s) for s in states] + \
            [name(v) for v in fwd.fields] + [_exp._IDIFF]
        known = set(leaves) | set(name(lhs) for lhs, _ in equations)
        partials = []
        local = {}               # name -> [(referenced name, factor)]
        for lhs, rhs in equations:
            n = name(lhs)
            local[n] = []
            bcd = fwd.cubic.get(n)
            if bcd is not None:
                # A refined root x of x^3 + b x^2 + c x + d (see _generate)
                b, c, d = bcd
                g = w.fma(w.fma('2', b, f'3 * {n}'), n, c)
                r = f'r_{n}'
                one = '-1 / g_' if self.single else 'mkg_div(-1.0, g_)'
                partials.append(f'{tab}Real {r};')
                partials.append(f'{tab}{{ const Real g_ = {g}; {r} = '
                                f'g_ != 0 ? {one} : (Real)0; }}')
                for x, p in ((b, f'{r} * {n} * {n}'), (c, f'{r} * {n}'),
                             (d, r)):
                    if x in known:
                        local[n].append((x, f'({p})'))
                continue
            for r in _references(rhs):
                rn = name(r)
                if rn not in known:
                    continue
                dp = local_partial(rhs, r)
                if dp is None:
                    continue
                if isinstance(dp, _N):
                    local[n].append((rn, float(dp.eval())))
                    continue
                if isinstance(dp, myokit.PrefixMinus) and \
                        isinstance(dp[0], _N):
                    local[n].append((rn, -float(dp[0].eval())))
                    continue
                p = f'p_{len(partials)}'
                partials.append(f'{tab}const Real {p} = {w.ex(dp)};')
                local[n].append((rn, p))

        def ref(var):
            x = fwd.literal_subst.get(myokit.Name(var))
            return w.ex(x) if x is not None else name(var)

        rows = []
        entries = {}             # column -> [(state, slot)]
        slots = 0
        order = [name(lhs) for lhs, _ in equations]
        for i, s in enumerate(states):
            acc = {}

            def add(rn, a, p=1.0):
                if isinstance(p, float) and abs(p) != 1.0:
                    p = f'(Real){p!r}'
                if isinstance(p, float):
                    a = a if p > 0 else f'-{a}'
                    if rn in acc:
                        rows.append(f'{tab}    {acc[rn]} += {a};')
                        return
                elif rn in acc:
                    rows.append(f'{tab}    {acc[rn]} = '
                                f'{w.fma(a, p, acc[rn])};')
                    return
                else:
                    a = f'{a} * {p}'
                acc[rn] = 'J_' + rn
                rows.append(f'{tab}    Real J_{rn} = {a};')

            rows.append(f'{tab}{{')
            n = name(s)
            if s in fwd.rl_states:
                inf, tau = fwd.rl_states[s]
                ri, rt = ref(inf), ref(tau)
                rows.append(f'{tab}    const Real E_ = '
                            f'{fwd.decay(tau, rt, fwd.rates)};')
                add(n, 'E_')
                if name(inf) in known and \
                        myokit.Name(inf) not in fwd.literal_subst:
                    add(name(inf), '(1 - E_)')
                if name(tau) in known and \
                        myokit.Name(tau) not in fwd.literal_subst:
                    num = f'-({ri} - {n}) * E_ * dt_'
                    den = f'{rt} * {rt}'
                    q = f'{num} / ({den})' if self.single else \
                        f'mkg_div({num}, {den})'
                    add(name(tau), q)
            else:
                add(name(s.lhs()), 'dt_')
            for x in reversed(order):
                if x in acc:
                    for rn, p in local[x]:
                        add(rn, acc[x], p)
            for x in leaves:
                if x in acc:
                    rows.append(f'{tab}    tape[{slots} * 32] = {acc[x]};')
                    entries.setdefault(x, []).append((i, slots))
                    slots += 1
            rows.append(f'{tab}}}')
        return partials, rows, entries, slots

    def _generate_map(self, tiles_per_sm):
        """
        The tape and sweep kernels (``csrc/adjoint_map.cu.in``) for a
        resident simulation with that many tiles on an SM, or None where
        the sweep's tiles would not fit.
        """
        fwd = self.fwd
        w = fwd.writer
        name = fwd._name
        tab = '    '
        states = fwd.states
        vm = fwd.i_vm
        if not fwd.team or vm < 0:
            return None
        partials, rows, entries, x0 = self._step_matrix(tab)
        diff = fwd.diffusion
        extra = {_exp.DIFF_NONE: 0, _exp.DIFF_GRID: 2 if fwd.two_d
                 else 1, _exp.DIFF_HETERO: 4 if fwd.two_d else 2,
                 _exp.DIFF_CONN: 5}[diff]
        self.slots = x0 + extra

        cols = [(name(s), j, None) for j, s in enumerate(states)]
        cols += [(name(v), None, k) for k, v in enumerate(fwd.fields)]
        current = entries.get(_exp._IDIFF, []) if diff else []

        def price(c):
            return 2 + 2 * len(entries.get(c[0], ()))
        words = 1 if self.single else 2
        shared = (2 * len(states) + 2) * 32 * 4 * words + 32
        for parts in (4, 2) if self.single else (8, 4, 2):
            # Columns to warps: V's, which the next step waits for, to the
            # first, the conductances' gradients to the last
            load = [0.0] * parts
            mine = [[] for _ in range(parts)]
            load[0] += 10 + 2 * len(current) + price(cols[vm])
            mine[0].append(cols[vm])
            load[-1] += 2 * extra
            for c in sorted((c for c in cols if c[1] != vm),
                            key=lambda c: (-price(c), c[0])):
                p = min(range(parts), key=load.__getitem__)
                mine[p].append(c)
                load[p] += price(c)
            # Registers of a thread: the numbers of two steps, and some
            held = [[t for c in mine[p] for _, t in entries.get(c[0], ())] +
                    ([t for _, t in current] if p == 0 else []) +
                    (list(range(x0, x0 + extra)) if p == parts - 1 else [])
                    for p in range(parts)]
            need = words * (2 * max(len(h) for h in held) + 16) + 40
            if need <= 255 and 32 * parts * tiles_per_sm * need <= 65536 \
                    and tiles_per_sm * (shared + 1024) <= 227 * 1024:
                break
        else:
            return None
        # (rows of the current besides V's wait for the other warps)
        meet_twice = any(i != vm for i, _ in current)
        self.parts = parts

        def step(p, cur, nxt, a):
            out = []
            o = lambda x: out.append(f'{tab * 3}{x}')  # noqa: E731
            o('if (s + 1 < n) tape -= back;')
            for q, t in enumerate(held[p]):
                o(f'{nxt}{q} = __ldcg(tape + {t} * 32);')
            at = {t: f'{cur}{q}' for q, t in enumerate(held[p])}
            if p == 0:
                # (a log row is known two steps ahead, its gradient one)
                o('const Real loss_ = next_;')
                o('next_ = row_ >= 0 && col_ >= 0 ? lgrad[(long long)row_ *'
                  ' b.nprobe + col_] : (Real)0;')
                o('row_ = s + 2 < n ? a.steps[n - 3 - s].log_row : -1;')
                lv = f'ls[{a}][{vm}][lane]'
                if diff:
                    o('MKG_GATHER(mu_)')
                    o(f'const Real l{vm}_ = {lv} + gather;')
                    o(f'{lv} = l{vm}_;')
                    o('mu_ = 0;')
                    for i, t in current:
                        x = f'l{vm}_' if i == vm else f'ls[{a}][{i}][lane]'
                        o(f'mu_ = {w.fma(x, at[t], "mu_")};')
                    o('MKG_PUBLISH(mu_)')
                    o(f'ms[{a}][lane] = mu_;')
                else:
                    o(f'const Real l{vm}_ = {lv};')
            o('mkg_parts_sync();')
            o(f'if (s_stop[{a}]) break;')
            rows_needed = sorted(set(
                i for c in mine[p] for i, _ in entries.get(c[0], ())) | set(
                c[1] for c in mine[p] if c[1] is not None and
                states[c[1]] not in fwd.rl_states))
            for i in rows_needed:
                if p or i != vm:
                    o(f'const Real l{i}_ = ls[{a}][{i}][lane];')
            for c, j, k in mine[p]:
                # The entries' sum first: added one by one to a forward Euler
                # state's lambda, each would round that. (Error of a field's
                # gradient against 64 bits, 96 x 52 cells, 48 states, 100
                # steps: general kernel 9.9e-7, one by one 1.7e-6, so 1.3e-6;
                # five sizes on average 1.19e-6, 1.29e-6, 1.14e-6.)
                own = j is not None and states[j] not in fwd.rl_states
                o('{ Real a_ = 0, b_ = 0;')
                for q, (i, t) in enumerate(entries.get(c, ())):
                    x = 'ab'[q & 1] + '_'
                    o(f'  {x} = {w.fma(f"l{i}_", at[t], x)};')
                o('  a_ += b_;')
                if j == vm:
                    o('  a_ += loss_;')
                    if diff:
                        o('  a_ += mu_ * cdiag;')
                if own:
                    o(f'  a_ = l{j}_ + a_;')
                if j is None:
                    o(f'  f{k}_ += a_; }}')
                else:
                    o(f'  ls[{1 - a}][{j}][lane] = a_; }}')
            if p == parts - 1 and diff:
                x = [at[x0 + q] for q in range(extra)]
                o(f'const Real mu_ = ms[{a}][lane];')
                if diff == _exp.DIFF_GRID:
                    o(f'gx_ += mu_ * {x[0]};')
                    if fwd.two_d:
                        o(f'gy_ += mu_ * {x[1]};')
                elif diff == _exp.DIFF_HETERO:
                    o(f'gx_ += mu_ * ({x[0]} + {x[1]});')
                    if fwd.two_d:
                        o(f'gy_ += mu_ * ({x[2]} + {x[3]});')
                    for q in range(extra):
                        o(f'e{q}_ += (double)mu_ * (double){x[q]};')
                else:
                    o(f'gx_ += mu_ * {x[4]};')
                    for q in range(4):
                        o(f'e{q}_ += (double)mu_ * (double){x[q]};')
                    o('if (p0_ + 4 < p1_) {')
                    o('  const Real *vk = (const Real *)b.traj + (long long)'
                      f'((n - 1 - s) * N_STATE + {vm}) * pitch;')
                    o('  const Real V = vk[cid];')
                    o('  for (int p = p0_ + 4; p < p1_; ++p)')
                    o('    b.ge[p] += (double)mu_ * (double)(V -'
                      ' vk[a.nbr_idx[p]]);')
                    o('}')
            if meet_twice:
                o('mkg_parts_sync();')
            return out

        body = []
        for p in range(parts):
            o = lambda x: body.append(tab + x)  # noqa: E731
            o(f'{"if" if p == 0 else "else if"} (part_ == {p}) {{')
            m = len(held[p])
            for q, t in enumerate(held[p]):
                o(f'    Real c{q} = __ldcg(tape + {t} * 32), n{q} = 0;')
            for _, j, k in mine[p]:
                if j is None:
                    o(f'    Real f{k}_ = ((const Real *)b.gfield)'
                      f'[(long long){k} * pitch + cid];')
            last = p == parts - 1 and diff
            edges = 0
            if p == 0:
                o('    const Real *lgrad = (const Real *)b.lgrad;')
                o('    const int col_ = live ? b.probe_col[cid] : -1;')
                o('    int row_ = a.steps[n - 1].log_row;')
                o('    Real next_ = row_ >= 0 && col_ >= 0 ? lgrad['
                  '(long long)row_ * b.nprobe + col_] : (Real)0;')
                o('    row_ = n > 1 ? a.steps[n - 2].log_row : -1;')
                if diff:
                    o('    Real mu_ = ms[1][lane];')
            if last:
                o('    Real gx_ = ((const Real *)b.gg)[cid];')
                o('    Real gy_ = ((const Real *)b.gg)[pitch + cid];')
                edges = {_exp.DIFF_GRID: 0, _exp.DIFF_CONN: 4}.get(
                    diff, extra)
                where = [f'live ? b.ge[{q} * pitch + cid] : 0'
                         for q in range(edges)]
                if diff == _exp.DIFF_CONN:
                    where = [f'p0_ + {q} < p1_ ? b.ge[p0_ + {q}] : 0'
                             for q in range(4)]
                for q in range(edges):
                    o(f'    double e{q}_ = {where[q]};')
            o('    for (int s = 0; s < n; ) {')
            body.extend(step(p, 'c', 'n', 0))
            o('        if (++s == n) break;')
            o('        {')
            body.extend(step(p, 'n', 'c', 1))
            o('        }')
            o('        ++s;')
            o('    }')
            for _, j, k in mine[p]:
                if j is None:
                    o(f'    if (live) ((Real *)b.gfield)[(long long){k} *'
                      f' pitch + cid] = f{k}_;')
            if last:
                o('    if (live) {')
                o('        ((Real *)b.gg)[cid] = gx_;')
                o('        ((Real *)b.gg)[pitch + cid] = gy_;')
                for q in range(edges):
                    if diff == _exp.DIFF_CONN:
                        o(f'        if (p0_ + {q} < p1_) b.ge[p0_ + {q}] ='
                          f' e{q}_;')
                    else:
                        o(f'        b.ge[{q} * pitch + cid] = e{q}_;')
                o('    }')
            o('}')
        subs = {
            '@NSLOT@': str(self.slots),
            '@PARTS@': str(parts),
            '@X0@': str(x0),
            '@MINB_ADJ@': str(tiles_per_sm),
            '@FORWARD@': '\n'.join(self._forward_values(tab)),
            '@PARTIALS@': '\n'.join(partials),
            '@ROWS@': '\n'.join(rows),
            '@SWEEP@': '\n'.join(body),
        }
        text = _exp._read('adjoint_map.cu.in')
        for k, v in subs.items():
            text = text.replace(k, v)
        return self.fwd.source() + '\n' + text

    @staticmethod
    def _join(fsrc, text):
        """Appends the adjoint kernel (the template from its declaration
        on) to the forward module, which defines what it uses."""
        start = text.index('extern "C" __global__')
        return fsrc + '\n' + text[start:]

    def source(self):
        return self._source

    def options(self):
        return self.fwd.options()

    def key(self):
        if self._key is None:
            import hashlib
            h = hashlib.sha256()
            h.update(self._source.encode())
            h.update('\0'.join(self.options()).encode())
            self._key = h.hexdigest()
        return self._key


class TissueAdjoint(object):
    """
    Forward runs and loss gradients for a :class:`SimulationCUDA`.

    ``sim``
        A simulation in any diffusion mode: homogeneous conductances gx, gy,
        per-edge conductances (``set_conductance_field``), connections
        (``set_connections``) or none. Its fields and its conductances are
        the parameters the gradients refer to. With an accumulation mode the
        forward
        runs (and is recomputed) exactly as the simulation's own, FP64 or
        compensated states included; the reverse sweep is in the
        simulation precision and takes the rounding of those states to it
        as the identity.
    ``probes``
        Cells whose V enters the loss: integers (1D) or ``(x, y)`` (2D).
    ``segment_steps``
        Steps between checkpoints: the backward pass recomputes each segment
        from its checkpoint, so memory is one segment's trajectory plus one
        state per segment.
    ``min_blocks``, ``threads``
        Resident CTAs per SM asked of the compiler for the reverse kernel,
        and its CTA size (default: the simulation's); the register cap is
        64K / (threads * min_blocks).
    ``guards``
        Skip the reverse of equations whose adjoint is still zero (one
        branch per equation). The default, straight-line code, lets the
        compiler schedule across equations and keeps the reverse kernel
        free of register spills; results are the same while the partial
        derivatives are finite.

    The simulation's state and time are not changed by :meth:`forward`.
    """
    def __init__(self, sim, probes, segment_steps=200, min_blocks=1,
                 threads=None, guards=False):
        self.sim = sim
        self.segment_steps = int(segment_steps)
        self.min_blocks = int(min_blocks)
        self.threads = threads
        self.guards = bool(guards)
        self._generated = {}
        vm = sim._vm
        if vm is None:
            raise ValueError('The adjoint needs a membrane potential.')
        self.cells = []
        for p in probes:
            if len(sim._dims) == 2:
                x, y = int(p[0]), int(p[1])
                if not (0 <= x < sim._nx and 0 <= y < sim._ny):
                    raise IndexError('Probe out of range: ' + str(p))
                self.cells.append(x + y * sim._nx)
            else:
                x = int(p)
                if not 0 <= x < sim._nx:
                    raise IndexError('Probe out of range: ' + str(p))
                self.cells.append(x)
        if len(set(self.cells)) != len(self.cells):
            raise ValueError('Duplicate probe cells.')
        self._attached = None
        self.rows = 0

    def field_names(self):
        """Qualified names of the fields, in gradient order."""
        return [v.qname() for v in self.sim._fields]

    def _prepare(self):
        from .simulation import compile_kernel, shared_kernel
        sim = self.sim
        kernel = sim._kernel([])
        be = sim._get_backend(kernel)
        # Generated once per forward kernel (the forward kernel's key covers
        # the model version, precision, fields and launch shape) and CTA size
        akey = (kernel.key(), self.min_blocks, self._threads(kernel),
                self.guards, self._tiles_per_sm(kernel))
        ak = self._generated.get(akey)
        if ak is None:
            ak = shared_kernel(
                ('adjoint', sim.model_code(), sim._rl) + akey,
                lambda: self._make(kernel, akey[-1]))
            self._generated = {akey: ak}
        key = (id(be), akey, self.segment_steps)
        if self._attached != key:
            cubin = compile_kernel(ak)
            if ak.parts:
                be.check(be.lib.mkg_adj_attach_map(
                    be.h, cubin, len(cubin), self.segment_steps, ak.slots,
                    ak.parts))
            else:
                be.check(be.lib.mkg_adj_attach(be.h, cubin, len(cubin),
                                               self.segment_steps))
            self._attached = key
        return be

    def _tiles_per_sm(self, kernel):
        """
        Tiles on an SM where the reverse of a resident simulation goes by
        tape and sweep (:meth:`AdjointKernel._generate_map`), 0 where the
        general reverse kernel runs: with launch options of its own, and on
        grids that fill the SMs with it.
        """
        sim = self.sim
        if not kernel.team or sim._team is not None or self.guards or \
                self.threads is not None or self.min_blocks != 1:
            return 0
        nx, ny = (sim._nx, sim._ny) if kernel.two_d else (sim._ntotal, 1)
        n = -(-(-(-nx // 32) * ny) // autotune._sm_count(sim._device))
        return n if n <= _MAP_TILES else 0

    def _threads(self, kernel):
        """The CTA size of the general reverse kernel."""
        if self.threads is not None:
            return self.threads
        if kernel.team:
            # A resident kernel's CTA is one tile; the reverse kernel's
            # warps each own tiles: as many warps as there are tiles for an
            # SM
            return 32 * min(kernel.min_blocks, 8)
        if self.sim._block is None:
            # The reverse kernel wants the registers of 256 threads (800 x
            # 800 cells, 48 states, 20 steps: 52.1 ms, with 512 53.3)
            return min(kernel.block[0], 256)
        return None

    def _make(self, kernel, tiles_per_sm):
        """The adjoint kernel of a forward kernel."""
        sim = self.sim
        # The trajectory-writing forward kernel has the launch shape,
        # register cap and tile staging of the simulation's own kernel
        fwd = _exp.TissueKernel(
            sim._model, sim._precision, sim._native_math,
            sim._bound_variables, [], kernel.diffusion, kernel.two_d,
            list(sim._fields.keys()), sim._rl_states, kernel.block,
            min_blocks=kernel.min_blocks, math=sim._fp32_math,
            accumulate=kernel.accumulate,
            accumulate_states=sim.accumulated_states(), traj=True,
            stage=kernel.stage, row_pad=kernel.row_pad,
            stage_lazy=kernel.stage_lazy, sync=kernel.sync,
            team=kernel.team, many=kernel.many)
        if tiles_per_sm:
            ak = AdjointKernel(fwd, tiles_per_sm=tiles_per_sm)
            if ak.parts:
                return ak
        return AdjointKernel(fwd, self.min_blocks, self._threads(kernel),
                             self.guards)

    def forward(self, duration, log_interval=1.0):
        """
        Runs ``duration`` time units from the simulation's state and time,
        and returns the probes' V as an array (log points x probes).
        """
        sim = self.sim
        be = self._prepare()
        lib, h = be.lib, be.h
        saved = (sim._state.copy(), sim._time)
        sim._upload(be)
        items = np.full(len(self.cells), sim._vm.index(), dtype=np.int32)
        cells = np.ascontiguousarray(self.cells, dtype=np.int64)
        be.log_sig = None
        be.check(lib.mkg_set_log(h, _lib.i32ptr(items), _lib.i64ptr(cells),
                                 len(cells), 0))
        be.check(lib.mkg_set_tuning(h, 0, 0, 0))
        rows = _lib.ctypes.c_int64()
        be.check(lib.mkg_adj_forward(
            h, sim._time, sim._time + duration, sim._step_size,
            float(log_interval), _lib.ctypes.byref(rows)))
        self.rows = rows.value
        out = np.empty((self.rows, len(self.cells)))
        be.check(lib.mkg_adj_read_log(h, _lib.dptr(out), self.rows))
        sim._state, sim._time = saved
        return out

    def backward(self, dl_dv):
        """
        Gradients for ``dl_dv = dL/dV`` at the logged points (the array
        returned by :meth:`forward`). Returns ``{field qname: gradient with
        the field's shape, 'gx': ..., 'gy': ...}`` where, by diffusion mode,

        - homogeneous conductances: ``gx`` and ``gy`` are floats;
        - per-edge conductances: ``gx`` has the shape of the simulation's
          gx field, ``(ny, nx - 1)`` in 2D or ``(nx - 1,)`` in 1D, and
          ``gy`` the shape ``(ny - 1, nx)`` (an empty array in 1D);
        - connections: ``'connections'`` holds one gradient per connection,
          in the order of the simulation's connection list, and ``gx`` is
          their sum (``gy`` is 0).
        """
        sim = self.sim
        be = self._prepare()
        g = np.ascontiguousarray(dl_dv, dtype=np.float64)
        if g.shape != (self.rows, len(self.cells)):
            raise ValueError('dl_dv must have shape %s' % (
                (self.rows, len(self.cells)),))
        nf = len(sim._fields)
        gf = np.zeros(max(nf, 1) * sim._ntotal)
        gg = np.zeros(2)
        be.check(be.lib.mkg_adj_backward(
            be.h, _lib.dptr(g), self.rows, _lib.dptr(gf), _lib.dptr(gg)))
        out = {}
        shape = (sim._ny, sim._nx) if len(sim._dims) == 2 else (sim._nx,)
        gf = gf[:nf * sim._ntotal].reshape(sim._ntotal, max(nf, 1))
        for k, name in enumerate(self.field_names()):
            out[name] = gf[:, k].reshape(shape)
        out['gx'] = float(gg[0])
        out['gy'] = float(gg[1])
        mode = sim._diffusion_mode()
        if mode in (_exp.DIFF_HETERO, _exp.DIFF_CONN):
            nx, ny = sim._nx, sim._ny
            two_d = len(sim._dims) == 2
            if mode == _exp.DIFF_HETERO:
                n = ny * (nx - 1) + ((ny - 1) * nx if two_d else 0)
            else:
                n = len(sim._connections)
            ge = np.zeros(max(n, 1))
            be.check(be.lib.mkg_adj_conductance_gradient(
                be.h, _lib.dptr(ge), n))
            if mode == _exp.DIFF_CONN:
                out['connections'] = ge[:n]
            elif two_d:
                out['gx'] = ge[:ny * (nx - 1)].reshape(ny, nx - 1)
                out['gy'] = ge[ny * (nx - 1):n].reshape(ny - 1, nx)
            else:
                out['gx'] = ge[:n]
                out['gy'] = np.zeros(0)
        return out

    def loss_and_gradient(self, duration, target, log_interval=1.0):
        """Sum of squared V errors against ``target`` and its gradients."""
        v = self.forward(duration, log_interval)
        d = v - np.asarray(target, dtype=float)
        return float(np.sum(d * d)), self.backward(2 * d)


def _make_function():
    import torch

    class TissueLossFunction(torch.autograd.Function):
        """
        ``loss = TissueLossFunction.apply(adjoint, duration, log_interval,
        target, g, *fields)``: the sum of squared V errors at the probes of
        a :class:`TissueAdjoint`, as a function of the scalar fields (tensors
        shaped like the grid, in ``adjoint.field_names()`` order) and of the
        diffusion conductances ``g``:

        - homogeneous conductances: a scalar tensor (gx = gy = g in 2D) or a
          two-element tensor (gx, gy);
        - per-edge conductances: one tensor of the gx field's values
          followed, in 2D, by the gy field's (the layout of
          ``set_conductance_field``, flattened);
        - connections: one tensor of per-connection conductances, in the
          order of the simulation's connection list.

        Gradients come from the discrete adjoint.
        """
        @staticmethod
        def forward(ctx, adj, duration, log_interval, target, g, *fields):
            sim = adj.sim
            for name, f in zip(adj.field_names(), fields):
                sim.set_field(name, f.detach().cpu().double().numpy())
            gv = g.detach().cpu().double().reshape(-1).numpy()
            mode = sim._diffusion_mode()
            ctx.mode = mode
            if mode == _exp.DIFF_HETERO:
                nx, ny = sim._nx, sim._ny
                n = ny * (nx - 1)
                if len(sim._dims) == 2:
                    sim.set_conductance_field(
                        gv[:n].reshape(ny, nx - 1), gv[n:].reshape(ny - 1, nx))
                else:
                    sim.set_conductance_field(gv[:n])
            elif mode == _exp.DIFF_CONN:
                sim.set_connections([(i, j, float(x)) for (i, j, _), x in
                                     zip(sim._connections, gv)])
            elif sim._diffusion_enabled:
                gx = float(gv[0])
                gy = float(gv[1]) if len(gv) > 1 else gx
                sim.set_conductance(gx, gy)
            v = adj.forward(duration, log_interval)
            tgt = target.detach().cpu().double().numpy() \
                if hasattr(target, 'detach') else np.asarray(target)
            d = v - tgt
            ctx.adj = adj
            ctx.lgrad = 2 * d
            ctx.g_len = len(gv)
            ctx.g_dtype = g.dtype
            ctx.f_meta = [(f.dtype, f.device) for f in fields]
            return torch.tensor(float(np.sum(d * d)), dtype=torch.float64)

        @staticmethod
        def backward(ctx, grad_out):
            adj = ctx.adj
            grads = adj.backward(ctx.lgrad)
            s = float(grad_out)
            if ctx.mode == _exp.DIFF_HETERO:
                gg = torch.as_tensor(np.concatenate(
                    [np.ravel(grads['gx']), np.ravel(grads['gy'])]) * s,
                    dtype=ctx.g_dtype)
            elif ctx.mode == _exp.DIFF_CONN:
                gg = torch.as_tensor(grads['connections'] * s,
                                     dtype=ctx.g_dtype)
            elif ctx.g_len > 1:
                gg = torch.tensor([grads['gx'] * s, grads['gy'] * s],
                                  dtype=ctx.g_dtype)
            else:
                gg = torch.tensor((grads['gx'] + grads['gy']) * s,
                                  dtype=ctx.g_dtype)
            out = [None, None, None, None, gg]
            for name, (dt, dev) in zip(adj.field_names(), ctx.f_meta):
                out.append(torch.as_tensor(grads[name] * s, dtype=dt,
                                           device=dev))
            return tuple(out)

    return TissueLossFunction


_FUNCTION = None


def tissue_loss(adj, duration, target, g, fields, log_interval=1.0):
    """
    Differentiable loss (see ``TissueLossFunction``): returns a 0-d torch
    tensor whose ``backward()`` fills ``g.grad`` and the fields' ``.grad``.
    """
    global _FUNCTION
    if _FUNCTION is None:
        _FUNCTION = _make_function()
    return _FUNCTION.apply(adj, duration, log_interval, target, g, *fields)
