"""
Division of a model's equations among the warps of a team, for the resident
kernel (``csrc/resident_kernel.cu.in``).

A step has two or three phases, between which the team meets and values
change hands through shared memory:

1. where several equations need the same dear ones (buffered concentrations,
   reversal potentials), those, each once, and beside them what needs none;
2. the new values of the Rush-Larsen gates, and the variables that
   derivatives are made of;
3. the derivatives of the forward-Euler states, with the cheap sums between
   them and the handed-over variables.

Equations are never divided, and every warp evaluates them in the words of
the undivided kernel, so the division does not change a bit of the results.
"""
from ._deps import myokit

# Estimated time of an operation in an equation, relative to an addition.
# Single precision: instructions, with the latency of a chain in mind.
# Double precision: an addition waits 67 cycles for the double precision
# pipe; exp and division run on the integer pipes (csrc/mkg_math64.h).
_COST = {
    True: {'div': 3, 'exp': 3, 'log': 20, 'sqrt': 14, 'trig': 25, 'pow': 28,
           'cond': 1, 'rl': 6},
    False: {'div': 4, 'exp': 6, 'log': 7, 'sqrt': 5, 'trig': 22, 'pow': 14,
            'cond': 1, 'rl': 9},
}
# The refinement of a cubic root (single precision)
CUBIC = 55
# Intermediate variables this cheap are evaluated where they are used
# rather than handed over
_CHEAP = 1
_AGAIN = 2.0
_SHARE = 32
# What the diffusion current adds to the warp that updates V (in single
# precision; with V in double precision there; in double precision)
_HALO = {'single': 22, 'mixed': 240, 'double': 18}
# What the wait and the current add to it in a last phase
_LATER = 40
# A trip to L2, 880 cycles, and what an addition counts as
_TRIP = {True: 880 / 5, False: 880 / 67}


def cost(e, single):
    """Estimated time of an expression (see above)."""
    from . import exporter as _exp
    c = _COST[single]
    t = 0
    for x in e.walk():
        if isinstance(x, (myokit.Plus, myokit.Minus, myokit.Multiply,
                          myokit.PrefixMinus, myokit.Abs)):
            t += 1
        elif isinstance(x, myokit.Divide):
            t += 1 if single and isinstance(x[1], myokit.Number) else c['div']
        elif isinstance(x, (myokit.Quotient, myokit.Remainder, myokit.Floor,
                            myokit.Ceil)):
            t += 2 * c['div']
        elif isinstance(x, myokit.Exp):
            t += c['exp']
        elif isinstance(x, (myokit.Log, myokit.Log10)):
            t += c['log']
        elif isinstance(x, myokit.Sqrt):
            t += c['sqrt']
        elif isinstance(x, myokit.Cos) and not single and \
                _exp.third_of_acos(x[0]) is not None:
            # (one root of a cubic instead of both functions)
            t += 10 - c['trig'] - c['div']
        elif isinstance(x, (myokit.Sin, myokit.Cos, myokit.Tan, myokit.ASin,
                            myokit.ACos, myokit.ATan)):
            t += c['trig']
        elif isinstance(x, myokit.Power):
            p = x[1].eval() if isinstance(x[1], myokit.Number) else None
            if p is not None and p == int(p) and 2 <= p <= 16:
                t += int(p).bit_length()
            elif p in (0.5, 1.5):
                t += c['sqrt'] + 1
            else:
                t += c['pow']
        elif isinstance(x, (myokit.If, myokit.Piecewise, myokit.Condition)):
            t += c['cond']
    return t


class Team(object):
    """
    The share of each of ``n`` warps.

    ``items``: the equations in evaluation order, ``(name, referenced names,
    cost)``. ``gates``: per Rush-Larsen state, the names its update needs.
    ``derivatives``: per forward-Euler state, the name of its derivative.
    ``first``: the forward-Euler state whose derivative the first warp takes
    (V), or None. ``halo``: the name that needs the neighbours.

    ``work[f][w]`` are the names warp ``w`` evaluates in phase ``f``, in
    evaluation order, ``gates_of[f][w]`` the gates it updates there and
    ``tails_of[w]`` the states whose derivatives it completes in the last
    phase. Between phases the team meets; ``slots`` maps the names handed
    over to their slots, ``written[f][w]`` and ``read[f][w]`` list those a
    warp writes at the end and reads at the start of a phase. ``cost[f][w]``
    is the estimated time. ``exchange`` is what the diffusion current adds to
    the first warp, in the first phase (``halo_first``, if ``soon``) where
    there is time for it and a ``trip`` for the words, else in the last (``halo_late``: the
    first phase has time for the trip).
    """
    def __init__(self, n, items, gates, derivatives, first, halo, rl_cost,
                 exchange=0, trip=0, soon=True):
        self.n = n
        order = [name for name, _, _ in items]
        refs = {name: r for name, r, _ in items}
        price = {name: c for name, _, c in items}
        refs = {name: set(x for x in r if x in price)
                for name, r in refs.items()}
        needs_halo = {name for name, r, _ in items if halo in r}

        def closure(roots, stop=()):
            out, todo = set(), [x for x in roots if x in refs]
            while todo:
                x = todo.pop()
                if x in out or x in stop:
                    continue
                out.add(x)
                todo.extend(refs[x])
            return out

        def total(names):
            return sum(price[x] for x in names)

        roots = set(derivatives.values())
        by_gate = set().union(*gates.values()) if gates else set()
        needed = closure(roots | by_gate)
        users = {name: set() for name in refs}
        for name in needed:
            for r in refs[name]:
                users[r].add(name)
        for i, need in gates.items():
            for x in need:
                users[x].add(('gate', i))
        share = total(needed) / n
        # (a share of the work: what one warp can do in a phase)
        cap = max(1.25 * share, 60)
        self.work = []
        if n == 1:
            self.work = [[[x for x in order if x in needed]]]
            self.gates_of = [[sorted(gates)]]
            self.tails_of = [sorted(derivatives)]
            self.slots, self.written, self.read = {}, [[[]]], [[[]]]
            self.cost = [[total(needed)]]
            self.halo = [bool(needs_halo & needed)]
            self.halo_early = [False]
            self.halo_first = self.halo_late = False
            return

        # What several equations need and is dear enough to be computed once,
        # before the rest
        size = max([cap] + [price[x] + 20 for x in needed])
        shared = set()
        for x in order:
            if x in needed and x not in roots and len(users[x]) > 1 and \
                    not closure([x]) & needs_halo and \
                    _SHARE <= total(closure([x])) <= size:
                shared.add(x)

        # Last phase: derivatives, and what is cheap or too much for one
        # warp and leads to derivatives only
        tail = set()
        for x in reversed(order):
            if x not in needed or x in shared or not users[x] <= tail:
                continue
            if x in roots or (users[x] and (
                    price[x] <= _CHEAP or x in needs_halo or
                    total(closure([x], shared)) > cap)):
                tail.add(x)
        handed = set()
        for x in tail:
            handed |= refs[x] - tail
        handed |= roots - tail
        units = [(('gate', i), closure(need, shared), rl_cost)
                 for i, need in gates.items()]
        units += [(('value', x), closure([x], shared), 1)
                  for x in order if x in handed and x not in shared]

        groups = []          # per phase and warp: names evaluated
        self.cost = []
        self.gates_of = []

        def phase():
            groups.append([set() for _ in range(n)])
            self.cost.append([0.0] * n)
            self.gates_of.append([[] for _ in range(n)])

        def place(unit, names, own, bias, limit=None):
            f = len(groups) - 1
            best, least = None, None
            for w in range(n):
                new = names - groups[f][w]
                c = self.cost[f][w] + total(new) + own + bias[w]
                again = total(new & set().union(*groups[f]))
                if least is None or c + _AGAIN * again < least - 1e-9:
                    best, least = w, c + _AGAIN * again
            if limit is not None and least > limit:
                return False
            self.cost[f][best] += total(names - groups[f][best]) + own
            groups[f][best] |= names
            if unit[0] == 'gate':
                self.gates_of[f][best].append(unit[1])
            return True

        def largest_first(us):
            return sorted(us, key=lambda u: (-(total(u[1]) + u[2]),
                                             str(u[0])))
        none = [0.0] * n
        # The current is taken in the first phase, by a warp that has so much
        # less to do there, where the words are back before that phase ends
        opening = (total(closure(shared)) if shared else sum(
            total(u[1]) + u[2] for u in units)) / n
        self.halo_first = soon and first is not None and exchange > 0 and \
            opening > trip + exchange
        self.halo_late = not self.halo_first and opening > trip
        begin = exchange if self.halo_first else 0
        later = 0 if self.halo_first else _LATER
        if shared:
            phase()
            self.cost[0][0] += begin
            for u in largest_first([(('value', x), closure([x]), 1)
                                    for x in order if x in shared]):
                place(*u, none)
            # Meanwhile the other warps take what needs none of it
            limit = max(self.cost[0])
            rest = []
            for u in largest_first(units):
                free = not any(refs[x] & shared for x in u[1]) and not (
                    u[0][0] == 'gate' and gates[u[0][1]] & shared)
                if not free or not place(*u, none, limit=limit):
                    rest.append(u)
            # (what is there by now is read, unless it is cheap)
            there = set(x for g in groups[0] for x in g
                        if price[x] > _CHEAP)
            units = [(u, closure(gates[u[1]] if u[0] == 'gate' else [u[1]],
                                 there), own) for u, _, own in rest]
        # V's warp completes the longest sum: fewer units
        tails = {}
        for i, d in derivatives.items():
            own = closure([d], [x for x in refs if x not in tail])
            tails[i] = own
        phase()
        if not shared:
            self.cost[0][0] += begin
        bias = list(none)
        if first is not None:
            bias[0] = later
        for u in largest_first(units):
            place(*u, bias)
        if shared:
            for w in range(n):
                groups[1][w] -= groups[0][w]

        # Derivatives: V's to the first warp, others where they end soonest
        at = {}              # name -> (phase, warps that evaluate it)
        for f, g in enumerate(groups):
            for w in range(n):
                for x in g[w]:
                    at.setdefault(x, (f, set()))
                    if at[x][0] == f:
                        at[x][1].add(w)
        phase()
        last = len(groups) - 1
        self.tails_of = [[] for _ in range(n)]

        def inputs(i):
            out = set()
            for x in tails[i]:
                out |= refs[x] - tail
            return out | ({derivatives[i]} - tail)

        def spend(i, w):
            have = set(x for f in range(last) for x in groups[f][w])
            return (total(tails[i] - groups[last][w]) + 2 +
                    2 * len(inputs(i) - have))
        if first is not None:
            self.cost[last][0] += spend(first, 0) + later
            groups[last][0] |= tails[first]
            self.tails_of[0].append(first)
        for i in sorted((i for i in derivatives if i != first),
                        key=lambda i: (-total(tails[i]), i)):
            # In the last phase the first warp stores V and publishes its
            # word as soon as it has them, so where the current is taken
            # there no other warp may: it would read V of the next step, or
            # wait for words that a neighbour has overwritten meanwhile
            alone = first is not None and exchange > 0 and \
                not self.halo_first and tails[i] & needs_halo
            w = 0 if alone else min(range(n), key=lambda w: (
                self.cost[last][w] + spend(i, w), w))
            self.cost[last][w] += spend(i, w)
            groups[last][w] |= tails[i]
            self.tails_of[w].append(i)

        # Hand-overs: a warp reads what it has not evaluated itself
        self.work = [[[x for x in order if x in g] for g in gs]
                     for gs in groups]
        self.slots = {}
        self.written = [[[] for _ in range(n)] for _ in groups]
        self.read = [[[] for _ in range(n)] for _ in groups]
        for f in range(len(groups)):
            for w in range(n):
                need = set()
                for x in groups[f][w]:
                    need |= refs[x]
                for i in self.gates_of[f][w]:
                    need |= gates[i]
                if f == last:
                    for i in self.tails_of[w]:
                        need.add(derivatives[i])
                have = set(x for g in range(f + 1) for x in groups[g][w])
                have |= set(x for g in range(f) for x in self.read[g][w])
                for x in order:
                    if x in need and x not in have:
                        self.read[f][w].append(x)
                        if x not in self.slots:
                            self.slots[x] = len(self.slots)
                            g, ws = at[x]
                            self.written[g][min(ws)].append(x)
        self.halo = [any(x in needs_halo for gs in groups for x in gs[w])
                     for w in range(n)]
        self.halo_early = [any(x in needs_halo for gs in groups[:-1]
                               for x in gs[w]) for w in range(n)]
