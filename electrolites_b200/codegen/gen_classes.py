"""Code generator for the per-angular-momentum-class ERI + J/K kernels.

For every quartet class (li lj | lk ll) with li >= lj, lk >= ll and the bra
pair class >= the ket pair class (55 classes up to f), this writes one CUDA
translation unit under csrc/generated/ holding

  * a `Cls_<li><lj><lk><ll>` struct of straight-line device functions,
    templated on the arithmetic type T (double for the plain form, float for
    the single-precision quartets of the mixed form):
      - `root_acc`: one Rys root's 2D integrals G_d[e][f] (VRR on centres i
        and k, e <= li+lj, f <= lk+ll) and the accumulation of the
        (e0|f0) Cartesian integrals, all in registers (register form);
      - `row_acc`: the accumulation for one runtime e-component given its
        three rows of 2D integrals (team form, rows staged in shared memory);
      - `hrr_bra` / `hrr_ket`: the horizontal transfers (e0| -> (ij| and
        |f0) -> |kl), applied once per contracted quartet;
  * the instantiation of the kernel templates of csrc/jk_kernels.cuh for
    that class, and a host launcher registered in a table.

The arithmetic follows the reference's Rys formulation (roots t^2, c0x, cpx,
b00, b10, b01 recurrences: electrolites/codegen/gen_khigh.py:128-181) with
one structural change: the transfer to the j and l centres is applied after
the primitive and root sums (late HRR) instead of per root and primitive.

Form selection: the register form is used when the (e0|f0) block has at most
REG_MAX elements, in several passes over the primitives (a group of f
components each, PASS_MAX elements at most) for the REG_PASSES classes;
otherwise the team form spreads the e-components over the lanes of a team
(16 or 32*k threads) and splits the f-components over warps.
"""
from __future__ import annotations

import os
import sys
from dataclasses import dataclass

REG_MAX = 100         # largest (e0|f0) block kept in one thread's registers
# larger classes that take the register form in passes all the same: a
# quartet per lane, (e0|f0) accumulated for a group of f components per pass,
# its roots and 2D integrals recomputed per pass
# (ms on (H2O)_13 def2-TZVP UHF, team form -> passes: (dp|pp) 3.11 -> 2.06,
# (dd|ds) 1.21 -> 0.66, (fs|dp) 4.63 -> 1.87, (fp|ds) 4.26 -> 1.68, (fd|ps)
# 3.19 -> 1.33, (ff|ps) 2.20 -> 0.84; the next larger ones lose: (fp|pp)
# 2.29 -> 3.15, (dp|dp) 1.60 -> 1.84, (dd|pp) 0.78 -> 1.29, (fp|fs) 1.73 ->
# 2.37, (fs|dd) 0.58 -> 0.79).  Builds of few quartets run them in the team
# form (PASS_MIN_QUARTETS in csrc/jk_api.cu), so both are compiled.  The passes
# bound the accumulators; the whole bra-transferred and (ij|kl) blocks after them
# spill (3.5 KB of stores per thread in (fd|ps) to 6.7 in (ff|ps))
REG_PASSES = frozenset({'2111', '2220', '3021', '3120', '3210', '3310'})
# classes whose mixed builds run low-bound quartets in FP32 by default: those
# where it does not lose (FP32 in every class: (H2O)_96 6-31G* 246 ms, in none
# 212; (H2O)_20 def2-TZVP 54.2 / 44.6; a batch of 16 clusters of up to six in
# def2-TZVP 62.6 ms with FP32 in every f class, 53.7 with these)
FP32_DEFAULT = frozenset({'2020', '2222', '3222', '3320', '3321', '3322', '3330', '3331', '3332',
                          '3333'})
PASS_MAX = 80         # largest group of (e0|f0) elements of a pass
FPART_MAX = 40        # f-components per warp in the team form
LMAX = 3


def ncart(l):
    return (l + 1) * (l + 2) // 2


def comps(l):
    return [(lx, ly, l - lx - ly) for lx in range(l, -1, -1)
            for ly in range(l - lx, -1, -1)]


def cidx(l, c):
    lx, ly, lz = c
    return (l - lx) * (l - lx + 1) // 2 + lz


@dataclass
class Cls:
    li: int
    lj: int
    lk: int
    ll: int

    @property
    def tag(self):
        return f'{self.li}{self.lj}{self.lk}{self.ll}'

    @property
    def lij(self):
        return self.li + self.lj

    @property
    def lkl(self):
        return self.lk + self.ll

    @property
    def nroots(self):
        return (self.lij + self.lkl) // 2 + 1

    def eset(self):
        return [(L, c) for L in range(self.li, self.lij + 1) for c in comps(L)]

    def fset(self):
        return [(L, c) for L in range(self.lk, self.lkl + 1) for c in comps(L)]

    @property
    def ne(self):
        return len(self.eset())

    @property
    def nf(self):
        return len(self.fset())

    @property
    def form(self):
        return 'reg' if self.ne * self.nf <= REG_MAX or self.tag in REG_PASSES else 'team'

    def passes(self):
        """f ranges of the register form's passes."""
        if self.ne * self.nf <= REG_MAX:
            return [(0, self.nf)]
        per = max(1, PASS_MAX // self.ne)
        n = (self.nf + per - 1) // per
        return [(p * self.nf // n, (p + 1) * self.nf // n) for p in range(n)]

    # team form geometry
    @property
    def team_lanes(self):          # lanes holding e-components
        return 16 if self.ne <= 16 else 32 * ((self.ne + 31) // 32)

    @property
    def nwf(self):                 # warps (or half-warp teams) over f
        return (self.nf + FPART_MAX - 1) // FPART_MAX

    @property
    def team_threads(self):
        return self.team_lanes * self.nwf

    def fparts(self):
        n = self.nwf
        size = (self.nf + n - 1) // n
        return [(p * size, min(self.nf, (p + 1) * size)) for p in range(n)]


def all_classes(lmax=LMAX):
    pairs = [(a, b) for a in range(lmax + 1) for b in range(a + 1)]
    out = []
    for A in range(len(pairs)):
        for B in range(A + 1):
            li, lj = pairs[A]
            lk, ll = pairs[B]
            out.append((A, B, Cls(li, lj, lk, ll)))
    return out


def pair_class_index(la, lb):
    return la * (la + 1) // 2 + lb


# ----------------------------------------------------------------------
# expression helpers
# ----------------------------------------------------------------------
class Emitter:
    def __init__(self, indent='        '):
        self.lines = []
        self.ind = indent

    def __call__(self, s):
        self.lines.append(self.ind + s)

    def text(self):
        return '\n'.join(self.lines)


def _mul(a, b):
    if a == '1':
        return b
    if b == '1':
        return a
    return f'{a} * {b}'


def _fma(coef, g, rest):
    """coef * g + rest, with g possibly the literal 1."""
    if g == '1':
        return f'({coef} + {rest})'
    return f'fma({coef}, {g}, {rest})'


def _scaled(n, name):
    return name if n == 1 else f'T({n}) * {name}'


def gen_vrr(em, cls, d, zero_one, lij=None, lkl=None):
    """Emit G_d[e][f] for e <= lij, f <= lkl (default: the class's); returns
    dict (e, f) -> expr.  zero_one: the value of G_d[0][0] ('1' for x and
    y, 'wz' for z)."""
    lij = cls.lij if lij is None else lij
    lkl = cls.lkl if lkl is None else lkl
    g = {(0, 0): zero_one}
    for e in range(lij):
        name = f'g{d}_{e + 1}_0'
        t = _mul(f'c0{d}', g[(e, 0)])
        if e > 0:
            t = _fma(_scaled(e, 'b10'), g[(e - 1, 0)], t)
        em(f'const T {name} = {t};')
        g[(e + 1, 0)] = name
    for f in range(lkl):
        for e in range(lij + 1):
            name = f'g{d}_{e}_{f + 1}'
            expr = _mul(f'cp{d}', g[(e, f)])
            if f > 0:
                expr = _fma(_scaled(f, 'b01'), g[(e, f - 1)], expr)
            if e > 0:
                expr = _fma(_scaled(e, 'b00'), g[(e - 1, f)], expr)
            em(f'const T {name} = {expr};')
            g[(e, f + 1)] = name
    return g


def gen_root_acc(cls, f0, f1):
    """acc[e * (f1 - f0) + f - f0] += Gx Gy Gz of one root for f in [f0, f1)."""
    em = Emitter('    ')
    gx = gen_vrr(em, cls, 'x', '1')
    gy = gen_vrr(em, cls, 'y', '1')
    gz = gen_vrr(em, cls, 'z', 'wz')
    E, F = cls.eset(), cls.fset()[f0:f1]
    # products of x and y factors, shared between accumulators
    uses = {}
    for (_, ec) in E:
        for (_, fc) in F:
            key = (ec[0], fc[0], ec[1], fc[1])
            uses[key] = uses.get(key, 0) + 1
    named = {}
    nf = len(F)
    for ie, (_, ec) in enumerate(E):
        for jf, (_, fc) in enumerate(F):
            a = gx[(ec[0], fc[0])]
            b = gy[(ec[1], fc[1])]
            c = gz[(ec[2], fc[2])]
            key = (ec[0], fc[0], ec[1], fc[1])
            if a == '1' and b == '1':
                xy = None
            elif a == '1':
                xy = b
            elif b == '1':
                xy = a
            elif uses[key] > 1:
                if key not in named:
                    nm = f'xy_{key[0]}{key[1]}{key[2]}{key[3]}'
                    em(f'const T {nm} = {a} * {b};')
                    named[key] = nm
                xy = named[key]
            else:
                xy = f'({a} * {b})'
            k = ie * nf + jf
            if xy is None:
                em(f'acc[{k}] += {c};')
            else:
                em(f'acc[{k}] = fma({xy}, {c}, acc[{k}]);')
    return em.text()


def gen_boys_acc(cls):
    """The (e0|f0) block of a one- or two-root class from its Boys functions
    F[m] (prefactor included) by the vertical recursion of Obara and Saika in
    the form of Head-Gordon and Pople (auxiliary index m):
      [e+1_i|f]^m = PA_i [e|f]^m + WP_i [e|f]^(m+1)
                    + e_i hp ([e-1_i|f]^m - sp [e-1_i|f]^(m+1)) + f_i hs [e|f-1_i]^(m+1)
    and [e|f+1_i]^m = QC_i [e|f]^m + WQ_i [e|f]^(m+1) + e_i hs [e-1_i|f]^(m+1) for the f
    up to p of these classes; hp = 1/(2 a_ij), hs = 1/(2 (a_ij + a_kl)),
    sp = a_kl/(a_ij + a_kl)."""
    em = Emitter('    ')
    memo = {}

    def low(v, i):
        w = list(v)
        w[i] -= 1
        return tuple(w)

    def name(e, f, m):
        return 'b' + ''.join(map(str, e)) + '_' + ''.join(map(str, f)) + f'_{m}'

    def temp(nm, expr):
        if nm not in memo:
            memo[nm] = nm
            em(f'const double {nm} = {expr()};')
        return nm

    def terms(e, f, m):
        """[(coefficient or None, value), ...] summing to [e|f]^m."""
        if any(f):
            i = next(d for d in range(3) if f[d])
            g = low(f, i)
            out = [(f'QC{"xyz"[i]}', val(e, g, m)), (f'WQ{"xyz"[i]}', val(e, g, m + 1))]
            if e[i]:
                el = low(e, i)
                v = val(el, g, m + 1)
                s = temp(f'hs_{name(el, g, m + 1)}', lambda: f'hs * {v}')
                out += [(None, s)] if e[i] == 1 else [(f'{e[i]}.0', s)]
            return out
        i = next(d for d in range(3) if e[d])
        el = low(e, i)
        out = [(f'PA{"xyz"[i]}', val(el, f, m)), (f'WP{"xyz"[i]}', val(el, f, m + 1))]
        if el[i]:
            e2 = low(el, i)
            a, b = val(e2, f, m), val(e2, f, m + 1)
            s = temp(f'hp_{name(e2, f, m)}', lambda: f'hp * fma(-sp, {b}, {a})')
            out += [(None, s)] if el[i] == 1 else [(f'{el[i]}.0', s)]
        return out

    def val(e, f, m):
        if not any(e) and not any(f):
            return f'F[{m}]'
        nm = name(e, f, m)
        if nm not in memo:
            ts = terms(e, f, m)
            expr = None
            for c, v in reversed(ts):
                if expr is None:
                    expr = v if c is None else f'{c} * {v}'
                else:
                    expr = f'{v} + {expr}' if c is None else f'fma({c}, {v}, {expr})'
            temp(nm, lambda: expr)
        return nm

    E, F = cls.eset(), cls.fset()
    nf = len(F)
    # values another one needs are temporaries; the rest go straight into acc
    inner = {(ec, fc) for _, ec in E for _, fc in F
             if not any(fc) and any(tuple(x + (d == i) for i, x in enumerate(ec)) in [c for _, c in E]
                    for d in range(3))}
    for ie, (_, ec) in enumerate(E):
        for jf, (_, fc) in enumerate(F):
            k = ie * nf + jf
            if (ec, fc) in inner or not (any(ec) or any(fc)):
                em(f'acc[{k}] += {val(ec, fc, 0)};')
                continue
            expr = f'acc[{k}]'
            for c, v in terms(ec, fc, 0):
                expr = f'({expr} + {v})' if c is None else f'fma({c}, {v}, {expr})'
            em(f'acc[{k}] = {expr};')
    return em.text()


def gen_row_acc(cls, f0, f1):
    """acc[f - f0] += gx[fx] * gy[fy] * gz[fz] for f in [f0, f1)."""
    em = Emitter('    ')
    F = cls.fset()
    for jf in range(f0, f1):
        _, fc = F[jf]
        em(f'acc[{jf - f0}] = fma(gx[{fc[0]}] * gy[{fc[1]}], gz[{fc[2]}], acc[{jf - f0}]);')
    return em.text()


def gen_hrr(la, lb, prefix, vec):
    """(a, b) from levels la..la+lb of the input: out[(a*nb + b) * SO] for a
    at level la, b at level lb.  in[k * SI] is ordered level by level (SI, SO:
    strides, 1 for register arrays, NF for a column of a shared-memory block)."""
    em = Emitter('    ')
    off = {}
    o = 0
    for L in range(la, la + lb + 1):
        off[L] = o
        o += ncart(L)
    memo = {}

    def val(L, a, k, b):
        """value of the (a at level L | b at level k) intermediate."""
        key = (L, a, k, b)
        if key in memo:
            return memo[key]
        if k == 0:
            expr = f'in[{off[L] + cidx(L, a)} * SI]'
            memo[key] = expr
            return expr
        # recurse on the first nonzero direction of b
        d = 0 if b[0] > 0 else (1 if b[1] > 0 else 2)
        bm = list(b)
        bm[d] -= 1
        bm = tuple(bm)
        ap = list(a)
        ap[d] += 1
        ap = tuple(ap)
        t1 = val(L + 1, ap, k - 1, bm)
        t2 = val(L, a, k - 1, bm)
        name = f'{prefix}{k}_{L}_{cidx(L, a)}_{cidx(k, b)}'
        em(f'const T {name} = fma({vec}{"xyz"[d]}, {t2}, {t1});')
        memo[key] = name
        return name

    nb = ncart(lb)
    outs = []
    for ia, a in enumerate(comps(la)):
        for ib, b in enumerate(comps(lb)):
            outs.append(f'out[{ia * nb + ib} * SO] = {val(la, a, lb, b)};')
    for s in outs:
        em(s)
    return em.text()


# ----------------------------------------------------------------------
# nuclear gradient: blocks of the (e|f) space accumulated per quartet
# ----------------------------------------------------------------------
def grad_rects(cls):
    """The four (e|f)-space blocks of the gradient kernel, (name, e-levels,
    f-levels, weight): U unweighted (the lowered shells' transfers read it),
    RA / RB / RC weighted by 2 alpha of the primitive of shell i / j / k
    (the raised shells').  d/dA_x g_a = 2 alpha g_{a+1x} - a_x g_{a-1x}."""
    li, lj, lk, ll = cls.li, cls.lj, cls.lk, cls.ll
    lij, lkl = cls.lij, cls.lkl
    return [('U', (max(li - 1, 0), lij), (max(lk - 1, 0), lkl), None),
            ('RA', (li + 1, lij + 1), (lk, lkl), 'wA'),
            ('RB', (li, lij + 1), (lk, lkl), 'wB'),
            ('RC', (li, lij), (lk + 1, lkl + 1), 'wC')]


def _level_set(l0, l1):
    return [(L, c) for L in range(l0, l1 + 1) for c in comps(L)]


def grad_passes(ne, nf):
    """f ranges of a block's passes in the split classes."""
    n = (nf + max(1, GRAD_PASS_MAX // ne) - 1) // max(1, GRAD_PASS_MAX // ne)
    return [(p * nf // n, (p + 1) * nf // n) for p in range(n)]


def gen_grad_root(cls, only=None, frange=None):
    """One Rys root's contribution to the four gradient blocks:
    R[fi * NE_R + ei] (+)= w * G_x G_y G_z over the block's components.
    only: one block's name -- its f components [frange) alone, written to R
    with weight w (a pass of the split classes)."""
    em = Emitter('    ')
    lij1, lkl1 = cls.lij + 1, cls.lkl + 1
    rects = grad_rects(cls)
    if only is not None:
        rects = [('R', e, f, None if w is None else 'w') for name, e, f, w in rects if name == only]
        # the recurrences only as far as this block reads them
        lij1 = max(e[1] for _, e, _, _ in rects)
        lkl1 = max(f[1] for _, _, f, _ in rects)
    gx = gen_vrr(em, cls, 'x', '1', lij1, lkl1)
    gy = gen_vrr(em, cls, 'y', '1', lij1, lkl1)
    gz = gen_vrr(em, cls, 'z', 'wz', lij1, lkl1)
    # every (e, f) component pair of any block, once
    members = {}
    for name, (e0, e1), (f0, f1), w in rects:
        E, F = _level_set(e0, e1), _level_set(f0, f1)
        if frange is not None:
            F = F[frange[0]:frange[1]]
        for jf, (_, fc) in enumerate(F):
            for ie, (_, ec) in enumerate(E):
                members.setdefault((ec, fc), []).append((name, jf * len(E) + ie, w))
    xy_named = {}
    n = 0
    for (ec, fc), targets in members.items():
        a = gx[(ec[0], fc[0])]
        b = gy[(ec[1], fc[1])]
        c = gz[(ec[2], fc[2])]
        key = (ec[0], fc[0], ec[1], fc[1])
        if a == '1' and b == '1':
            xy = None
        elif a == '1':
            xy = b
        elif b == '1':
            xy = a
        else:
            if key not in xy_named:
                nm = f'xy{len(xy_named)}'
                em(f'const T {nm} = {a} * {b};')
                xy_named[key] = nm
            xy = xy_named[key]
        pv = f'p{n}'
        n += 1
        em(f'const T {pv} = {c if xy is None else xy + " * " + c};')
        for name, k, w in targets:
            if w is None:
                em(f'{name}[{k}] += {pv};')
            else:
                em(f'{name}[{k}] = fma({w}, {pv}, {name}[{k}]);')
    return em.text()


MD_LMAX = 6              # = JK_MD_LMAX (csrc/jk_mdj.cuh)
# classes whose J-only builds take the McMurchie-Davidson kernel by default
# (the per-class choice measured against the Rys J engine)
MD_DEFAULT = frozenset()

# gradient forms: a quartet per lane for the classes of at most
# GRAD_LANE_MAX integrals, a warp per quartet for the rest.  Per-lane classes
# with more block products than GRAD_SPLIT_MIN accumulate a group of at most
# GRAD_PASS_MAX block elements per pass over the primitives (recurrences and
# roots recomputed per pass), which bounds what the primitive loops hold.  W, the
# bra-transferred block and the shifted integrals around them are whole and
# spill: 1 to 11 KB of stores per thread ((dp|ds) 10.6, (dd|ps) 9.9, (pp|pp) 5.2)
GRAD_LANE_MAX = 108
GRAD_SPLIT_MIN = 150
GRAD_PASS_MAX = 64


def grad_members(cls):
    """The distinct (e, f) component pairs of the four gradient blocks."""
    mem = set()
    for _, (e0, e1), (f0, f1), _ in grad_rects(cls):
        for _, ec in _level_set(e0, e1):
            for _, fc in _level_set(f0, f1):
                mem.add((ec, fc))
    return mem


def gen_grad_struct(cls):
    """Lines inside the class struct for the gradient kernel: block sizes,
    level ranges and offsets, the root accumulation (straight-line code for
    the smaller classes; the larger ones loop, see jk_grad.cuh, which keeps
    their compile time bounded), and the transfers of the shells raised and
    lowered by one."""
    li, lj, lk, ll = cls.li, cls.lj, cls.lk, cls.ll
    lines = []
    rects = grad_rects(cls)
    small = ncart(li) * ncart(lj) * ncart(lk) * ncart(ll) <= GRAD_LANE_MAX
    split = small and len(grad_members(cls)) > GRAD_SPLIT_MIN
    lines.append(f'    static constexpr bool G_SMALL = {"true" if small else "false"};')
    lines.append(f'    static constexpr bool G_SPLIT = {"true" if split else "false"};')
    lines.append(f'    static constexpr int G_NMEM = {len(grad_members(cls))};   // block products')
    for name, (e0, e1), (f0, f1), _ in rects:
        ne = len(_level_set(e0, e1))
        nf = len(_level_set(f0, f1))
        lines.append(f'    static constexpr int G_{name}_NE = {ne}, G_{name}_NF = {nf};')
    passes = [grad_passes(len(_level_set(*e)), len(_level_set(*f))) for _, e, f, _ in rects]
    lines.append('    // passes of block r (U, RA, RB, RC) and first f component of pass p')
    lines.append('    static constexpr int g_passes(int r) { return '
                 + ''.join(f'r == {r} ? {len(p)} : ' for r, p in enumerate(passes)) + '0; }')
    lines.append('    static constexpr int g_pass_f(int r, int p) { return '
                 + ''.join(f'r == {r} && p == {k} ? {f0} : ' for r, ps in enumerate(passes)
                           for k, (f0, _) in enumerate(ps))
                 + ''.join(f'r == {r} ? {ps[-1][1]} : ' for r, ps in enumerate(passes)) + '0; }')
    lines.append(f'    static constexpr int G_NROOTS = {(cls.lij + cls.lkl + 1) // 2 + 1};')
    # offsets into U of the lowered transfers' inputs
    ue0, uf0 = max(li - 1, 0), max(lk - 1, 0)
    def off(l0, l):
        return sum(ncart(x) for x in range(l0, l))
    lines.append(f'    static constexpr int G_U_E_LI = {off(ue0, li)};    // level li in U\'s e range')
    lines.append(f'    static constexpr int G_U_F_LK = {off(uf0, lk)};    // level lk in U\'s f range')
    tpl = 'template <class T> __device__ static __forceinline__ void'
    if small and not split:
        lines.append(f'    {tpl} grad_root(T c0x, T c0y, T c0z, T cpx, T cpy, T cpz, T b00, '
                     'T b10, T b01, T wz, T wA, T wB, T wC, T *U, T *RA, T *RB, T *RC) {')
        lines.append(gen_grad_root(cls))
        lines.append('    }')
    if split:
        lines.append('    template <int R, int P, class T> __device__ static __forceinline__ void '
                     'grad_pass(T c0x, T c0y, T c0z, T cpx, T cpy, T cpz, T b00, T b10, T b01, '
                     'T wz, T w, T *R_) {')
        for r, (name, _, _, _) in enumerate(rects):
            for p, fr in enumerate(passes[r]):
                lines.append(f'    if constexpr (R == {r} && P == {p}) {{')
                lines.append(gen_grad_root(cls, only=name, frange=fr).replace('R[', 'R_['))
                lines.append('    }')
        lines.append('    }')
    tpl_s = ('template <class T, int SI = 1, int SO = 1> __device__ static __forceinline__ '
             'void')
    shifts = [('ip', li + 1, lj, 'hbi', 'AB'), ('jp', li, lj + 1, 'hbj', 'AB'),
              ('kp', lk + 1, ll, 'hkk', 'CD')]
    if li > 0:
        shifts.append(('im', li - 1, lj, 'hbm', 'AB'))
    if lj > 0:
        shifts.append(('jm', li, lj - 1, 'hbn', 'AB'))
    if lk > 0:
        shifts.append(('km', lk - 1, ll, 'hkm', 'CD'))
    for tag, la, lb, prefix, vec in shifts:
        args = 'T ABx, T ABy, T ABz' if vec == 'AB' else 'T CDx, T CDy, T CDz'
        lines.append(f'    {tpl_s} hrr_{tag}(const T *in, T *out, {args}) {{')
        lines.append(gen_hrr(la, lb, prefix, vec))
        lines.append('    }')
    return lines


def gen_class_header(cls):
    E = cls.eset()
    tpl = 'template <class T> __device__ static __forceinline__ void'
    lines = [f'struct Cls_{cls.tag} {{',
             f'    static constexpr int LI = {cls.li}, LJ = {cls.lj}, '
             f'LK = {cls.lk}, LL = {cls.ll};',
             f'    static constexpr int LIJ = {cls.lij}, LKL = {cls.lkl}, '
             f'NROOTS = {cls.nroots};',
             f'    static constexpr int NI = {ncart(cls.li)}, NJ = {ncart(cls.lj)}, '
             f'NK = {ncart(cls.lk)}, NL = {ncart(cls.ll)};',
             f'    static constexpr int NE = {cls.ne}, NF = {cls.nf};',
             f'    static constexpr bool REG = {"true" if cls.form == "reg" else "false"};']
    if cls.form == 'team' or len(cls.passes()) > 1:
        parts = cls.fparts()
        lines.append(f'    static constexpr int TEAM_LANES = {cls.team_lanes}, '
                     f'NWF = {cls.nwf}, TEAM = {cls.team_threads};')
        lines.append(f'    static constexpr int FPART = {parts[0][1] - parts[0][0]};')
        # e-component table: ex, ey, ez per e index
        ex = ', '.join(str(c[0]) for _, c in E)
        ey = ', '.join(str(c[1]) for _, c in E)
        ez = ', '.join(str(c[2]) for _, c in E)
        lines.append(f'    __device__ static __forceinline__ int ex(int e) '
                     f'{{ constexpr int t[NE] = {{{ex}}}; return t[e]; }}')
        lines.append(f'    __device__ static __forceinline__ int ey(int e) '
                     f'{{ constexpr int t[NE] = {{{ey}}}; return t[e]; }}')
        lines.append(f'    __device__ static __forceinline__ int ez(int e) '
                     f'{{ constexpr int t[NE] = {{{ez}}}; return t[e]; }}')
        for p, (f0, f1) in enumerate(parts):
            lines.append(f'    {tpl} row_acc_{p}('
                         'const T *gx, const T *gy, const T *gz, T *acc) {')
            lines.append(gen_row_acc(cls, f0, f1))
            lines.append('    }')
        lines.append('    template <int P, class T> __device__ static __forceinline__ void '
                     'row_acc(const T *gx, const T *gy, const T *gz, T *acc) {')
        for p in range(len(parts)):
            lines.append(f'        if (P == {p}) row_acc_{p}<T>(gx, gy, gz, acc);')
        lines.append('    }')
        lines.append('    template <int P> __device__ static constexpr int fbegin() {')
        lines.append('        return ' + ' '.join(f'P == {p} ? {f0} :' for p, (f0, _) in enumerate(parts)) + ' 0;')
        lines.append('    }')
        lines.append('    template <int P> __device__ static constexpr int fend() {')
        lines.append('        return ' + ' '.join(f'P == {p} ? {f1} :' for p, (_, f1) in enumerate(parts)) + ' 0;')
        lines.append('    }')
    else:
        lines.append('    static constexpr int TEAM_LANES = 1, NWF = 1, TEAM = 1, FPART = NF;')
    if cls.form == 'team':
        lines.append('    static constexpr int NPASS = 0;')
    else:
        passes = cls.passes()
        lines.append(f'    static constexpr int NPASS = {len(passes)};')
        lines.append('    static constexpr int pass_f(int p) { return '
                     + ''.join(f'p == {p} ? {f0} : ' for p, (f0, _) in enumerate(passes))
                     + 'NF; }')
        if cls.nroots <= 2:
            lines.append('    __device__ static __forceinline__ void boys_acc(const double *F, '
                         'double PAx, double PAy, double PAz, double WPx, double WPy, double WPz, '
                         'double QCx, double QCy, double QCz, double WQx, double WQy, double WQz, '
                         'double hp, double sp, double hs, double *acc) {')
            lines.append(gen_boys_acc(cls))
            lines.append('    }')
        lines.append('    template <int P, class T> __device__ static __forceinline__ void root_acc('
                     'T c0x, T c0y, T c0z, T cpx, T cpy, T cpz, T b00, T b10, T b01, '
                     'T wz, T *acc) {')
        for p, (f0, f1) in enumerate(passes):
            if len(passes) > 1:
                lines.append(f'    if constexpr (P == {p}) {{')
            lines.append(gen_root_acc(cls, f0, f1))
            if len(passes) > 1:
                lines.append('    }')
        lines.append('    }')
    tpl_s = ('template <class T, int SI = 1, int SO = 1> __device__ static __forceinline__ '
             'void')
    lines.append(f'    {tpl_s} hrr_bra(const T *in, T *out, T ABx, T ABy, T ABz) {{')
    lines.append(gen_hrr(cls.li, cls.lj, 'hb', 'AB'))
    lines.append('    }')
    lines.append(f'    {tpl_s} hrr_ket(const T *in, T *out, T CDx, T CDy, T CDz) {{')
    lines.append(gen_hrr(cls.lk, cls.ll, 'hk', 'CD'))
    lines.append('    }')
    lines += gen_grad_struct(cls)
    lines.append('};')
    return '\n'.join(lines)


def gen_unit(A, B, cls):
    lines = ['// Generated by electrolites_b200/codegen/gen_classes.py -- do not edit.',
             '#include "../jk_kernels.cuh"',
             '',
             gen_class_header(cls),
             '',
             f'JK_DEFINE_CLASS({cls.tag}, {A}, {B})']
    lines.append('')
    return '\n'.join(lines)


def gen_pairs(lmax):
    """The J engine's pair transforms: a struct per pair class (sizes and its
    bra transfer) and one kernel each way over the pairs of every class."""
    pairs = [(la, lb) for la in range(lmax + 1) for lb in range(la + 1)]
    lines = ['// Generated by electrolites_b200/codegen/gen_classes.py -- do not edit.',
             '#include "../jk_pairs.cuh"', '']
    for la, lb in pairs:
        cls = Cls(la, lb, 0, 0)
        lines += [f'struct Pair_{la}{lb} {{',
                  f'    static constexpr int LI = {la}, LJ = {lb}, LK = 0, LL = 0;',
                  f'    static constexpr int NI = {ncart(la)}, NJ = {ncart(lb)}, NE = {cls.ne};',
                  '    template <class T, int SI = 1, int SO = 1> __device__ static __forceinline__ '
                  'void hrr_bra(const T *in, T *out, T ABx, T ABy, T ABz) {',
                  gen_hrr(la, lb, 'hb', 'AB'),
                  '    }', '};']
    for name, per in (('dens', 'Pair_{0}{1}::NE'), ('post', '1')):
        lines += [f'__global__ void __launch_bounds__(JX_THREADS) jx_{name}_kernel(const PairBatch a)',
                  '{',
                  '    int k = 0;',
                  '    while ((int)blockIdx.x >= a.blk0[k + 1]) ++k;',
                  '    const long long t = (long long)(blockIdx.x - a.blk0[k]) * JX_THREADS + threadIdx.x;',
                  '    switch (k) {']
        for k, (la, lb) in enumerate(pairs):
            lines.append(f'    case {k}: jx_{name}_one<Pair_{la}{lb}>(a, a.pairs[{k}], a.npairs[{k}], t); break;')
        lines += ['    }', '}',
                  f'int jk_jx_{name}(PairBatch a, cudaStream_t st)', '{',
                  '    const int per[JK_PAIR_CLASSES] = {'
                  + ', '.join(per.format(la, lb) for la, lb in pairs)
                  + ', 0' * (10 - len(pairs)) + '};',
                  '    long long blk = 0;',
                  '    for (int k = 0; k < JK_PAIR_CLASSES; ++k) {',
                  '        a.blk0[k] = (int)blk;',
                  '        blk += ((long long)a.npairs[k] * a.n_j * per[k] + JX_THREADS - 1) / JX_THREADS;',
                  '    }',
                  '    if (blk > 0x7fffffff) return (int)cudaErrorInvalidValue;',
                  '    a.blk0[JK_PAIR_CLASSES] = (int)blk;',
                  '    if (blk == 0) return 0;',
                  f'    jx_{name}_kernel<<<(unsigned)blk, JX_THREADS, 0, st>>>(a);',
                  '    return (int)cudaGetLastError();', '}', '']
    return '\n'.join(lines)


def _write(path, src):
    old = open(path).read() if os.path.exists(path) else None
    if old != src:
        with open(path + '.tmp', 'w') as f:
            f.write(src)
        os.replace(path + '.tmp', path)
    return path


def write_all(outdir, lmax=LMAX):
    os.makedirs(outdir, exist_ok=True)
    classes = all_classes(lmax)
    written = []
    for A, B, cls in classes:
        written.append(_write(os.path.join(outdir, f'class_{cls.tag}.cu'), gen_unit(A, B, cls)))
    written.append(_write(os.path.join(outdir, 'jx_pairs.cu'), gen_pairs(lmax)))
    # registry: declarations + table in pair-class order
    reg = ['// Generated by electrolites_b200/codegen/gen_classes.py -- do not edit.',
           '#pragma once',
           '#include "../jk_launch.h"']
    for A, B, cls in classes:
        reg.append(f'int jk_launch_{cls.tag}(const ClassArgs &a, const PlanView *views, '
                   'const LaunchCfg &cfg);')
    reg.append(f'#define JK_NCLASSES {len(classes)}')
    reg.append('static const ClassEntry jk_class_table[JK_NCLASSES] = {')
    for A, B, cls in classes:
        form = 0 if cls.form == 'reg' else 1
        small = cls.ne * cls.nf <= REG_MAX
        fp32 = 1 if cls.tag in FP32_DEFAULT else 0
        # McMurchie-Davidson J kernel (J-only builds): register-form classes
        # up to JK_MD_LMAX; md_default: the classes where it measured faster
        # than the Rys J engine
        md = 1 if small and cls.li + cls.lj + cls.lk + cls.ll <= MD_LMAX else 0
        md_def = 1 if md and cls.tag in MD_DEFAULT else 0
        reg.append(f'    {{{A}, {B}, {cls.li}, {cls.lj}, {cls.lk}, {cls.ll}, '
                   f'{form}, {1 if small else cls.team_threads}, {fp32}, '
                   f'{md}, {md_def}, jk_launch_{cls.tag}}},')
    reg.append('};')
    with open(os.path.join(outdir, 'class_table.inc.tmp'), 'w') as f:
        f.write('\n'.join(reg) + '\n')
    os.replace(os.path.join(outdir, 'class_table.inc.tmp'),
               os.path.join(outdir, 'class_table.inc'))
    return written


if __name__ == '__main__':
    out = sys.argv[1] if len(sys.argv) > 1 else os.path.join(
        os.path.dirname(os.path.abspath(__file__)), '..', 'csrc', 'generated')
    for p in write_all(out):
        print(p)
