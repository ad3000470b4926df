"""
Cases for timing the tissue simulations of this package: short runs through
``SimulationCUDA`` (logged runs and device frames), ``CableBatch`` and the
differentiable ``tissue_loss``, over cables, sheets and connection graphs
from ten cells to four million, in both precisions.

The package takes its models as myokit objects. So that the cases need
nothing but this repository, the part of that model layer which the package
calls (expressions, a model of equations in solvable order, events, a log)
is stated here in a small form of its own and registered under the name the
package imports. Two models are written below as plain equations:

- ``br``: Beeler-Reuter 1977, 8 states, forward Euler;
- ``v48``: a generic ventricular cell of 48 states around the currents of
  Luo-Rudy 1991 (gates, a Markov channel, buffered calcium with cubic roots,
  ion concentrations), Rush-Larsen gates. It stands for detailed human and
  canine models of that size.

``exact`` evaluates the same equation text with torch in 64 bits.
"""
import ast
import math
import sys
import types
from collections import OrderedDict, namedtuple

import numpy as np
import torch

# ---------------------------------------------------------------------------
# Models as text: "name = expression", "dot(name) = expression @ initial
# value"; "gate(name) = inf, tau @ initial value" for a gate that relaxes to
# inf with time constant tau. A trailing [mM] marks a concentration.
# ---------------------------------------------------------------------------

BR = '''
engine.time := time
engine.pace := pace
membrane.i_diff := diffusion_current
membrane.amplitude = -25
membrane.i_stim = engine.pace * membrane.amplitude
dot(membrane.V) = -(ik1.I + ix1.I + ina.I + isi.I + membrane.i_stim + membrane.i_diff) / 1.0 @ -84.622
ik1.I = 0.35 * (4 * (exp(0.04 * (membrane.V + 85)) - 1) / (exp(0.08 * (membrane.V + 53)) + exp(0.04 * (membrane.V + 53))) + 0.2 * where(abs(membrane.V + 23) >= 0.01, (membrane.V + 23) / (1 - exp(-0.04 * (membrane.V + 23))), 25))
ix1.a = 0.0005 * exp(0.083 * (membrane.V + 50)) / (exp(0.057 * (membrane.V + 50)) + 1)
ix1.b = 0.0013 * exp(-0.06 * (membrane.V + 20)) / (exp(-0.04 * (membrane.V + 20)) + 1)
dot(ix1.x1) = ix1.a * (1 - ix1.x1) - ix1.b * ix1.x1 @ 0.0004
ix1.I = ix1.x1 * 0.8 * (exp(0.04 * (membrane.V + 77)) - 1) / exp(0.04 * (membrane.V + 35))
ina.g = 4
ina.gc = 0.003
ina.E = 50
ina.am = where(abs(membrane.V + 47) >= 0.01, (membrane.V + 47) / (1 - exp(-0.1 * (membrane.V + 47))), 10)
ina.bm = 40 * exp(-0.056 * (membrane.V + 72))
dot(ina.m) = ina.am * (1 - ina.m) - ina.bm * ina.m @ 0.01
ina.ah = 0.126 * exp(-0.25 * (membrane.V + 77))
ina.bh = 1.7 / (1 + exp(-0.082 * (membrane.V + 22.5)))
dot(ina.h) = ina.ah * (1 - ina.h) - ina.bh * ina.h @ 0.99
ina.aj = 0.055 * exp(-0.25 * (membrane.V + 78)) / (1 + exp(-0.2 * (membrane.V + 78)))
ina.bj = 0.3 / (1 + exp(-0.1 * (membrane.V + 32)))
dot(ina.j) = ina.aj * (1 - ina.j) - ina.bj * ina.j @ 0.98
ina.I = (ina.g * ina.m ** 3 * ina.h * ina.j + ina.gc) * (membrane.V - ina.E)
isi.g = 0.09
isi.ad = 0.095 * exp(-0.01 * (membrane.V - 5)) / (1 + exp(-0.072 * (membrane.V - 5)))
isi.bd = 0.07 * exp(-0.017 * (membrane.V + 44)) / (1 + exp(0.05 * (membrane.V + 44)))
dot(isi.d) = isi.ad * (1 - isi.d) - isi.bd * isi.d @ 0.003
isi.af = 0.012 * exp(-0.008 * (membrane.V + 28)) / (1 + exp(0.15 * (membrane.V + 28)))
isi.bf = 0.0065 * exp(-0.02 * (membrane.V + 30)) / (1 + exp(-0.2 * (membrane.V + 30)))
dot(isi.f) = isi.af * (1 - isi.f) - isi.bf * isi.f @ 0.99
dot(isi.Ca) = -1e-7 * isi.I + 0.07 * (1e-7 - isi.Ca) @ 2e-7 [M]
isi.E = -82.3 - 13.0287 * log(isi.Ca)
isi.I = isi.g * isi.d * isi.f * (membrane.V - isi.E)
'''


def _sigmoid(v, k):
    return f'1 / (1 + exp((membrane.V + {v}) / {k}))'


def _bell(t0, t1, v, w):
    return f'{t0} + {t1} * exp(-((membrane.V + {v}) / {w}) ** 2)'


def _cubic(name, total, b1, k1, b2, k2):
    """Free concentration under two buffers: root of a cubic."""
    return f'''
{name}_b = {b1} + {b2} - {total} + {k1} + {k2}
{name}_c = {k1} * {k2} - {total} * ({k1} + {k2}) + {b1} * {k2} + {b2} * {k1}
{name}_d = -{k1} * {k2} * {total}
{name} = (2 / 3) * sqrt({name}_b ** 2 - 3 * {name}_c) * cos(acos((9 * {name}_b * {name}_c - 2 * {name}_b ** 3 - 27 * {name}_d) / (2 * ({name}_b ** 2 - 3 * {name}_c) ** 1.5)) / 3) - {name}_b / 3
'''


V48 = f'''
engine.time := time
engine.pace := pace
membrane.i_diff := diffusion_current
phys.F = 96.485
phys.RTF = 26.7137
phys.Ko = 5.4
phys.Nao = 140
phys.Cao = 1.8
phys.Clo = 100
cell.vcell = 3.8e-5
cell.acap = 1.534e-4
cell.vi = cell.vcell * 0.58
cell.vss = cell.vcell * 0.04
cell.vnsr = cell.vcell * 0.08
cell.vjsr = cell.vcell * 0.02
membrane.amplitude = -60
membrane.i_stim = engine.pace * membrane.amplitude
membrane.i_ion = ina.I + inal.I + ical.I + icat.I + ik.I + ik1.I + ikp.I + ito.I + ikr.I + iks.I + iherg.I + ifun.I + icl.I + inaca.Ii + inaca.Iss + inak.I + ipca.I + ib.I
dot(membrane.V) = -(membrane.i_ion + membrane.i_stim + membrane.i_diff) @ -84.5
ina.Gbar = 16
ina.E = phys.RTF * log(phys.Nao / na.ss)
ina.am = where(abs(membrane.V + 47.13) >= 0.01, 0.32 * (membrane.V + 47.13) / (1 - exp(-0.1 * (membrane.V + 47.13))), 3.2)
ina.bm = 0.08 * exp(-membrane.V / 11)
ina.tm = 1 / (ina.am + ina.bm)
ina.im = ina.am * ina.tm
gate(ina.m) = ina.im, ina.tm @ 0.0017
ina.ah = where(membrane.V >= -40, 0, 0.135 * exp((80 + membrane.V) / -6.8))
ina.bh = where(membrane.V >= -40, 1 / (0.13 * (1 + exp((membrane.V + 10.66) / -11.1))), 3.56 * exp(0.079 * membrane.V) + 310000 * exp(0.35 * membrane.V))
ina.th = 1 / (ina.ah + ina.bh)
ina.ih = ina.ah * ina.th
gate(ina.h) = ina.ih, ina.th @ 0.983
ina.aj = where(membrane.V >= -40, 0, (-127140 * exp(0.2444 * membrane.V) - 3.474e-5 * exp(-0.04391 * membrane.V)) * (membrane.V + 37.78) / (1 + exp(0.311 * (membrane.V + 79.23))))
ina.bj = where(membrane.V >= -40, 0.3 * exp(-2.535e-7 * membrane.V) / (1 + exp(-0.1 * (membrane.V + 32))), 0.1212 * exp(-0.01052 * membrane.V) / (1 + exp(-0.1378 * (membrane.V + 40.14))))
ina.tj = 1 / (ina.aj + ina.bj)
ina.ij = ina.aj * ina.tj
gate(ina.j) = ina.ij, ina.tj @ 0.989
ina.phi = 1 / (1 + 0.05 / camk.active)
ina.I = ina.Gbar * ina.m ** 3 * ina.h * ina.j * (membrane.V - ina.E) * (1 - 0.02 * ina.phi)
inal.G = 0.0075
inal.im = {_sigmoid(42.85, -5.264)}
gate(inal.m) = inal.im, ina.tm @ 0.0002
inal.ih = {_sigmoid(87.61, 7.488)}
inal.th = 200
gate(inal.h) = inal.ih, inal.th @ 0.5
inal.I = inal.G * inal.m * inal.h * (membrane.V - ina.E) * (1 + 0.1 * ina.phi)
ical.G = 0.09
ical.E = 7.7 - 13.0287 * log(ca.cal)
ical.ad = 0.095 * exp(-0.01 * (membrane.V - 5)) / (1 + exp(-0.072 * (membrane.V - 5)))
ical.bd = 0.07 * exp(-0.017 * (membrane.V + 44)) / (1 + exp(0.05 * (membrane.V + 44)))
ical.td = 1 / (ical.ad + ical.bd)
ical.id = ical.ad * ical.td
gate(ical.d) = ical.id, ical.td @ 0.003
ical.af = 0.012 * exp(-0.008 * (membrane.V + 28)) / (1 + exp(0.15 * (membrane.V + 28)))
ical.bf = 0.0065 * exp(-0.02 * (membrane.V + 30)) / (1 + exp(-0.2 * (membrane.V + 30)))
ical.tf = 1 / (ical.af + ical.bf)
ical.if = ical.af * ical.tf
gate(ical.f) = ical.if, ical.tf @ 0.999
ical.if2 = 0.4 + 0.6 / (1 + exp((membrane.V + 15) / 6))
ical.tf2 = 1 / (0.0197 * exp(-(0.0337 * (membrane.V + 10)) ** 2) + 0.02)
gate(ical.f2) = ical.if2, ical.tf2 @ 0.999
ical.ifca = 0.3 / (1 - ical.I / 0.05) + 0.55 / (1 + ca.cal / 0.003) + 0.15
ical.tfca = 10 * ina.phi + 0.5 + 1 / (1 + ca.cal / 0.003)
dot(ical.fca) = (ical.ifca - ical.fca) / ical.tfca @ 0.98
ical.I = ical.G * ical.d * ical.f * ical.f2 * (0.7 + 0.3 * ical.fs ** 4) * (membrane.V - ical.E)
ical.fs = 1 / (1 + (ca.cal / 0.01) ** 2)
icat.G = 0.005
icat.ib = {_sigmoid(54, -7.4)}
icat.tb = 0.6 + 5.4 / (1 + exp(0.03 * (membrane.V + 100)))
gate(icat.b) = icat.ib, icat.tb @ 0.016
icat.ig = {_sigmoid(68, 5.6)}
icat.tg = 1 + 40 / (1 + exp(0.08 * (membrane.V + 65)))
gate(icat.g) = icat.ig, icat.tg @ 0.95
icat.I = icat.G * icat.b ** 2 * icat.g * (membrane.V - 50)
ik.G = 0.282
ik.a = 0.0005 * exp(0.083 * (membrane.V + 50)) / (1 + exp(0.057 * (membrane.V + 50)))
ik.b = 0.0013 * exp(-0.06 * (membrane.V + 20)) / (1 + exp(-0.04 * (membrane.V + 20)))
ik.t = 1 / (ik.a + ik.b)
ik.i = ik.a * ik.t
gate(ik.x) = ik.i, ik.t @ 0.006
ik.xi = where(abs(membrane.V + 77.6) >= 0.01, 2.837 * (exp(0.04 * (membrane.V + 77.6)) - 1) / ((membrane.V + 77.6) * exp(0.04 * (membrane.V + 35))), 0.1135 / exp(0.04 * (membrane.V + 35)))
ik.I = ik.G * ik.x * ik.xi * (membrane.V + 77.6)
ik1.G = 0.6047
ik1.E = phys.RTF * log(phys.Ko / k.i)
ik1.a = 1.02 / (1 + exp(0.2385 * (membrane.V - ik1.E - 59.215)))
ik1.b = (0.49124 * exp(0.08032 * (membrane.V - ik1.E + 5.476)) + exp(0.06175 * (membrane.V - ik1.E - 594.31))) / (1 + exp(-0.5143 * (membrane.V - ik1.E + 4.753)))
ik1.I = ik1.G * ik1.a / (ik1.a + ik1.b) * (membrane.V - ik1.E)
ikp.I = 0.0183 / (1 + exp((7.488 - membrane.V) / 5.98)) * (membrane.V - ik1.E)
ito.G = 0.05
ito.aa = 1 / (1.2089 * (1 + exp((membrane.V - 18.41) / -29.38)))
ito.ab = 3.5 / (1 + exp((membrane.V + 100) / 29.38))
ito.ia = {_sigmoid(9.437, -7.133)}
ito.ta = 1 / (ito.aa / 1.2 + ito.ab / 2.5)
gate(ito.a) = ito.ia, ito.ta @ 0.0001
ito.ii = {_sigmoid(58.5, 10.5)}
ito.ti1 = 2 + 1 / (0.025 / (1 + exp((membrane.V + 58) / 5)) + 1 / (9.7953 * (1 + exp((membrane.V + 19) / -9))))
gate(ito.i1) = ito.ii, ito.ti1 @ 0.92
ito.ti2 = 10 + 250 / (1 + exp((membrane.V + 60) / 5)) + 43 / (1 + exp((membrane.V + 16) / -9))
gate(ito.i2) = ito.ii, ito.ti2 @ 0.92
ito.r = 1 / (1 + exp((membrane.V - 60) / -100))
ito.I = ito.G * ito.a ** 3 * (0.7 * ito.i1 + 0.3 * ito.i2) * ito.r * (membrane.V - ik1.E)
ikr.Gbar = 0.0138
ikr.ix = {_sigmoid(10.085, -4.25)}
ikr.ta = where(abs(membrane.V - 1.7384) >= 0.01, 0.0006 * (membrane.V - 1.7384) / (1 - exp(-0.136 * (membrane.V - 1.7384))), 0.0044)
ikr.tb = where(abs(membrane.V + 38.3608) >= 0.01, 0.0003 * (membrane.V + 38.3608) / (exp(0.1522 * (membrane.V + 38.3608)) - 1), 0.00197)
ikr.tx = 1 / (ikr.ta + ikr.tb)
gate(ikr.x) = ikr.ix, ikr.tx @ 0.0001
ikr.r = 1 / (1 + exp((membrane.V + 10) / 15.4))
ikr.I = ikr.Gbar * sqrt(phys.Ko / 5.4) * ikr.x * ikr.r * (membrane.V - ik1.E)
iks.Gbar = 0.0826
iks.E = phys.RTF * log((phys.Ko + 0.01833 * phys.Nao) / (k.i + 0.01833 * na.i))
iks.ix = {_sigmoid(-10.5, -24.7)}
iks.ta = where(membrane.V >= -44.5, 7.61e-5 * (membrane.V + 44.6) / (1 - exp(-0.997 * (membrane.V + 44.6))), 7.61e-5)
iks.tb = where(abs(membrane.V - 0.55) >= 0.01, 3.6e-4 * (membrane.V - 0.55) / (exp(0.128 * (membrane.V - 0.55)) - 1), 0.0028)
iks.tx1 = 1 / (iks.ta + iks.tb)
gate(iks.x1) = iks.ix, iks.tx1 @ 0.02
iks.tx2 = 2 * iks.tx1
gate(iks.x2) = iks.ix, iks.tx2 @ 0.02
iks.ca = 1 + 0.6 / (1 + (3.8e-5 / ca.i) ** 1.4)
iks.I = iks.Gbar * iks.ca * iks.x1 * iks.x2 * (membrane.V - iks.E)
iherg.G = 0.01
iherg.a1 = 0.02 * exp(0.03 * (membrane.V + 20))
iherg.b1 = 0.025 * exp(-0.03 * (membrane.V + 20))
iherg.a2 = 0.05 * exp(0.012 * membrane.V)
iherg.b2 = 0.04 * exp(-0.035 * membrane.V)
iherg.ai = 0.1 * exp(0.02 * (membrane.V + 10))
iherg.bi = 0.02 * exp(-0.018 * (membrane.V + 10))
dot(iherg.c3) = iherg.b1 * iherg.c2 - iherg.a1 * iherg.c3 @ 0.9
dot(iherg.c2) = iherg.a1 * iherg.c3 + 0.05 * iherg.c1 - (iherg.b1 + 0.08) * iherg.c2 @ 0.05
dot(iherg.c1) = 0.08 * iherg.c2 + iherg.b2 * iherg.o - (0.05 + iherg.a2) * iherg.c1 @ 0.03
dot(iherg.o) = iherg.a2 * iherg.c1 + iherg.bi * iherg.inact - (iherg.b2 + iherg.ai) * iherg.o @ 0.01
dot(iherg.inact) = iherg.ai * iherg.o - iherg.bi * iherg.inact @ 0.01
iherg.I = iherg.G * iherg.o * (membrane.V - ik1.E)
ifun.G = 0.0003
ifun.iy = {_sigmoid(87, 9.5)}
ifun.ty = 2000 / (exp(-(membrane.V + 132) / 10) + exp((membrane.V + 57) / 60))
gate(ifun.y) = ifun.iy, ifun.ty @ 0.1
ifun.I = ifun.G * ifun.y * (0.35 * (membrane.V - ina.E) + 0.65 * (membrane.V - ik1.E))
icl.P = 2e-5
icl.i2 = 1 / (1 + ca.ss / 0.0015)
icl.in = {_sigmoid(30, 12.0)}
icl.tn = 8 / (1 + 0.09 / ca.ss) + 3
gate(icl.n) = icl.in, icl.tn @ 0.99
icl.z = membrane.V / phys.RTF
icl.flux = where(abs(icl.z) >= 0.001, icl.P * icl.z * phys.F * (cl.i - phys.Clo * exp(icl.z)) / (1 - exp(icl.z)), icl.P * phys.F * (phys.Clo - cl.i))
icl.I = icl.flux * icl.n * (1 - icl.i2)
inaca.hna = exp(0.27 * membrane.V / phys.RTF)
inaca.hca = exp(-0.73 * membrane.V / phys.RTF)
inaca.di = (1 + (1.25e-4 / ca.i) ** 2) * (87.5 ** 3 + phys.Nao ** 3) * (1.38 + phys.Cao) * (1 + 0.27 * inaca.hca)
inaca.Ii = 1500 * (inaca.hna * na.i ** 3 * phys.Cao - inaca.hca * phys.Nao ** 3 * ca.i * 1.5) / inaca.di
inaca.ds = (1 + (1.25e-4 / ca.ss) ** 2) * (87.5 ** 3 + phys.Nao ** 3) * (1.38 + phys.Cao) * (1 + 0.27 * inaca.hca)
inaca.Iss = 60 * (inaca.hna * na.ss ** 3 * phys.Cao - inaca.hca * phys.Nao ** 3 * ca.ss * 1.5) / inaca.ds
inak.f = 1 / (1 + 0.1245 * exp(-0.1 * membrane.V / phys.RTF) + 0.0365 * 1.2 * exp(-membrane.V / phys.RTF))
inak.I = 0.6 * inak.f * phys.Ko / (phys.Ko + 1.5) / (1 + (10 / na.i) ** 1.5)
ipca.I = 0.03 * ca.i / (0.0005 + ca.i)
ib.I = 0.03921 * (membrane.V + 63)
{_cubic('ca.i', 'cabuf.i', 0.05, 0.00238, 0.07, 0.0005)}
{_cubic('ca.cal', 'cabuf.cal', 0.3, 0.02, 0.047, 0.004)}
{_cubic('ca.jsr', 'cabuf.jsr', 10.0, 0.8, 2.0, 0.1)}
ca.ss = cabuf.ss / (1 + 1.124 / (0.0087 + cabuf.ss) + 0.047 / (0.00087 + cabuf.ss))
camk.bound = 0.05 * (1 - camk.trap) / (1 + 0.0015 / ca.ss)
camk.active = camk.bound + camk.trap
dot(camk.trap) = 0.05 * camk.active * camk.bound - 0.00068 * camk.trap @ 0.02
irel.drive = 1 / (1 + (1.0 / ca.jsr) ** 8)
irel.iro = irel.drive / (1 + (0.001 / ca.ss) ** 2) * (1 - ical.I / (1 + abs(ical.I)))
irel.tro = 2 + 1 / (1 + (ca.ss / 0.01) ** 2)
dot(irel.ro) = (irel.iro - irel.ro) / irel.tro @ 0.001
irel.iri = 1 / (1 + exp((ca.ss - 4e-4 + 0.002 * camk.active) / 2.5e-4))
irel.tri = (350 - irel.cafac) / (1 + exp((ca.ss - 0.003 + 0.003 * irel.drive) / 0.0002)) + 3 + irel.cafac
irel.cafac = 50 / (1 + exp((ical.I + 0.05) / 0.015))
dot(irel.ri) = (irel.iri - irel.ri) / irel.tri @ 0.8
irel.tj = 4.75 / (1 + 0.0123 / ca.jsr)
dot(irel.j1) = (0.02 * irel.ro * irel.ri * (ca.jsr - ca.ss) - irel.j1) / irel.tj @ 0.0001
dot(irel.j2) = (irel.j1 - irel.j2) / (1 + 2 * irel.tj) @ 0.0001
jup.plb = 0.00017 * camk.active / (0.15 + camk.active)
jup.I = 0.004375 * (1 + 0.75 * camk.active / (0.15 + camk.active)) * ca.i / (ca.i + 0.00092 - jup.plb) - 0.004375 / 15 * ca.nsr
jtr.I = (ca.nsr - ca.jsr) / 120
jdiff.ca = (ca.ss - ca.i) / 0.2
jdiff.cal = (ca.cal - ca.ss) / 2
jdiff.na = (na.ss - na.i) / 2
jdiff.k = (k.ss - k.i) / 2
jdiff.cl = (cl.ss - cl.i) / 2
dot(na.i) = -(ib.I * 0.1 + 3 * inak.I + 3 * inaca.Ii) * cell.acap / (cell.vi * phys.F * 1000) + jdiff.na * cell.vss / cell.vi @ 9.5 [mM]
dot(na.ss) = -(ina.I + inal.I + 3 * inaca.Iss) * cell.acap / (cell.vss * phys.F * 1e5) - jdiff.na @ 9.5 [mM]
dot(k.i) = -(ik1.I + ik.I + ikp.I + ikr.I + iks.I + ito.I + iherg.I - 2 * inak.I) * cell.acap / (cell.vi * phys.F * 1000) + jdiff.k * cell.vss / cell.vi @ 141 [mM]
dot(k.ss) = -(0.1 * ik1.I + ifun.I) * cell.acap / (cell.vss * phys.F * 1e5) - jdiff.k @ 141 [mM]
dot(cl.i) = icl.I * cell.acap / (cell.vi * phys.F * 1000) + jdiff.cl * cell.vss / cell.vi @ 18 [mM]
dot(cl.ss) = 0.5 * icl.I * cell.acap / (cell.vss * phys.F * 1e5) - jdiff.cl @ 18 [mM]
dot(cabuf.i) = -(ipca.I - 2 * inaca.Ii) * cell.acap / (2 * cell.vi * phys.F * 1000) - jup.I * cell.vnsr / cell.vi + jdiff.ca * 0.1 * cell.vss / cell.vi - buf.jtrpn @ 0.0137 [mM]
dot(cabuf.ss) = jdiff.cal * 0.1 + irel.j1 * cell.vjsr / cell.vss + 2 * inaca.Iss * cell.acap / (2 * cell.vss * phys.F * 1e5) - jdiff.ca * 0.1 @ 0.02 [mM]
dot(cabuf.cal) = -ical.I * cell.acap / (2 * cell.vss * phys.F * 12000) - jdiff.cal * 0.03 @ 0.0027 [mM]
dot(ca.nsr) = jup.I - jtr.I * cell.vjsr / cell.vnsr @ 1.3 [mM]
dot(cabuf.jsr) = jtr.I - irel.j2 @ 9.0 [mM]
buf.jtrpn = 1e-4 * buf.jt
buf.jt = 20 * ca.i * (1 - buf.trpn) - 0.02 * buf.trpn
dot(buf.trpn) = buf.jt @ 0.08
dot(buf.cmdn) = 30 * ca.i * (1 - buf.cmdn) - 0.07 * buf.cmdn @ 0.04
dot(buf.csqn) = 0.01 * ca.jsr * (1 - buf.csqn) - 0.008 * buf.csqn @ 0.6
dot(slow.atp) = 0.0005 * (1 - slow.atp) - 0.0001 * inak.I * slow.atp / (0.1 + slow.atp) @ 0.95
dot(slow.adp) = 0.0001 * inak.I * slow.atp / (0.1 + slow.atp) - 0.0005 * slow.adp @ 0.05
dot(slow.ros) = 0.0002 * slow.adp / (0.2 + slow.adp) - 0.0003 * slow.ros @ 0.05
'''

TEXT = {'br': BR, 'v48': V48}

# ---------------------------------------------------------------------------
# The model layer the package calls
# ---------------------------------------------------------------------------

SINGLE, DOUBLE = 32, 64


class Expression:
    """A node with operands; equal when type, operands and value are."""
    def __init__(self, *operands):
        self._ops = operands
        self._hash = hash((type(self), self._value(), operands))

    def _value(self):
        return None

    def __len__(self):
        return len(self._ops)

    def __getitem__(self, i):
        return self._ops[i]

    def __iter__(self):
        return iter(self._ops)

    def __hash__(self):
        return self._hash

    def __eq__(self, other):
        return self is other or (
            type(self) is type(other) and self._hash == other._hash
            and self._value() == other._value() and self._ops == other._ops)

    def walk(self):
        yield self
        for x in self._ops:
            yield from x.walk()

    def references(self):
        return set(x for x in self.walk() if isinstance(x, (Name, Derivative)))

    def clone(self, subst=None):
        if subst and self in subst:
            return subst[self]
        if not self._ops:
            return self
        return type(self)(*[x.clone(subst) for x in self._ops])

    def eval(self, subst=None, precision=DOUBLE):
        kind = np.float32 if precision == SINGLE else np.float64
        return self._eval(subst or {}, kind)

    def _eval(self, subst, kind):
        if self in subst:
            return subst[self]._eval({}, kind)
        return self.apply(*[x._eval(subst, kind) for x in self._ops])


class Number(Expression):
    def __init__(self, value):
        self.value = float(value)
        super().__init__()

    def _value(self):
        return self.value

    def _eval(self, subst, kind):
        return kind(self.value)


class Name(Expression):
    def __init__(self, variable):
        self._variable = variable
        super().__init__()

    def _value(self):
        return self._variable

    def var(self):
        return self._variable

    def _eval(self, subst, kind):
        if self in subst:
            return subst[self]._eval({}, kind)
        return self._variable.rhs()._eval(subst, kind)


class Derivative(Expression):
    def var(self):
        return self._ops[0].var()

    def references(self):
        return {self}

    def walk(self):
        yield self


class Condition(Expression):
    pass


def _node(name, fn, base=Expression):
    return type(name, (base,), {'apply': staticmethod(fn)})


PrefixPlus = _node('PrefixPlus', lambda a: a)
PrefixMinus = _node('PrefixMinus', lambda a: -a)
Plus = _node('Plus', lambda a, b: a + b)
Minus = _node('Minus', lambda a, b: a - b)
Multiply = _node('Multiply', lambda a, b: a * b)
Divide = _node('Divide', lambda a, b: a / b)
Quotient = _node('Quotient', lambda a, b: a // b)
Remainder = _node('Remainder', lambda a, b: a % b)
Power = _node('Power', lambda a, b: a ** b)
Exp = _node('Exp', np.exp)
Log10 = _node('Log10', np.log10)
Log = _node('Log', lambda a, *b: np.log(a) / np.log(b[0]) if b
            else np.log(a))
Sqrt = _node('Sqrt', np.sqrt)
Sin, Cos, Tan = (_node(n.title(), getattr(np, n)) for n in ('sin', 'cos',
                                                            'tan'))
ASin = _node('ASin', np.arcsin)
ACos = _node('ACos', np.arccos)
ATan = _node('ATan', np.arctan)
Floor = _node('Floor', np.floor)
Ceil = _node('Ceil', np.ceil)
Abs = _node('Abs', np.abs)
MoreEqual = _node('MoreEqual', lambda a, b: a >= b, Condition)
LessEqual = _node('LessEqual', lambda a, b: a <= b, Condition)
More = _node('More', lambda a, b: a > b, Condition)
Less = _node('Less', lambda a, b: a < b, Condition)


class If(Expression):
    apply = staticmethod(lambda i, t, e: t if i else e)

    def __init__(self, i, t, e):
        self._i, self._t, self._e = i, t, e
        super().__init__(i, t, e)


class Piecewise(Expression):
    def __init__(self, *ops):
        self._i, self._e = list(ops[:-1:2]), list(ops[1::2]) + [ops[-1]]
        super().__init__(*ops)

    @staticmethod
    def apply(*v):
        for i in range(0, len(v) - 1, 2):
            if v[i]:
                return v[i + 1]
        return v[-1]


_CALLS = {'exp': Exp, 'log': Log, 'sqrt': Sqrt, 'cos': Cos, 'acos': ACos,
          'abs': Abs, 'where': If}
_BIN = {ast.Add: Plus, ast.Sub: Minus, ast.Mult: Multiply, ast.Div: Divide,
        ast.Pow: Power}
_CMP = {ast.GtE: MoreEqual, ast.LtE: LessEqual, ast.Gt: More, ast.Lt: Less}


def _tree(node, var):
    """An expression from Python's parse of its text."""
    if isinstance(node, ast.Constant):
        return Number(node.value)
    if isinstance(node, ast.Attribute):
        return Name(var(node.value.id + '.' + node.attr))
    if isinstance(node, ast.UnaryOp):
        x = _tree(node.operand, var)
        return Number(-x.value) if isinstance(x, Number) else PrefixMinus(x)
    if isinstance(node, ast.BinOp):
        return _BIN[type(node.op)](_tree(node.left, var),
                                   _tree(node.right, var))
    if isinstance(node, ast.Compare):
        return _CMP[type(node.ops[0])](_tree(node.left, var),
                                       _tree(node.comparators[0], var))
    return _CALLS[node.func.id](*[_tree(a, var) for a in node.args])


class Unit:
    def __init__(self, text):
        self.text = text

    def exponents(self):
        return self.text


class Variable:
    def __init__(self, qname):
        self._qname = qname
        self._rhs = Number(0)
        self._initial = None
        self._index = None
        self._unit = None
        self._bind = None
        self._uses = ()
        self.gate = None         # (inf, tau) variables
        self.constant = False

    def qname(self):
        return self._qname

    def uname(self):
        return self._qname.replace('.', '_')

    def rhs(self):
        return self._rhs

    def lhs(self):
        return Derivative(Name(self)) if self.is_state() else Name(self)

    def index(self):
        return self._index

    def unit(self):
        return self._unit

    def binding(self):
        return self._bind

    def initial_value(self, as_float=True):
        return self._initial

    def eval(self):
        return float(self._rhs.eval())

    def is_state(self):
        return self._index is not None

    def is_bound(self):
        return self._bind is not None

    def is_constant(self):
        return self.constant

    def is_literal(self):
        return isinstance(self._rhs, Number) and not self.is_state()

    def is_intermediary(self):
        return not (self.constant or self.is_state())


Equation = namedtuple('Equation', 'lhs rhs')


class Group:
    def __init__(self, variables):
        self._variables = variables

    def equations(self, const=None):
        for v in self._variables:
            if const is None or bool(const) == v.constant:
                yield Equation(v.lhs(), v.rhs())


class Model:
    """Equations parsed from text, with the queries the package makes."""
    def __init__(self, name, text):
        self._name, self._text = name, text
        self._vars = OrderedDict()
        self._states = []
        gates = []
        for line in text.strip().splitlines():
            line = line.strip()
            if not line:
                continue
            if ':=' in line:
                n, b = [x.strip() for x in line.split(':=')]
                self._var(n)._bind = b
                continue
            left, right = [x.strip() for x in line.split('=', 1)] \
                if not line.startswith('where') else (None, None)
            if '(' not in left:
                self._var(left)._rhs = self._parse(right)
                continue
            kind, n = left[:-1].split('(')
            right, init = [x.strip() for x in right.split('@')]
            v = self._var(n)
            v._index = len(self._states)
            self._states.append(v)
            if '[' in init:
                init, unit = init.split('[')
                v._unit = Unit(unit.strip(' ]'))
            v._initial = float(init)
            if kind == 'gate':
                inf, tau = [self._var(x.strip()) for x in right.split(',')]
                gates.append((v, inf, tau))
                v._rhs = Divide(Minus(Name(inf), Name(v)), Name(tau))
                v.gate = (inf, tau)
            else:
                v._rhs = self._parse(right)
        self._order = self._solve()

    def _var(self, name):
        if name not in self._vars:
            self._vars[name] = Variable(name)
        return self._vars[name]

    def _parse(self, text):
        # ("if" is a word of Python: a variable may still be called that)
        text = text.replace('.if ', '.if_ ').replace('.in ', '.in_ ')
        node = ast.parse(text.strip(), mode='eval').body
        return _tree(node, lambda n: self._var(n.rstrip('_')))

    def _solve(self):
        """Variables so that each follows what it refers to."""
        order, seen = [], set()

        def visit(v, path=()):
            if v in seen:
                return
            if v in path:
                raise ValueError('cyclic equations at ' + v.qname())
            refs = sorted((r.var() for r in v.rhs().references()),
                          key=lambda x: x.qname())
            for r in refs:
                if not r.is_state():
                    visit(r, path + (v,))
            v.constant = not (v.is_state() or v.is_bound()) and all(
                r.constant for r in refs)
            seen.add(v)
            order.append(v)
        for v in self._vars.values():
            visit(v)
        return order

    def clone(self):
        return Model(self._name, self._text)

    def name(self):
        return self._name

    def code(self):
        return self._text

    def is_valid(self):
        return True

    def has_interdependent_components(self):
        return False

    def create_unique_names(self):
        pass

    def get(self, name):
        if isinstance(name, Variable):
            name = name.qname()
        return self._vars[name]

    def label(self, name):
        return self._vars.get('membrane.V')

    def binding(self, name):
        for v in self._vars.values():
            if v._bind == name:
                return v

    def time(self):
        return self.binding('time')

    def states(self):
        return iter(self._states)

    def count_states(self):
        return len(self._states)

    def initial_values(self, as_float=True):
        return [v._initial for v in self._states]

    def solvable_order(self):
        return OrderedDict(cell=Group(self._order))


class Writer:
    """Writes expressions as C text; kinds have a method ``_ex_<kind>``."""
    def __init__(self):
        self._lhs = None

    def set_lhs_function(self, f):
        self._lhs = f

    def ex(self, e):
        if isinstance(e, (Name, Derivative)):
            return self._lhs(e)
        kind = type(e).__name__
        if kind in self._INFIX:
            return f'({self.ex(e[0])} {self._INFIX[kind]} {self.ex(e[1])})'
        return getattr(self, '_ex_' + self._KINDS.get(kind, kind.lower()))(e)

    _INFIX = {'Plus': '+', 'Minus': '-', 'Multiply': '*', 'MoreEqual': '>=',
              'LessEqual': '<=', 'More': '>', 'Less': '<'}
    _KINDS = {'PrefixMinus': 'minus', 'PrefixPlus': 'plus'}

    def _ex_minus(self, e):
        return f'(-{self.ex(e[0])})'

    def _ex_plus(self, e):
        return self.ex(e[0])

    def _ex_divide(self, e):
        return f'({self.ex(e[0])} / {self.ex(e[1])})'

    def _ex_function(self, e, name):
        return name + '(' + ', '.join(self.ex(x) for x in e) + ')'

    def _ex_if(self, e):
        return f'({self.ex(e._i)} ? {self.ex(e._t)} : {self.ex(e._e)})'

    def _ex_piecewise(self, e):
        s = self.ex(e._e[-1])
        for c, x in list(zip(e._i, e._e))[::-1]:
            s = f'({self.ex(c)} ? {self.ex(x)} : {s})'
        return s


class DataLog(OrderedDict):
    def has_nan(self):
        return any(len(v) and math.isnan(v[-1]) for v in self.values())


def split_key(key):
    """('3.4.', 'membrane.V') for '3.4.membrane.V'."""
    parts = key.rsplit('.', 2)
    return (parts[0] + '.' if len(parts) > 2 else '', '.'.join(parts[-2:]))


def prepare_log(log, model, dims=None, global_vars=None, if_empty=0,
                allowed_classes=0, precision=DOUBLE):
    """An empty log of the named variables; one without cell indices stands
    for all cells."""
    import array
    out = DataLog()
    one = array.array('d' if precision == DOUBLE else 'f')
    for name in log if isinstance(log, (list, tuple)) else []:
        if split_key(name)[0] or name in global_vars:
            out[name] = one[:]
        elif len(dims) == 1:
            out.update(('%d.%s' % (x, name), one[:]) for x in range(dims[0]))
        else:
            out.update(('%d.%d.%s' % (x, y, name), one[:])
                       for y in range(dims[1]) for x in range(dims[0]))
    return out


class Event:
    def __init__(self, *v):
        self._v = v

    def level(self):
        return self._v[0]

    def start(self):
        return self._v[1]

    def duration(self):
        return self._v[2]

    def period(self):
        return self._v[3]

    def multiplier(self):
        return self._v[4]


class Protocol:
    """One block train."""
    def __init__(self, *event):
        self._event = event

    def clone(self):
        return Protocol(*self._event)

    def events(self):
        return [Event(*self._event)]


def _bindings(model, inputs):
    return {v: inputs[v._bind] for v in model._vars.values()
            if v._bind in inputs}


def _register():
    """Makes the above importable under the name the package imports."""
    m = types.ModuleType('myokit')
    for name, value in list(globals().items()):
        if isinstance(value, type) and value.__module__ in (__name__, 'abc'):
            setattr(m, name, value)
    m.SINGLE_PRECISION, m.DOUBLE_PRECISION = SINGLE, DOUBLE
    m.LOG_NONE, m.LOG_STATE, m.LOG_BOUND, m.LOG_INTER = 0, 1, 2, 4
    m.split_key, m.prepare_log = split_key, prepare_log
    m.parse_unit = Unit
    m._prepare_bindings = _bindings
    m._simulation_progress = None
    for name in ('ProgressReporter', 'FiberTissueSimulation'):
        setattr(m, name, type(name, (), {}))
    for name in ('SimulationCancelledError', 'FindNanError',
                 'SimulationError', 'NumericalError'):
        setattr(m, name, type(name, (Exception,), {}))
    hh = types.ModuleType('myokit.lib.hh')
    hh.convert_hh_states_to_inf_tau_form = lambda model, vm: model.clone()
    hh.get_inf_and_tau = lambda state, vm: state.gate
    ansic = types.ModuleType('myokit.formats.ansic')
    ansic.CBasedExpressionWriter = Writer
    m.lib = types.ModuleType('myokit.lib')
    m.formats = types.ModuleType('myokit.formats')
    m.lib.hh, m.formats.ansic = hh, ansic
    m.__path__, m.lib.__path__, m.formats.__path__ = [], [], []
    for x in (m, m.lib, hh, m.formats, ansic):
        sys.modules[x.__name__] = x


_register()
import myokit_gb300 as mg  # noqa: E402
from myokit_gb300 import adjoint as mg_adjoint  # noqa: E402

MODELS = {name: Model(name, text) for name, text in TEXT.items()}
DT = 0.005
FIELDS = {'v48': ('ina.Gbar', 'ikr.Gbar', 'iks.Gbar', 'ical.G', 'ito.G',
                  'ik1.G'),
          'br': ('ina.g', 'isi.g')}

# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------


def case(name=None, kind='run', model='v48', nx=1, ny=0, precision=SINGLE,
         accumulate='', diffusion='grid', fields=0, steps=200, every=50,
         probes=0):
    """
    ``kind``: 'run' (logged), 'frames' (V frames of every cell on the
    device), 'batch' (uneven cables in one simulation) or 'adjoint' (loss
    and gradients). ``ny`` 0: a cable. A log point every ``every`` of
    ``steps`` steps; ``probes`` logged cells (0: all).
    """
    c = dict(kind=kind, model=model, nx=nx, ny=ny, precision=precision,
             accumulate=accumulate, diffusion=diffusion, fields=fields,
             steps=steps, every=every, probes=probes)
    if name:
        c['name'] = name
    return c


def listed():
    return [
        # A short cable between two log calls: latency of a whole call
        case('cable10-fp64', model='br', nx=10, precision=DOUBLE),
        # The classic strand in double precision, as Simulation1d runs it
        case('cable200-fp64', model='br', nx=200, precision=DOUBLE,
             steps=1000, every=200),
        # The same strand in single precision
        case('cable200-fp32', model='br', nx=200, steps=1000, every=200),
        # A small sheet of odd size, detailed model, some probes logged
        case('sheet61x47-fp32', nx=61, ny=47, steps=400, every=100,
             probes=32),
        # A sheet for accuracy studies: compensated sums, device frames
        case('sheet128-kahan', kind='frames', nx=128, ny=128,
             accumulate='kahan', steps=400, every=100),
        # The medium sheet: conductance fields, 256 probes
        case('sheet512-fp32', nx=512, ny=512, fields=2, steps=400,
             every=100, probes=256),
        # The large sheet: frames stay on the device
        case('sheet2048-kahan', kind='frames', nx=2048, ny=2048,
             accumulate='kahan', steps=1000, every=500),
        # Double precision reference solution of a sheet
        case('sheet256-fp64', nx=256, ny=256, precision=DOUBLE, steps=40,
             every=20, probes=64),
        # Uneven cables with parameter sets, one simulation
        case('cables-kahan', kind='batch', nx=96, accumulate='kahan',
             diffusion='hetero', fields=6, steps=400, every=100, probes=96),
        # An unstructured tissue: connections, one odd size
        case('graph4001-fp32', nx=4001, diffusion='conn', steps=400,
             every=100, probes=64),
        # Gradients for fitting conductance fields, single precision with
        # accumulated states in double
        case('adjoint96-fp32', kind='adjoint', nx=96, ny=96,
             accumulate='double', fields=2, steps=200, every=50, probes=32),
        # Gradients in double precision on a strand
        case('adjoint-cable64-fp64', kind='adjoint', nx=64, model='br',
             precision=DOUBLE, fields=1, steps=200, every=50, probes=8),
    ]


def _between(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    pick = rng.randrange(9)
    steps = rng.choice((100, 200, 400))
    if pick == 0:
        return case(model='br', nx=_between(rng, 8, 4000), precision=DOUBLE,
                    steps=steps, every=steps // 4)
    if pick == 1:
        return case(model=rng.choice(('br', 'v48')),
                    nx=_between(rng, 8, 20000), steps=steps,
                    every=steps // 2, probes=8)
    if pick == 2:
        return case(nx=_between(rng, 20, 700), ny=_between(rng, 20, 700),
                    steps=steps, every=steps // 4, probes=16,
                    fields=rng.choice((0, 2)))
    if pick == 3:
        n = _between(rng, 64, 1024)
        return case(kind='frames', nx=n, ny=n + rng.randrange(-9, 10),
                    accumulate=rng.choice(('kahan', 'double', '')),
                    steps=steps, every=steps // 4)
    if pick == 4:
        return case(nx=_between(rng, 12, 300), ny=_between(rng, 12, 300),
                    precision=DOUBLE, steps=20, every=10, probes=16)
    if pick == 5:
        return case(kind='batch', nx=_between(rng, 8, 200),
                    accumulate=rng.choice(('kahan', '')), diffusion='hetero',
                    fields=6, steps=steps, every=steps // 4,
                    probes=8)
    if pick == 6:
        return case(nx=_between(rng, 200, 20000), diffusion='conn',
                    steps=steps, every=steps // 2, probes=16,
                    precision=SINGLE)
    if pick == 7:
        # Sheet rows of whole warps; any number of rows
        return case(kind='adjoint', nx=32 * rng.randrange(1, 6),
                    ny=_between(rng, 24, 160), accumulate='double',
                    fields=2, steps=100, every=25, probes=16)
    return case(nx=_between(rng, 30, 300), ny=_between(rng, 30, 300),
                diffusion='hetero', steps=steps, every=steps // 4, probes=16,
                accumulate=rng.choice(('kahan', '')))


def _cells(c):
    if c['kind'] == 'batch':
        return int(_lengths(c).sum())
    return c['nx'] * max(c['ny'], 1)


def _lengths(c):
    """Cells of each cable of a batch: uneven, 50 to about 700."""
    k = np.arange(c['nx'])
    return 50 + (k * 271 + 13 * (k % 7)) % 653


def _problem(c, seed):
    """
    The inputs of a case, from the seed alone: per-cell initial states (the
    model's own, spread by a percent), conductance fields (lognormal
    spread), conductances of edges or connections, logged cells.
    """
    rng = np.random.default_rng(seed)
    n = _cells(c)
    m = MODELS[c['model']]
    p = types.SimpleNamespace(n=n, model=m)
    init = torch.tensor(m.initial_values(), dtype=torch.float64)
    z = torch.from_numpy(rng.standard_normal(n))
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    state = init.to(dev) * (1 + 0.005 * torch.tanh(z.to(dev)))[:, None]
    p.state = state.cpu().numpy().reshape(-1)
    p.fields = OrderedDict(
        (k, m.get(k).eval() * rng.lognormal(0, 0.2, n))
        for k in FIELDS[c['model']][:c['fields']])
    p.gx, p.gy = (9.0, None) if not c['ny'] else (10.0, 5.0)
    p.lengths = None
    if c['kind'] == 'batch':
        p.lengths = _lengths(c)
        p.g = rng.uniform(6, 12, len(p.lengths))
        p.fields = OrderedDict(
            (k, m.get(k).eval() * rng.lognormal(0, 0.2, len(p.lengths)))
            for k in FIELDS[c['model']][:c['fields']])
    elif c['diffusion'] == 'hetero':
        p.gx = rng.uniform(5, 12, (c['ny'], c['nx'] - 1))
        p.gy = rng.uniform(3, 8, (c['ny'] - 1, c['nx']))
    elif c['diffusion'] == 'conn':
        # A strand with side links, as an unstructured mesh numbers them
        i = np.arange(n - 1)
        far = np.arange(0, n - 40, 3)
        a = np.concatenate([i, far])
        b = np.concatenate([i + 1, far + 2 + far % 37])
        p.conn = list(zip(a.tolist(), b.tolist(),
                          rng.uniform(3, 9, len(a)).tolist()))
    cells = np.arange(n) if not c['probes'] else np.sort(
        rng.choice(n, min(c['probes'], n), replace=False))
    p.probes = cells
    p.paced = np.zeros(n, dtype=bool)
    if c['kind'] == 'batch':
        p.paced[:] = np.concatenate(
            [np.arange(k) < 5 for k in p.lengths])
    elif c['ny']:
        p.paced[:] = np.arange(n) % c['nx'] < 4
    else:
        p.paced[:5] = True
    p.target = rng.normal(-80, 5, (-(-c['steps'] // c['every']), len(cells)))
    return p


def prepare(case, seed):
    c = case
    p = _problem(c, seed)
    m = p.model
    kw = dict(precision=c['precision'], rl=c['model'] == 'v48',
              accumulate=c['accumulate'] or None)
    protocol = Protocol(1, 0, 2, 1000, 0)
    if c['kind'] == 'batch':
        s = mg.CableBatch(m, p.lengths, protocol, conductance=p.g,
                          paced_cells=5, fields=p.fields, **kw).sim
    else:
        s = mg.SimulationCUDA(
            m, protocol, ncells=(c['nx'], c['ny']) if c['ny'] else c['nx'],
            **kw)
        if c['diffusion'] == 'hetero':
            s.set_conductance_field(p.gx, p.gy)
        elif c['diffusion'] == 'conn':
            s.set_connections(p.conn)
        elif c['ny']:
            s.set_conductance(p.gx, p.gy)
        else:
            s.set_conductance(p.gx)
        if c['ny']:
            s.set_paced_cells(4, c['ny'])
        else:
            s.set_paced_cells(5)
        for k, v in p.fields.items():
            s.set_field(k, v.reshape(c['ny'], c['nx']) if c['ny'] else v)
    s.set_step_size(DT)
    s.set_state(p.state)
    st = types.SimpleNamespace(case=c, sim=s, ms=c['steps'] * DT,
                               interval=c['every'] * DT)
    if c['kind'] == 'adjoint':
        at = [(int(i % c['nx']), int(i // c['nx'])) for i in p.probes] \
            if c['ny'] else [int(i) for i in p.probes]
        st.adj = mg_adjoint.TissueAdjoint(s, at)
        st.target = p.target
        real = torch.float32 if c['precision'] == SINGLE else torch.float64
        st.real = real
        st.g = torch.tensor([p.gx, p.gy] if c['ny'] else p.gx,
                            dtype=real, requires_grad=True)
        st.fields = [torch.tensor(
            v.reshape(c['ny'], c['nx']) if c['ny'] else v, dtype=real,
            requires_grad=True) for v in p.fields.values()]
        return st
    if c['ny']:
        st.keys = ['%d.%d.membrane.V' % (i % c['nx'], i // c['nx'])
                   for i in p.probes]
    else:
        st.keys = ['%d.membrane.V' % i for i in p.probes]
    st.log = ['engine.time'] + st.keys
    # Small tissues hand their state on, as a user's next run would start
    # from it elsewhere; of large ones the frames or probes are the result
    st.state = p.n <= 20000 and c['kind'] != 'frames'
    return st


def run(state):
    s, c = state.sim, state.case
    if c['kind'] == 'adjoint':
        state.g.grad = None
        for f in state.fields:
            f.grad = None
        loss = mg_adjoint.tissue_loss(
            state.adj, state.ms, state.target, state.g, state.fields,
            state.interval)
        loss.backward()
        return {'loss': loss.detach().to(state.real), 'g': state.g.grad,
                'fields': [f.grad for f in state.fields]}
    if c['kind'] == 'frames':
        t, v = s.run_frames(state.ms, state.interval)
        return {'v': v}
    d = s.run(state.ms, log=state.log, log_interval=state.interval)
    real = np.float32 if c['precision'] == SINGLE else np.float64
    out = {'v': np.array([d[k] for k in state.keys], dtype=real)}
    if state.state:
        out['state'] = s.state_array().astype(real, copy=False)
    return out


def work(case):
    c = case
    m = MODELS[c['model']]
    n, b = _cells(c), c['precision'] // 8
    rows = -(-c['steps'] // c['every'])
    count = 0
    for v in m._order:
        if not v.constant:
            count += sum(1 for x in v.rhs().walk()
                         if len(x) and not isinstance(x, Derivative))
    count += 4 * m.count_states() + 8
    out = n if c['kind'] == 'frames' else len(_log_cells(c, n))
    # The state in and out, fields in, logged values out
    nbytes = n * (2 * m.count_states() + c['fields']) * b + rows * out * b
    # The reverse sweep of an equation is at least as long as the equation
    flops = n * c['steps'] * count * (3 if c['kind'] == 'adjoint' else 1)
    return {'bytes': nbytes, 'flops': flops}


def _log_cells(c, n):
    return range(min(c['probes'], n) if c['probes'] else n)


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------


def _program(model, rl, fields):
    """
    One time step as a Python function of (states, V neighbours' current,
    pace, dt, fields), written out from the model's equations.
    """
    def name(v):
        return v.qname().replace('.', '_') + '_'

    class Text(Writer):
        _ex_exp = _ex_log = _ex_sqrt = _ex_cos = _ex_acos = _ex_abs = \
            lambda self, e: self._ex_function(e, type(e).__name__.lower())

        def _ex_number(self, e):
            return repr(e.value)

        def _ex_power(self, e):
            return f'({self.ex(e[0])} ** {self.ex(e[1])})'

        def _ex_if(self, e):
            return f'where({self.ex(e._i)}, {self.ex(e._t)}, {self.ex(e._e)})'

    w = Text()
    w.set_lhs_function(lambda x: ('d_' if isinstance(x, Derivative) else '')
                       + name(x.var()))
    lines = ['def step(x, idiff, pace, dt, fields):']
    for i, v in enumerate(model._states):
        lines.append(f'  {name(v)} = x[{i}]')
    for v in model._order:
        if v._bind:
            r = {'time': '0.0', 'pace': 'pace',
                 'diffusion_current': 'idiff'}[v._bind]
            lines.append(f'  {name(v)} = {r}')
        elif v.qname() in fields:
            lines.append(f'  {name(v)} = fields["{v.qname()}"]')
        elif v.is_state():
            if not (rl and v.gate):
                lines.append(f'  d_{name(v)} = {w.ex(v.rhs())}')
        else:
            lines.append(f'  {name(v)} = {w.ex(v.rhs())}')
    out = []
    for v in model._states:
        if rl and v.gate:
            i, t = name(v.gate[0]), name(v.gate[1])
            out.append(f'{i} - ({i} - {name(v)}) * exp(-dt / {t})')
        else:
            out.append(f'{name(v)} + dt * d_{name(v)}')
    lines.append('  return [' + ', '.join(out) + ']')

    def lift(f):
        def g(x):
            return f(x) if torch.is_tensor(x) else float(
                f(torch.tensor(x, dtype=torch.float64)))
        return g

    def where(c, a, b):
        if not torch.is_tensor(c):
            return a if c else b
        a, b = [x if torch.is_tensor(x) else torch.full_like(
            c, x, dtype=torch.float64) for x in (a, b)]
        return torch.where(c, a, b)
    space = {k: lift(getattr(torch, k))
             for k in ('exp', 'log', 'sqrt', 'cos', 'acos', 'abs')}
    space['where'] = where
    exec('\n'.join(lines), space)
    return space['step']


def exact(case, seed):
    c = case
    n, steps = _cells(c), c['steps']
    if n * steps > 3e8:
        return None
    p = _problem(c, seed)
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    rl = c['model'] == 'v48'
    step = _program(p.model, rl, set(p.fields))
    ns = p.model.count_states()

    def tensor(a):
        return torch.as_tensor(np.asarray(a, dtype=float), device=dev)
    fields = {k: tensor(np.repeat(v, p.lengths) if p.lengths is not None
                        else v) for k, v in p.fields.items()}
    x0 = tensor(p.state).reshape(n, ns).T.contiguous()
    paced = tensor(p.paced.astype(float))
    iv = p.model.get('membrane.V').index()
    ny, nx = max(c['ny'], 1), n // max(c['ny'], 1)
    conn = gx = gy = None
    if c['diffusion'] == 'conn':
        conn = [torch.tensor([e[k] for e in p.conn], device=dev)
                for k in (0, 1)] + [tensor([e[2] for e in p.conn])]
    elif c['kind'] == 'batch':
        g = np.repeat(p.g, p.lengths)[:-1]
        g[np.cumsum(p.lengths)[:-1] - 1] = 0
        gx = tensor(g).reshape(1, -1)
    elif c['diffusion'] == 'hetero':
        gx, gy = tensor(p.gx), tensor(p.gy)
    else:
        gx, gy = tensor(p.gx), tensor(p.gy if p.gy is not None else 0.0)

    def current(v, gx, gy):
        if conn is not None:
            i = conn[2] * (v[conn[0]] - v[conn[1]])
            return torch.zeros_like(v).index_add(0, conn[0], i).index_add(
                0, conn[1], -i)
        v = v.reshape(ny, nx)
        dx = gx * (v[:, :-1] - v[:, 1:])
        i = torch.nn.functional.pad(dx, (0, 1)) - torch.nn.functional.pad(
            dx, (1, 0))
        if ny > 1:
            dy = gy * (v[:-1] - v[1:])
            i = i + torch.nn.functional.pad(
                dy, (0, 0, 0, 1)) - torch.nn.functional.pad(dy, (0, 0, 1, 0))
        return i.reshape(-1)

    def pace(k):
        return 1.0 if (k + 0.5) * DT < 2 else 0.0

    if c['kind'] == 'adjoint':
        return _exact_gradient(c, p, step, current, x0, fields, gx, gy,
                               paced, pace, iv, dev)
    x = x0.clone()
    level = torch.zeros((), dtype=torch.float64, device=dev)

    def advance():
        y = step(list(x), current(x[iv], gx, gy), level * paced, DT, fields)
        for i, v in enumerate(y):
            x[i].copy_(v)
    graph = None
    if dev == 'cuda':
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            advance()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            advance()
        x.copy_(x0)
    at = torch.as_tensor(p.probes, device=dev)
    rows = []
    for k in range(steps):
        if k % c['every'] == 0:
            rows.append(x[iv].clone() if c['kind'] == 'frames'
                        else x[iv][at].clone())
        level.fill_(pace(k))
        graph.replay() if graph is not None else advance()
    v = torch.stack(rows)
    if c['kind'] == 'frames':
        return {'v': v.reshape((len(rows), ny, nx) if c['ny']
                               else (len(rows), nx)).cpu().numpy()}
    out = {'v': v.T.cpu().numpy()}
    if n <= 20000:
        out['state'] = x.T.contiguous().cpu().numpy().reshape(-1)
    return out


def _exact_gradient(c, p, step, current, x0, fields, gx, gy, paced, pace, iv,
                    dev):
    """Loss and gradients, one step's derivatives at a time in reverse."""
    at = torch.as_tensor(p.probes, device=dev)
    target = torch.as_tensor(p.target, device=dev)
    fields = {k: v.requires_grad_() for k, v in fields.items()}
    gx = gx.clone().requires_grad_()
    gy = gy.clone().requires_grad_()
    leaves = list(fields.values()) + [gx, gy]

    def advance(x, k):
        return torch.stack(step(list(x), current(x[iv], gx, gy),
                                pace(k) * paced, DT, fields))
    xs = [x0]
    with torch.no_grad():
        for k in range(c['steps']):
            xs.append(advance(xs[-1], k))
    loss = 0.0
    lam = torch.zeros_like(x0)
    sums = [torch.zeros_like(v) for v in leaves]
    for k in range(c['steps'] - 1, -1, -1):
        x = xs[k].detach().requires_grad_()
        y = advance(x, k)
        got = torch.autograd.grad(y, [x] + leaves, lam, allow_unused=True)
        lam = got[0].clone()
        sums = [a if b is None else a + b for a, b in zip(sums, got[1:])]
        if k % c['every'] == 0:
            d = xs[k][iv][at] - target[k // c['every']]
            loss = loss + (d * d).sum()
            lam[iv, at] += 2 * d
    g = torch.stack(sums[-2:]) if c['ny'] else sums[-2]
    shape = (c['ny'], c['nx']) if c['ny'] else (c['nx'],)
    return {'loss': loss.cpu().numpy().reshape(()),
            'g': g.cpu().numpy(),
            'fields': [v.reshape(shape).cpu().numpy() for v in sums[:-2]]}
