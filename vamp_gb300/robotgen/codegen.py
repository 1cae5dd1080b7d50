"""Straight-line forward-kinematics + collision-schedule generator.

Input: a robot model JSON (vamp_gb300/robots/<robot>.json, written by extract.py).
Output:
  * vamp_gb300/csrc/robots/<robot>.cuh  - CUDA device code for sm_103a: FP32 FK of every sphere and
    the robot's fkcc check schedule, written against a small context interface (see
    vamp_gb300/csrc/vg_check.cuh);
  * oracle/port/robots/<robot>.h        - C code for the CPU oracle: the same FP32 FK (bit-identical
    operation sequence), an FP64 FK for centre tolerances and distance-to-contact, and the check
    schedule as tables.

Design.  Each movable joint gets one frame (R, t) in registers.  Links attached by fixed joints
share their moving ancestor's frame; their spheres are re-expressed in that frame at generation
time (float64, then rounded once to float32).  A frame is the parent frame times a constant
transform times the joint motion, with exact zeros and ones folded out, so an axis-aligned joint
costs 12 multiply-adds.  Every floating-point operation is emitted explicitly (fused multiply-add,
multiply, add) so that the CUDA and C versions round identically: the GPU kernels and the CPU
oracle compute bit-identical sphere centres.

The reference's generated kernels compute the same kinematics with a different operation order
(src/impl/vamp/robots/panda.hh:5229-5627), so centres agree with the reference to a few ulp, not
bit for bit; the FP64 FK bounds that difference.
"""
from __future__ import annotations

import argparse
import json
import re
import math
import os
from pathlib import Path

import numpy as np

from .urdf import axis_rotation, rpy_matrix

ROOT = Path(__file__).resolve().parents[2]
MODELS = ROOT / "vamp_gb300" / "robots"
CUDA_OUT = ROOT / "vamp_gb300" / "csrc" / "robots"
C_OUT = ROOT / "oracle" / "port" / "robots"


def f32(v: float) -> float:
    return float(np.float32(v))


def lit32(v: float) -> str:
    v = f32(v)
    if v == 0.0:
        return "0.0f"
    r = repr(v)
    if "e" not in r and "." not in r:
        r += ".0"
    return r + "f"


def lit64(v: float) -> str:
    r = repr(float(v))
    if "e" not in r and "." not in r and "inf" not in r and "nan" not in r:
        r += ".0"
    return r


class Emitter:
    """Emits explicit arithmetic for one target.

    A value is a Python float (a constant, already rounded for the target), a variable name, or a
    variable name prefixed with '-' (its negation, folded into the operation that uses it).
    `snap` folds constants within `snap` of 0 or +-1 to exact values (float targets only).
    """

    def __init__(self, target: str, snap: float):
        self.target = target  # "cuda" | "c32" | "c64"
        self.snap = snap
        self.lines: list[str] = []
        self.n = 0
        self.ty = "double" if target == "c64" else "float"
        self.flops = 0  # floating-point operations emitted (a fused multiply-add counts 2)

    def const(self, v: float) -> float:
        if self.snap:
            if abs(v) < self.snap:
                v = 0.0
            elif abs(v - 1.0) < self.snap:
                v = 1.0
            elif abs(v + 1.0) < self.snap:
                v = -1.0
        return float(v) if self.target == "c64" else f32(v)

    def lit(self, v) -> str:
        return lit64(v) if self.target == "c64" else lit32(v)

    def ref(self, v) -> str:
        if isinstance(v, float):
            return self.lit(v)
        return f"(-{v[1:]})" if v.startswith("-") else v

    def _fma(self, a, b, c) -> str:
        self.flops += 2
        a, b, c = self.ref(a), self.ref(b), self.ref(c)
        if self.target == "cuda":
            return f"__fmaf_rn({a}, {b}, {c})"
        return f"{'fma' if self.target == 'c64' else 'fmaf'}({a}, {b}, {c})"

    def _mul(self, a, b) -> str:
        self.flops += 1
        a, b = self.ref(a), self.ref(b)
        return f"__fmul_rn({a}, {b})" if self.target == "cuda" else f"({a} * {b})"

    def _add(self, a, b) -> str:
        self.flops += 1
        a, b = self.ref(a), self.ref(b)
        return f"__fadd_rn({a}, {b})" if self.target == "cuda" else f"({a} + {b})"

    def assign(self, expr: str, name: str | None = None) -> str:
        if name is None:
            name = f"_v{self.n}"
            self.n += 1
        self.lines.append(f"const {self.ty} {name} = {expr};")
        return name

    @staticmethod
    def _neg(v):
        if isinstance(v, float):
            return -v
        return v[1:] if v.startswith("-") else "-" + v

    def lincomb(self, terms, const=0.0, name=None):
        """Emit const + sum(coef * a * b) for terms (coef, a, b|None).  Returns a value.

        Order: the constant (if non-zero) starts the accumulator, then each product is fused
        in turn; a lone product starts with a multiply.
        """
        prods = []
        c0 = const
        for coef, a, b in terms:
            k = coef
            vs = []
            for x in (a, b):
                if x is None:
                    continue
                if isinstance(x, float):
                    k *= x
                else:
                    if x.startswith("-"):
                        k = -k
                        x = x[1:]
                    vs.append(x)
            k = self.const(k)
            if k == 0.0:
                continue
            if not vs:
                c0 += k
                continue
            prods.append((k, vs))
        c0 = self.const(c0)
        if not prods:
            return c0
        # start the accumulator from a bare variable when there is one (saves an operation)
        if c0 == 0.0:
            for i, (k, vs) in enumerate(prods):
                if len(vs) == 1 and k in (1.0, -1.0):
                    prods.insert(0, prods.pop(i))
                    break

        def operand(k, vs):
            # returns (x, y) with x * y == k * prod(vs); may emit one multiply for 3-factor terms
            if len(vs) == 1:
                if k == 1.0:
                    return None, vs[0]
                if k == -1.0:
                    return None, "-" + vs[0]
                return k, vs[0]
            if k == 1.0:
                return vs[0], vs[1]
            if k == -1.0:
                return "-" + vs[0], vs[1]
            t = self.assign(self._mul(k, vs[0]))
            return t, vs[1]

        if c0 != 0.0:
            acc = c0
            rest = prods
        else:
            x, y = operand(*prods[0])
            if x is None:
                acc = y
            else:
                acc = self.assign(self._mul(x, y))
            rest = prods[1:]
        for k, vs in rest:
            x, y = operand(k, vs)
            if x is None:
                if y.startswith("-"):
                    acc = self.assign(self._add(acc, y))  # acc + (-y)
                else:
                    acc = self.assign(self._add(acc, y))
            else:
                acc = self.assign(self._fma(x, y, acc))
        if name is not None and isinstance(acc, str):
            last = self.lines[-1] if self.lines else ""
            if acc.startswith("_v") and last.startswith(f"const {self.ty} {acc} ="):
                self.lines[-1] = last.replace(f"const {self.ty} {acc} =", f"const {self.ty} {name} =", 1)
                return name
            return self.assign(self.ref(acc), name)
        return acc


# --------------------------------------------------------------------------------------------
# kinematic structure


class Kin:
    """Frames of a robot: one per movable joint plus the root, with fixed links folded."""

    def __init__(self, model: dict):
        self.m = model
        joints = model["joints"]
        self.by_child = {j["child"]: j for j in joints}
        self.jindex = {n: i for i, n in enumerate(model["joint_names"])}
        # frame of every link: (frame_id, constant 4x4 from frame to link)
        self.link_frame = {model["root"]: ("root", np.eye(4))}
        self.frames = []  # movable frames in topological order: dict
        pending = list(joints)
        while pending:
            rest = []
            for j in pending:
                if j["parent"] not in self.link_frame:
                    rest.append(j)
                    continue
                fid, C = self.link_frame[j["parent"]]
                O = np.eye(4)
                O[:3, :3] = rpy_matrix(j["rpy"])
                O[:3, 3] = j["xyz"]
                K = C @ O
                if j["type"] == "fixed" or j["name"] not in self.jindex:
                    if j["type"] != "fixed":
                        # a movable joint the configuration does not drive: hold it at zero
                        pass
                    self.link_frame[j["child"]] = (fid, K)
                else:
                    name = f"F{len(self.frames)}"
                    self.frames.append(
                        {
                            "id": name,
                            "parent": fid,
                            "K": K,
                            "axis": np.asarray(j["axis"], dtype=np.float64),
                            "type": j["type"],
                            "q": self.jindex[j["name"]],
                            "joint": j["name"],
                        }
                    )
                    self.link_frame[j["child"]] = (name, np.eye(4))
            assert len(rest) < len(pending)
            pending = rest

    def sphere_in_frame(self, link: str, p) -> tuple:
        fid, C = self.link_frame[link]
        v = C @ np.array([p[0], p[1], p[2], 1.0])
        return fid, v[:3]


def emit_frames(kin: Kin, em: Emitter, qname="q", sc_fn=None):
    """Emit every movable frame; returns {frame_id: (R, t)} with values (floats or names)."""
    frames = {"root": ([[1.0, 0.0, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]], [0.0, 0.0, 0.0])}
    for f in kin.frames:
        Rp, tp = frames[f["parent"]]
        K = f["K"]
        fid = f["id"]
        # fixed part: M = Rp @ K_R, t0 = tp + Rp @ K_t
        t0 = [em.lincomb([(float(K[k, 3]), Rp[r][k], None) for k in range(3)] + [(1.0, tp[r], None)]) for r in range(3)]
        M = [[em.lincomb([(float(K[k, c]), Rp[r][k], None) for k in range(3)]) for c in range(3)] for r in range(3)]
        axis = f["axis"] / np.linalg.norm(f["axis"])
        qv = f"{qname}[{f['q']}]"
        if f["type"] in ("revolute", "continuous"):
            s, c = f"{fid}_s", f"{fid}_c"
            em.lines.append(sc_fn(qv, s, c))
            # joint rotation (Rodrigues): Rj = c (I - a a^T) + s [a]x + a a^T
            kx = np.array([[0, -axis[2], axis[1]], [axis[2], 0, -axis[0]], [-axis[1], axis[0], 0]])
            aa = np.outer(axis, axis)
            R = []
            for r in range(3):
                row = []
                for cc in range(3):
                    terms = []
                    for k in range(3):
                        terms.append(((1.0 if k == cc else 0.0) - aa[k, cc], M[r][k], c))
                        terms.append((kx[k, cc], M[r][k], s))
                        terms.append((aa[k, cc], M[r][k], None))
                    row.append(em.lincomb(terms, 0.0, name=f"{fid}_r{r}{cc}"))
                R.append(row)
            t = [em.lincomb([(1.0, t0[r], None)], 0.0, name=f"{fid}_t{r}") for r in range(3)]
        elif f["type"] == "prismatic":
            R = M
            t = [
                em.lincomb(
                    [(1.0, t0[r], None)] + [(float(axis[k]), M[r][k], qv) for k in range(3)],
                    0.0,
                    name=f"{fid}_t{r}",
                )
                for r in range(3)
            ]
        else:
            raise ValueError(f["type"])
        frames[fid] = (R, t)
    return frames


def emit_centre(em: Emitter, frames, kin: Kin, link: str, p, prefix: str):
    """Centre of a sphere at offset p of `link`: t + R p, evaluated as t, then one fused
    multiply-add per column of R, for every coordinate.  The frame's entries are used as they
    are (constants are not folded into the chain), so a centre computed from frame values held in
    registers, in local memory or on the CPU rounds identically."""
    fid, v = kin.sphere_in_frame(link, p)
    return emit_point(em, frames[fid], v, prefix)


def emit_point(em: Emitter, frame, v, prefix: str):
    """A point at offset v of a frame (R, t), in emit_centre's order of operations."""
    R, t = frame
    out = []
    for r in range(3):
        acc = t[r]
        for k in range(3):
            acc = em.assign(em._fma(R[r][k], em.const(float(v[k])), acc))
        last = em.lines[-1]
        name = f"{prefix}{'xyz'[r]}"
        em.lines[-1] = last.replace(f"const {em.ty} {acc} =", f"const {em.ty} {name} =", 1)
        out.append(name)
    return out


def emit_ee_pose(em: Emitter, frames, kin: Kin, link: str):
    """Transform of `link` (the end effector, where fkcc_attach poses the attachment): its
    frame's R and t composed with the constant link offset, R row-major then t, each entry one
    lincomb (the same operation sequence as the frames themselves).  Returns 12 values."""
    fid, C = kin.link_frame[link]
    Rp, tp = frames[fid]
    R = [[em.lincomb([(float(C[k, c]), Rp[r][k], None) for k in range(3)]) for c in range(3)] for r in range(3)]
    t = [em.lincomb([(float(C[k, 3]), Rp[r][k], None) for k in range(3)] + [(1.0, tp[r], None)]) for r in range(3)]
    return [R[r][c] for r in range(3) for c in range(3)] + t


def attach_tables(model: dict, coarse_slot: dict):
    """Per robot link checked against an attachment (fkcc_attach, in the reference's order): its
    coarse slot and the range of its fine slots in the flat fine list."""
    rows, fine = [], []
    for c in model.get("attach_checks", []):
        rows.append((coarse_slot[c["link"]], len(fine), len(fine) + len(c["fine"])))
        fine += c["fine"]
    return rows, fine


# sin_ref + cos_ref of one joint angle: 24 + 25 floating-point operations (vg_check.cuh)
SINCOS_FLOPS = 49
# one sphere centre from its frame: 9 fused multiply-adds
CENTRE_FLOPS = 18


def fk_flops(model: dict) -> dict:
    """Floating-point operations of the generated FP32 kinematics for one configuration."""
    kin = Kin(model)
    em = Emitter("cuda", SNAP32)
    emit_frames(kin, em, "q", sc_fn=lambda x, s_, c: "")
    n_rev = sum(1 for f in kin.frames if f["type"] in ("revolute", "continuous"))
    slots, _ = slot_table(model)
    return {"frames": em.flops + SINCOS_FLOPS * n_rev, "centre": CENTRE_FLOPS, "slots": len(slots)}


def struct_name(name: str) -> str:
    return name[0].upper() + name[1:]


def slot_table(model: dict):
    """Slot order: fine spheres 0..n-1 (reference order), then one coarse sphere per env link."""
    slots = [(f["link"], f["p"], f["r"]) for f in model["fine_spheres"]]
    coarse_slot = {}
    for e in model["env_checks"]:
        link = e["link"]
        c = model["coarse_spheres"][link]
        coarse_slot[link] = len(slots)
        slots.append((link, c["p"], c["r"]))
    return slots, coarse_slot


# --------------------------------------------------------------------------------------------
# CUDA output


# FP32 constants this close to 0 or +-1 are folded to exact values: URDF angles such as
# 1.570796325 leave ~1e-9 residues that only cost operations (their effect is below 1e-8 m)
SNAP32 = 1e-7

def f32_down(v: float) -> float:
    """Largest float32 <= v (a conservative lower bound in FP32)."""
    x = np.float32(v)
    return float(x) if float(x) <= v else float(np.nextafter(x, np.float32(-np.inf)))


def f32_up(v: float) -> float:
    """Smallest float32 >= v."""
    x = np.float32(v)
    return float(x) if float(x) >= v else float(np.nextafter(x, np.float32(np.inf)))


BIG = 3.0e38  # an unbounded box side (joint values are finite)


def danger_boxes(model: dict, cull) -> list:
    """Per self check its two joint indices, whether it was analysed, and the union of its live
    pairs' boxes as FP32 bounds rounded outwards (unbounded if not analysed)."""
    checks = []
    for ci, e in enumerate(model["self_checks"]):
        bx = None if cull is None or "boxes" not in cull else cull["boxes"][ci]
        if not bx:
            checks.append(((0, 0, False), (-BIG, BIG, -BIG, BIG)))
            continue
        j = bx[0]["joints"]
        two = len(j) == 2
        jj = (j[0], j[1] if two else j[0])
        per = []
        for b in bx:
            lo1, hi1 = (b["lo"][1], b["hi"][1]) if two else (-BIG, BIG)
            per.append((f32_down(b["lo"][0]), f32_up(b["hi"][0]), f32_down(lo1) if two else -BIG, f32_up(hi1) if two else BIG))
        union = (min(p[0] for p in per), max(p[1] for p in per), min(p[2] for p in per), max(p[3] for p in per))
        checks.append(((jj[0], jj[1], True), union))
    return checks


# Resident 128-thread blocks per SM that the same-edge kernels are built for: five for the robots
# whose checks then stay in registers (102 a thread; 16,384 motions among 60 primitives, built for
# 4 -> 5 -> 6 blocks: Panda 302 -> 278 -> 299 us, UR5 396 -> 388 -> 401, Fetch 571 -> 492 -> 541);
# Baxter's stage leaves room for three (built for 4, with spills: 1,270 us; for 3: 1,224).
EDGE_BLOCKS = {"panda": 5, "ur5": 5, "fetch": 5, "baxter": 3}
CONTAIN_MARGIN = 1e-4  # metres between a link's fine spheres and its containing sphere
# A joint value beyond this (radians or metres) may leave frames that do not keep distances: the sine
# and the cosine each round the angle, so they stand for angles that differ by up to half a unit of
# its last place.  At 64 that is 4e-6 a joint, under 0.02 mm over seven joints and a group's half
# metre, a fifth of CONTAIN_MARGIN; at 10^6 it is 0.03, and containing spheres contain no more.
FAR_JOINT = 64.0
# Where such lanes are dealt with: between the lookups and their words, a branch that also keeps the
# compiler from drawing the lookups forward (16,384 Panda motions 295 -> 287 us, UR5 338 -> 336, Baxter
# equal), or, for the Fetch, whose states kernel then needs 114 registers and loses its fifth resident
# block (262,144 configurations 321 -> 352 us, 32,768 blocks 277 -> 321), after the words (324 and 279).
# Its motions take 421 or 425 us, 405 without the test.
FAR_LATE = {"fetch"}


def containing_radius(model: dict, kin, env_check: dict) -> float:
    """Largest |fine centre - coarse centre| + fine radius of a link, in float64."""
    slots, cslot = slot_table(model)
    link = env_check["link"]
    fc, pc = kin.sphere_in_frame(slots[cslot[link]][0], slots[cslot[link]][1])
    best = 0.0
    for f in env_check["fine"]:
        ff, pf = kin.sphere_in_frame(slots[f][0], slots[f][1])
        assert ff == fc, "a link's fine spheres and its coarse sphere share one frame"
        best = max(best, float(np.linalg.norm(np.asarray(pf, float) - np.asarray(pc, float))) + float(slots[f][2]))
    return best


def load_cull(name: str):
    """Live fine self pairs per self check (None: all live), from robots/<name>.cull.json."""
    path = MODELS / f"{name}.cull.json"
    if not path.exists():
        return None
    return json.loads(path.read_text())


def limits_code(model: dict, cull) -> list:
    """Lines setting ctx.in_limits: every active lane's configuration lies in the joint limits
    widened by the culling slack (the precondition for skipping culled self pairs)."""
    if cull is None:
        return ["ctx.in_limits = false;"]
    slack = cull["slack_rad"]
    lines = ["bool inl = true;"]
    for d, (m_, a_) in enumerate(zip(model["s_m"], model["s_a"])):
        lo = f32(a_ - slack)
        hi = f32(a_ + m_ + slack)
        lines.append(f"inl &= (q[{d}] >= {lit32(lo)}) & (q[{d}] <= {lit32(hi)});")
    lines.append("ctx.in_limits = __all_sync(vg::kFull, inl || !((ctx.alive >> (threadIdx.x & 31)) & 1u));")
    return lines


def _aliases(lines) -> dict:
    """name -> (name, sign) for the emitted copies `const float A = B;` and `const float A = (-B);`."""
    out = {}
    for line in lines:
        m = re.fullmatch(r"const float (\w+) = (?:\(-(\w+)\)|(\w+));", line.strip())
        if m:
            out[m.group(1)] = (m.group(2), -1) if m.group(2) else (m.group(3), 1)
    return out


def stage_layout(model: dict, kin, cull) -> dict:
    """The shared-memory stage, per thread: each distinct non-constant value among the entries of
    the frames the checks use (an entry that is a copy of another takes that value's slot), then
    the joint values the danger boxes test."""
    slots, _ = slot_table(model)
    em = Emitter("cuda", SNAP32)
    fr = emit_frames(kin, em, "q", sc_fn=lambda x, s_, c: "")
    alias = _aliases(em.lines)

    def resolve(name):
        sign = 1
        while name in alias:
            name, sg = alias[name]
            sign *= sg
        return name, sign

    frames, fslots, fconsts, values = {}, [], [], {}
    for e in model["env_checks"]:
        fid = kin.sphere_in_frame(slots[e["fine"][0]][0], slots[e["fine"][0]][1])[0]
        if fid in frames:
            continue
        frames[fid] = len(fslots)
        R, t = fr[fid]
        row_s, row_c = [], []
        for v in [R[r][c] for r in range(3) for c in range(3)] + list(t):
            if isinstance(v, float):
                row_s.append(-1)
                row_c.append(v)
                continue
            neg = v.startswith("-")
            base, sign = resolve(v[1:] if neg else v)
            sign = -sign if neg else sign
            # a negated copy gets its own slot: decoding a sign per entry costs more in the fine
            # checks than the slot saves
            key = base if sign > 0 else "-" + base
            if key not in values:
                values[key] = len(values)
            row_s.append(values[key])
            row_c.append(0.0)
        fslots.append(row_s)
        fconsts.append(row_c)
    checks = danger_boxes(model, cull)
    joints = sorted({j for (j0, j1, found), _ in checks if found for j in (j0, j1)})
    return {"frames": frames, "slots": fslots, "consts": fconsts, "values": list(values),
            "joints": joints, "joint_pos": {j: i for i, j in enumerate(joints)},
            "q0": len(values), "total": len(values) + len(joints)}


def enclosing_sphere(spheres) -> tuple:
    """A sphere that contains the given ones ((x, y, z), r), near the smallest: Badoiu and
    Clarkson's iteration (move towards the farthest by 1 / (i + 1)), the radius then rounded up
    with CONTAIN_MARGIN to spare."""
    c = [sum(p[k] for p, _ in spheres) / len(spheres) for k in range(3)]

    def far(q):
        return max((math.sqrt(sum((p[k] - q[k]) ** 2 for k in range(3))) + r, p) for p, r in spheres)

    for i in range(1, 400):
        d, p = far(c)
        n = math.sqrt(sum((p[k] - c[k]) ** 2 for k in range(3)))
        if n == 0.0:
            break
        # towards the farthest point of the farthest sphere
        c = [c[k] + (p[k] - c[k]) / n * d / (i + 1) * 0.5 for k in range(3)]
    best = c
    return best, f32_up(far(best)[0] + CONTAIN_MARGIN)


def link_groups(model: dict, kin) -> dict:
    """The environment-checked links grouped by the frame their coarse spheres are fixed in: a
    rigid group's coarse spheres lie in one sphere of that frame, which stands for all of them
    until something comes near it (Baxter: 349 self checks of 33 links are 64 pairs of 15 groups)."""
    slots, coarse_slot = slot_table(model)
    groups = {}
    for k, e in enumerate(model["env_checks"]):
        link, p, r = slots[coarse_slot[e["link"]]]
        fid, off = kin.sphere_in_frame(link, p)
        for f in e["fine"]:
            assert kin.sphere_in_frame(slots[f][0], slots[f][1])[0] == fid
        assert e["fine"] == list(range(e["fine"][0], e["fine"][0] + len(e["fine"]))), "a link's fine slots are consecutive"
        groups.setdefault(fid, []).append((k, [float(v) for v in off], float(r)))
    order = list(groups)
    of = {k: g for g, fid in enumerate(order) for k, _, _ in groups[fid]}
    pairs = {}
    env_ix = {e["link"]: k for k, e in enumerate(model["env_checks"])}
    for c, e in enumerate(model["self_checks"]):
        a, b = of[env_ix[e["links"][0]]], of[env_ix[e["links"][1]]]
        assert a != b, "links of one rigid group are not checked against each other"
        A, B = (list(dict.fromkeys(p[k] for p in e["fine"])) for k in (0, 1))
        assert [[x, y] for x in A for y in B] == e["fine"], "fine self pairs are a cross product"
        pairs.setdefault((a, b), []).append(c)
    return {"frames": order, "members": [groups[f] for f in order], "pairs": pairs, "env_ix": env_ix}


def gen_cuda(model: dict) -> str:
    name = model["name"]
    S = struct_name(name)
    pre = f"k{S}"
    kin = Kin(model)
    slots, coarse_slot = slot_table(model)
    dim = model["dimension"]
    cull = load_cull(name)
    lay = stage_layout(model, kin, cull)
    groups = link_groups(model, kin)
    members, pairs = groups["members"], groups["pairs"]
    n_groups = len(members)
    assert n_groups <= 32, "one bit of a word per link group"
    boxes_of = danger_boxes(model, cull)
    all_pairs = [tuple(p_) for e in model["self_checks"] for p_ in e["fine"]]
    lines = []
    w = lines.append
    w("// Generated by vamp_gb300/robotgen/codegen.py from vamp_gb300/robots/%s.json. Do not edit." % name)
    w("//")
    w("// FP32 forward kinematics and the fkcc checks of the %s robot, one configuration per thread." % name)
    w("// The checks are the reference's generated Robot::fkcc (src/impl/vamp/robots/%s.hh): environment" % name)
    w("// checks link by link, each a coarse link sphere gating that link's fine spheres, then")
    w("// self-collision link pairs, a coarse pair gating the cross product of the two links' fine")
    w("// spheres.  A state collides if any check does, so their order is free: here a straight-line")
    w("// pass over rigid groups of links finds the checks that can matter, and loops run those.")
    w("#pragma once")
    w("")
    w('#include "../vg_check.cuh"')
    w("")
    w("namespace vg::robots")
    w("{")

    def frames_block(em):
        return emit_frames(kin, em, "q", sc_fn=lambda x, s_, c: f"float {s_}, {c}; vg_sincos_ref({x}, &{s_}, &{c});")

    def table(kind, ctype, ident, rows, fmt):
        body = ", ".join(fmt(r) for r in rows) if rows else fmt(None)
        w(f"    {kind} {ctype} {pre}{ident}[{max(1, len(rows))}] = {{{body}}};")

    def i4(r):
        return "{%d, %d, %d, %d}" % tuple(r if r is not None else (0, 0, 0, 0))

    def f4(r):
        return "{%s}" % ", ".join(lit32(v) for v in (r if r is not None else (0.0, 0.0, 0.0, 0.0)))

    # ---- tables
    em0 = Emitter("cuda", SNAP32)
    offs = []
    for l, p, r in slots:
        v = kin.sphere_in_frame(l, p)[1]
        offs.append((em0.const(float(v[0])), em0.const(float(v[1])), em0.const(float(v[2])), r))
    w("    // slot -> its centre's offset in its frame, and its radius")
    table("__constant__", "float4", "SlotOff", offs, f4)
    w("    // per staged frame and entry: its stage slot, or -1 and the constant value (global memory: see")
    w("    // self_checks)")
    nfr = len(lay["slots"])
    w(f"    __device__ const int {pre}FrameSlot[{nfr}][12] = {{{', '.join('{' + ', '.join(map(str, r)) + '}' for r in lay['slots'])}}};")
    w(f"    __device__ const float {pre}FrameConst[{nfr}][12] = {{{', '.join('{' + ', '.join(lit32(v) for v in r) + '}' for r in lay['consts'])}}};")
    env_rows, group_rows = [], []
    for g, fid in enumerate(groups["frames"]):
        first = len(env_rows)
        for k, _, _ in members[g]:
            e = model["env_checks"][k]
            env_rows.append((coarse_slot[e["link"]], e["fine"][0], e["fine"][0] + len(e["fine"]), 0))
        group_rows.append((lay["frames"][fid], first, len(env_rows), 0))
    w("    // rigid link groups: staged frame, their environment checks; per check its coarse slot and")
    w("    // fine slots")
    table("__constant__", "int4", "Group", group_rows, i4)
    table("__constant__", "int4", "Env", env_rows, i4)
    pair_rows, check_a, check_b, check_box, contain, row_rows, row_b = [], [], [], [], [], [], []
    full0 = [0]
    for e in model["self_checks"]:
        full0.append(full0[-1] + len(e["fine"]))
    for (ga, gb), cs in pairs.items():
        first = len(check_a)
        for c in cs:
            e = model["self_checks"][c]
            sel = range(len(e["fine"])) if cull is None or cull["live"][c] is None else cull["live"][c]
            (j0, j1, found), union = boxes_of[c]
            r0 = len(row_rows)
            last = None
            for i in sel:
                x, y = e["fine"][i]
                if x != last:
                    row_rows.append([x, len(row_b), len(row_b), 0])
                    last = x
                row_b.append(y)
                row_rows[-1][2] = len(row_b)
            check_a.append((coarse_slot[e["links"][0]], coarse_slot[e["links"][1]], r0, len(row_rows)))
            jp = lay["joint_pos"]
            check_b.append((full0[c], full0[c + 1], jp[j0] if found else -1, jp[j1] if found else -1))
            check_box.append(union)
            contain.append(f32_up(containing_radius(model, kin, model["env_checks"][groups["env_ix"][e["links"][1]]]) + CONTAIN_MARGIN))
        fa, fb = groups["frames"][ga], groups["frames"][gb]
        pair_rows.append((lay["frames"][fa], lay["frames"][fb], first, len(check_a)))
    w("    // pairs of link groups: staged frames A and B, their self checks")
    table("__constant__", "int4", "Pair", pair_rows, i4)
    w("    // per self check: coarse slots A and B, its rows of live fine pairs (those that can collide")
    w("    // inside the widened joint limits); all its fine pairs and, where its danger boxes were")
    w("    // found, the staged joints they test (-1: none)")
    table("__constant__", "int4", "CheckA", check_a, i4)
    table("__constant__", "int4", "CheckB", check_b, i4)
    w("    // per self check the union of its live pairs' danger boxes (lo0, hi0, lo1, hi1), joint-space")
    w("    // boxes outside which a live pair keeps the culling margin, and the radius about B's coarse")
    w(f"    // centre that contains B's fine spheres with {CONTAIN_MARGIN} m to spare")
    table("__constant__", "float4", "CheckBox", check_box, f4)
    w(f"    __constant__ float {pre}ContainR[{len(contain)}] = {{{', '.join(lit32(v) for v in contain)}}};")
    w("    // rows: a fine sphere of A (offset and radius), its live pairs' range; per live pair the fine")
    w("    // slot of B, and its sphere (global memory: see self_checks)")
    table("__constant__", "float4", "RowA", [offs[r[0]] for r in row_rows], f4)
    table("__constant__", "int2", "Row", row_rows, lambda r: "{%d, %d}" % (tuple(r[1:3]) if r else (0, 0)))
    table("__device__ const", "float4", "RowSphere", [offs[y] for y in row_b], f4)
    w(f"    __constant__ int {pre}RowB[{max(1, len(row_b))}] = {{{', '.join(map(str, row_b)) or '0'}}};")
    w("    // every fine self pair, in the reference's order (debug reports, and configurations outside")
    w("    // the widened joint limits; global memory)")
    w(f"    __device__ const int2 {pre}AllPair[{max(1, len(all_pairs))}] = {{{', '.join('{%d, %d}' % p for p in all_pairs) or '{0, 0}'}}};")
    arows, afine = attach_tables(model, coarse_slot)
    w("    // links checked against an attachment (fkcc_attach): coarse slot, fine range, staged frame; fine")
    w("    // slots")
    table("__device__ const", "int4", "AttachLink", [r + (lay["frames"][kin.sphere_in_frame(*slots[r[0]][:2])[0]],) for r in arows], i4)
    w(f"    __device__ const int {pre}AttachFine[{max(1, len(afine))}] = {{{', '.join(map(str, afine)) or '0'}}};")
    w("")

    w("struct %s" % S)
    w("{")
    w("    static constexpr const char *kName = \"%s\";" % name)
    w("    static constexpr int kDim = %d;" % dim)
    w("    static constexpr int kFine = %d;" % len(model["fine_spheres"]))
    w("    static constexpr int kSlots = %d;" % len(slots))
    w("    static constexpr int kSelfPairs = %d;" % len(all_pairs))
    w(f"    static __device__ __forceinline__ int2 self_pair(int i) {{ return {pre}AllPair[i]; }}")
    w("    // floats of shared-memory staging per thread: the non-constant entries of the checks' frames")
    w("    // and the joint values the danger boxes test")
    w("    static constexpr int kStage = %d;" % lay["total"])
    w("    // resident blocks per SM of the same-edge kernels")
    w("    static constexpr int kEdgeBlocks = %d;" % EDGE_BLOCKS[name])
    w("    static constexpr int kResolution = %d;" % model["resolution"])
    w("    static constexpr float kMinRadius = %s;" % lit32(model["min_radius"]))
    w("    static constexpr float kMaxRadius = %s;" % lit32(model["max_radius"]))
    w("    static constexpr float kScaleM[%d] = {%s};" % (dim, ", ".join(lit32(v) for v in model["s_m"])))
    w("    static constexpr float kScaleA[%d] = {%s};" % (dim, ", ".join(lit32(v) for v in model["s_a"])))
    w("")

    # ---- all sphere slots, straight-line (FK queries)
    em = Emitter("cuda", SNAP32)
    fr = frames_block(em)
    body = list(em.lines)
    for i, (link, p, r) in enumerate(slots):
        em.lines = []
        x, y, z = emit_centre(em, fr, kin, link, p, f"s{i}_")
        body += em.lines
        body.append(f"out[{4 * i}] = {x}; out[{4 * i + 1}] = {y}; out[{4 * i + 2}] = {z}; out[{4 * i + 3}] = {lit32(r)};")
    w("    // Every sphere slot: fine spheres 0..kFine-1, then the coarse sphere of each checked link.")
    w("    static __device__ __forceinline__ void spheres(const float *q, float *out)")
    w("    {")
    for l in body:
        w("        " + l)
    w("    }")
    w("")

    # ---- end-effector transform and the attachment checks (fkcc_attach)
    em = Emitter("cuda", SNAP32)
    fr = frames_block(em)
    vals = emit_ee_pose(em, fr, kin, model["end_effector"])
    body = list(em.lines) + [" ".join(f"T[{i}] = {em.ref(v)};" for i, v in enumerate(vals))]
    w(f"    // Transform of {model['end_effector']}, where fkcc_attach poses an attachment: R row-major, then t.")
    w("    static __device__ __forceinline__ void ee_pose(const float *q, float *T)")
    w("    {")
    for l in body:
        w("        " + l)
    w("    }")
    # the same transform from the staged frame of the end effector's link
    ee_fid = kin.link_frame[model["end_effector"]][0]
    em = Emitter("cuda", SNAP32)
    R0, t0 = fr[ee_fid]
    entry = lambda v, i: v if isinstance(v, float) else f"f.m[{i}]"  # noqa: E731
    staged = ([[entry(R0[r][c], 3 * r + c) for c in range(3)] for r in range(3)], [entry(t0[r], 9 + r) for r in range(3)])
    vals = emit_ee_pose(em, {ee_fid: staged}, kin, model["end_effector"])
    w(f"    // The same from the staged frame kEeFrame.")
    w(f"    static constexpr int kEeFrame = {lay['frames'][ee_fid]};")
    w("    static __device__ __forceinline__ void ee_of(const vg::Frame &f, float *T)")
    w("    {")
    for l in em.lines + [" ".join(f"T[{i}] = {em.ref(v)};" for i, v in enumerate(vals))]:
        w("        " + l)
    w("    }")
    w(f"    static __device__ __forceinline__ float4 slot_offset(int i) {{ return {pre}SlotOff[i]; }}")
    w("    // links checked against an attachment, in the reference's order: coarse slot, fine range, frame")
    w(f"    static constexpr int kAttachLinks = {len(arows)};")
    w(f"    static __device__ __forceinline__ int4 attach_link(int i) {{ return k{S}AttachLink[i]; }}")
    w(f"    static __device__ __forceinline__ int attach_fine(int i) {{ return k{S}AttachFine[i]; }}")
    w("")

    # ---- fkcc.  Straight-line: the kinematics, the frames to the shared-memory stage, one sphere
    # per link group, the groups' field lookups and the group pairs' tests into per-lane bit words
    # (independent operations, no votes).  Then loops over the set bits of the words' warp-wide OR.
    # What bounds it is latency: the loop over every link pair that this replaces was a chain of
    # table loads, shared-memory loads and a vote per pair, 60 % of the edge check once the field
    # had taken most environment queries out.  65,536 Panda motions 1.70 -> 0.69 ms, 9,973 UR5
    # vectors 0.23 -> 0.13, four robots' graph 5.36 -> 3.37 (the smaller stage, 33 instead of 53 KB
    # a block for the Panda, and five resident blocks instead of four included).
    em = Emitter("cuda", SNAP32)
    fr = frames_block(em)
    body = list(em.lines)
    body += limits_code(model, cull)
    near = " & ".join(f"(fabsf(q[{d}]) <= {lit32(FAR_JOINT)})" for d in range(dim))
    far_test = f"ctx.far = __any_sync(vg::kFull, !({near}) && ((ctx.alive >> (threadIdx.x & 31)) & 1u));"
    if name in FAR_LATE:
        body += ["if (__builtin_expect(!ctx.in_limits, 0))", "{", f"    {far_test}", "}"]
    body.append("float *const st = ctx.stage;")
    vals_ = [f"(-{v[1:]})" if v.startswith("-") else v for v in lay["values"]]
    for i in range(0, len(vals_), 6):
        body.append(" ".join(f"st[{j} * vg::kStageStride] = {vals_[j]};" for j in range(i, min(i + 6, len(vals_)))))
    for i, d in enumerate(lay["joints"]):
        body.append(f"st[{lay['q0'] + i} * vg::kStageStride] = q[{d}];")
    group_sphere = []
    for g, fid in enumerate(groups["frames"]):
        names = ", ".join(model["env_checks"][k]["link"] for k, _, _ in members[g])
        body.append(f"// group {g}: {names}")
        em.lines = []
        if len(members[g]) == 1:
            link, p, r = slots[coarse_slot[model["env_checks"][members[g][0][0]]["link"]]]
            xyz = emit_centre(em, fr, kin, link, p, f"g{g}_")
        else:
            c, r = enclosing_sphere([(tuple(off), rad) for _, off, rad in members[g]])
            xyz = emit_point(em, fr[fid], c, f"g{g}_")
        body += em.lines
        group_sphere.append((xyz, float(r)))
        body.append(f"unsigned v{g} = ctx.clearance({', '.join(xyz)});")
    em.lines = []
    body.append("// per lane: the pairs of groups that overlap, and those whose joints lie in a danger box")
    plist = list(pairs)
    n_words = -(-len(plist) // 32)
    gate = []
    for wd in range(n_words):
        part = plist[32 * wd:32 * wd + 32]
        body.append(f"unsigned over{wd} = 0u;")
        for j, (ga, gb) in enumerate(part):
            (A, ra), (B, rb) = group_sphere[ga], group_sphere[gb]
            # the reference's own coarse test where both groups are single links, else one that
            # contains it
            body.append(f"over{wd} = vg::shift_in(over{wd}, vg::self_bits({', '.join(A)}, {', '.join(B)}, "
                        f"__fadd_rn({lit32(ra)}, {lit32(rb)})));")
            if all(boxes_of[c][0][2] for c in pairs[(ga, gb)]):
                gate.append((wd, len(part) - 1 - j, [boxes_of[c] for c in pairs[(ga, gb)]]))
        body.append(f"unsigned boxed{wd} = ~0u;")
    body.append("if (ctx.in_limits)")
    body.append("{")
    for wd, bit, bs in gate:
        cond = " | ".join("((q[%d] >= %s) & (q[%d] <= %s) & (q[%d] >= %s) & (q[%d] <= %s))" % (
            b[0][0], lit32(b[1][0]), b[0][0], lit32(b[1][1]), b[0][1], lit32(b[1][2]), b[0][1], lit32(b[1][3])) for b in bs)
        body.append(f"    boxed{wd} &= {cond} ? ~0u : ~{1 << bit}u;")
    body.append("}")
    # far lanes: what stands for a group contains nothing for sure, so every check is run
    far_over = [f"over{wd} = {hex((1 << len(plist[32 * wd:32 * wd + 32])) - 1)}u;" for wd in range(n_words)]
    if name not in FAR_LATE:
        body += ["else", "{", f"    {far_test}", "    if (ctx.far)  // no sphere that stands for others is relied on", "    {"]
        body += [f"        {line}" for line in far_over]
        body += ["        %s = 0u;" % " = ".join(f"v{g}" for g in range(n_groups)), "    }", "}"]
    body.append("// per lane: the groups that may touch something")
    body.append("unsigned near = 0u;")
    for g in range(n_groups):
        body.append(f"near = vg::shift_in(near, v{g} - vg::field_reach({lit32(group_sphere[g][1])}));")
    if name in FAR_LATE:
        body += ["if (__builtin_expect(ctx.far, 0))  // no sphere that stands for others is relied on", "{"]
        body += [f"    {line}" for line in far_over]
        body += [f"    near = {hex((1 << n_groups) - 1)}u;", "}"]
    body.append("const unsigned on = (ctx.alive >> (threadIdx.x & 31)) & 1u ? ~0u : 0u;")
    body += f"""// environment checks of those groups
unsigned todo = __reduce_or_sync(vg::kFull, near & on);
#pragma unroll 1
while (todo)
{{
    const int bit = 31 - __clz(static_cast<int>(todo));
    todo ^= 1u << bit;
    const unsigned m = ctx.vote_near((near >> bit) & 1u, ctx.alive);
    if (!m)
    {{
        continue;
    }}
    const int4 g = {pre}Group[{n_groups - 1} - bit];
    const vg::Frame f = frame_at(st, g.x);
#pragma unroll 1
    for (int k = g.y; k < g.z; ++k)
    {{
        // the coarse sphere, then (where it hit) the fine ones: one copy of the query
        const int4 e = {pre}Env[k];
        unsigned need = m & ctx.alive;
        int next = e.y;
        bool coarse = true;
#pragma unroll 1
        for (int slot = e.x;; slot = next++)
        {{
            const float4 c = vg::frame_point(f, {pre}SlotOff[slot]);
            const unsigned may = ctx.may_touch(c, need);
            const unsigned hit = may ? ctx.env_hit(c, vg::seg_any<Ctx::kW>(may), may) : 0u;
            if (coarse)
            {{
                need = hit;
                coarse = false;
            }}
            else if (hit)
            {{
                if (!ctx.kill(hit))
                {{
                    return;
                }}
                need &= ctx.alive;
            }}
            if (!need || next >= e.z)
            {{
                break;
            }}
        }}
    }}
}}""".split("\n")
    for wd in range(n_words):
        part = plist[32 * wd:32 * wd + 32]
        body += f"""// self checks of the group pairs that overlap
if (!self_checks(ctx, st, over{wd}, boxed{wd}, on, {32 * wd + len(part) - 1}))
{{
    return;
}}""".split("\n")
    box_gate = ""
    if any(found for (_, _, found), _ in boxes_of):
        box_gate = f"""
                const int4 cb4 = {pre}CheckB[k];
                float qa = 0.0f, qb = 0.0f;
                if (cb4.z >= 0)
                {{
                    // only the lanes whose joints lie in the check's danger box
                    qa = st[({lay['q0']} + cb4.z) * vg::kStageStride];
                    qb = st[({lay['q0']} + cb4.w) * vg::kStageStride];
                    mine &= __ballot_sync(vg::kFull, vg::in_box({pre}CheckBox[k], qa, qb));
                    if (!mine)
                    {{
                        continue;
                    }}
                }}"""
    w(f"""    // Staged frame f: its non-constant entries from this thread's stage, the rest constants.
    static __device__ __forceinline__ vg::Frame frame_at(const float *st, int f)
    {{
        vg::Frame r;
#pragma unroll
        for (int c = 0; c < 12; ++c)
        {{
            const int slot = {pre}FrameSlot[f][c];
            r.m[c] = slot >= 0 ? st[slot * vg::kStageStride] : {pre}FrameConst[f][c];
        }}
        return r;
    }}

    // Self checks of the group pairs last, last - 1, ... whose bit (0, 1, ...) is set in some
    // lane's word `over` and in some lane's word `boxed`; `on`: all bits in the lanes checked.
    // Each pair's checks run the reference's coarse test; where it overlaps, each fine sphere of A
    // against B's containing sphere (every fine sphere of B lies inside it with CONTAIN_MARGIN to
    // spare), and only rows that may touch it against B's spheres.  False once no segment is left.
    //
    // What bounds it is the latency of its tables, which are many times what the constant cache
    // holds.  The frames' entries lie in global memory, where the L1 cache holds them.  Single
    // configurations, whose warps walk nearly every check, read the pairs' spheres there too, two
    // rows and two pairs a step, and only for lanes inside the check's danger box and not yet found
    // colliding: 1,048,576 of Panda 598 -> 352 us (570 with constant tables, 390 with every table in
    // global memory; Fetch 2,172 -> 1,186, 1,643 and 1,337; a danger box per pair cost more than it
    // saved).  Segments, whose lanes are neighbours, walk few rows: one at a time from the constant
    // tables, 65,536 Panda motions 639 us and 646 from global memory, 648 in the other form.
    template <typename Ctx>
    static __device__ __forceinline__ bool self_checks(Ctx &ctx, const float *st, unsigned over, unsigned boxed, unsigned on, int last)
    {{
        const int lane = threadIdx.x & 31;
        unsigned todo = __reduce_or_sync(vg::kFull, over & on) & __reduce_or_sync(vg::kFull, boxed & on);
#pragma unroll 1
        while (todo)
        {{
            const int bit = 31 - __clz(static_cast<int>(todo));
            todo ^= 1u << bit;
            const unsigned some = ctx.vote_near((over >> bit) & 1u, ctx.alive) & ctx.vote_near((boxed >> bit) & 1u, ctx.alive);
            if (!some)
            {{
                continue;
            }}
            const int4 p = {pre}Pair[last - bit];
            const vg::Frame a = frame_at(st, p.x), b = frame_at(st, p.y);
#pragma unroll 1
            for (int k = p.z; k < p.w; ++k)
            {{
                const int4 ck = {pre}CheckA[k];
                const float4 ca = vg::frame_point(a, {pre}SlotOff[ck.x]);
                float4 cb = vg::frame_point(b, {pre}SlotOff[ck.y]);
                const unsigned need = ctx.self_hit(ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w, some & ctx.alive);
                if (!need)
                {{
                    continue;
                }}
                unsigned acc = 0u;
                if (!ctx.in_limits)
                {{
                    const int4 all = {pre}CheckB[k];
#pragma unroll 1
                    for (int i = all.x; i < all.y; ++i)
                    {{
                        const int2 pr = {pre}AllPair[i];
                        const float4 sa = vg::frame_point(a, {pre}SlotOff[pr.x]), sb = vg::frame_point(b, {pre}SlotOff[pr.y]);
                        acc |= vg::self_bits(sa.x, sa.y, sa.z, sb.x, sb.y, sb.z, __fadd_rn(sa.w, sb.w));
                    }}
                    const unsigned hit = ctx.vote(acc, need);
                    if (hit && !ctx.kill(hit))
                    {{
                        return false;
                    }}
                    continue;
                }}
                unsigned mine = need;  // the lanes still in question{box_gate}
                cb.w = {pre}ContainR[k];
                if constexpr (Ctx::kW > 1)  // one row at a time
                {{
#pragma unroll 1
                    for (int r = ck.z; r < ck.w; ++r)
                    {{
                        const int2 row = {pre}Row[r];
                        const float4 sa = vg::frame_point(a, {pre}RowA[r]);
                        if (!(__ballot_sync(vg::kFull, vg::spheres_meet(sa, cb)) & mine))
                        {{
                            continue;
                        }}
#pragma unroll 1
                        for (int i = row.x; i < row.y; ++i)
                        {{
                            const float4 sb = vg::frame_point(b, {pre}SlotOff[{pre}RowB[i]]);
                            acc |= vg::self_bits(sa.x, sa.y, sa.z, sb.x, sb.y, sb.z, __fadd_rn(sa.w, sb.w));
                        }}
                    }}
                    const unsigned hit = ctx.vote(acc, need);
                    if (hit && !ctx.kill(hit))
                    {{
                        return false;
                    }}
                    continue;
                }}
                constexpr int kRows = 2;
#pragma unroll 1
                for (int r = ck.z; r < ck.w && mine; r += kRows)
                {{
                    unsigned meet = 0u;
#pragma unroll
                    for (int j = 0; j < kRows; ++j)
                    {{
                        const bool hit = vg::spheres_meet(vg::frame_point(a, {pre}RowA[min(r + j, ck.w - 1)]), cb);
                        meet |= hit && r + j < ck.w ? 1u << j : 0u;
                    }}
                    unsigned rows = __reduce_or_sync(vg::kFull, (mine >> lane) & 1u ? meet : 0u);
#pragma unroll 1
                    for (; rows; rows &= rows - 1u)
                    {{
                        const int j = __ffs(static_cast<int>(rows)) - 1;
                        const unsigned m = __ballot_sync(vg::kFull, (meet >> j) & 1u) & mine;
                        if (!m)
                        {{
                            continue;
                        }}
                        const int2 row = {pre}Row[r + j];
                        const float4 sa = vg::frame_point(a, {pre}RowA[r + j]);
#pragma unroll 2
                        for (int i = row.x; i < row.y; ++i)
                        {{
                            const float4 sb = vg::frame_point(b, {pre}RowSphere[i]);
                            acc |= vg::self_bits(sa.x, sa.y, sa.z, sb.x, sb.y, sb.z, __fadd_rn(sa.w, sb.w));
                        }}
                        mine &= ~__ballot_sync(vg::kFull, acc >> 31);
                    }}
                }}
                const unsigned hit = ctx.vote(acc, need);
                if (hit && !ctx.kill(hit))
                {{
                    return false;
                }}
            }}
        }}
        return true;
    }}
""")
    w("    // Robot::fkcc for the lanes of ctx.alive.  Clears the lanes of every segment found in collision.")
    w("    template <typename Ctx>")
    w("    static __device__ __forceinline__ void fkcc(const float *q, Ctx &ctx)")
    w("    {")
    for l in body:
        w("        " + l)
    w("    }")
    w("};")
    w("}  // namespace vg::robots")
    return "\n".join(lines) + "\n"


# --------------------------------------------------------------------------------------------
# C oracle output


def gen_c(model: dict) -> str:
    name = model["name"]
    kin = Kin(model)
    slots, coarse_slot = slot_table(model)
    dim = model["dimension"]
    P = name.upper()
    lines = []
    w = lines.append
    w("/* Generated by vamp_gb300/robotgen/codegen.py from vamp_gb300/robots/%s.json. Do not edit." % name)
    w(" *")
    w(" * CPU oracle tables and kinematics for the %s robot.  Test infrastructure only." % name)
    w(" * Schedule: the reference's Robot::fkcc (src/impl/vamp/robots/%s.hh), as tables." % name)
    w(" * FK: the same FP32 operation sequence as the CUDA kernels, plus an FP64 version. */")
    w("#pragma once")
    w("#include <math.h>")
    w('#include "../vgo_math.h"')
    w("")
    w("#define VGO_%s_DIM %d" % (P, dim))
    w("#define VGO_%s_FINE %d" % (P, len(model["fine_spheres"])))
    w("#define VGO_%s_SLOTS %d" % (P, len(slots)))
    w("#define VGO_%s_RESOLUTION %d" % (P, model["resolution"]))
    w("static const float vgo_%s_s_m[%d] = {%s};" % (name, dim, ", ".join(lit32(v) for v in model["s_m"])))
    w("static const float vgo_%s_s_a[%d] = {%s};" % (name, dim, ", ".join(lit32(v) for v in model["s_a"])))
    w("static const float vgo_%s_radius_range[2] = {%s, %s};" % (name, lit32(model["min_radius"]), lit32(model["max_radius"])))
    # env schedule
    env_coarse = [coarse_slot[e["link"]] for e in model["env_checks"]]
    env_start, env_fine = [], []
    for e in model["env_checks"]:
        env_start.append(len(env_fine))
        env_fine += e["fine"]
    env_start.append(len(env_fine))
    w("#define VGO_%s_ENV_CHECKS %d" % (P, len(env_coarse)))
    w("static const int vgo_%s_env_coarse[] = {%s};" % (name, ", ".join(map(str, env_coarse))))
    w("static const int vgo_%s_env_start[] = {%s};" % (name, ", ".join(map(str, env_start))))
    w("static const int vgo_%s_env_fine[] = {%s};" % (name, ", ".join(map(str, env_fine))))
    self_coarse, self_start, self_fine = [], [], []
    for e in model["self_checks"]:
        a, b = e["links"]
        self_coarse += [coarse_slot[a], coarse_slot[b]]
        self_start.append(len(self_fine) // 2)
        for sa, sb in e["fine"]:
            self_fine += [sa, sb]
    self_start.append(len(self_fine) // 2)
    arows, afine = attach_tables(model, coarse_slot)
    w("#define VGO_%s_ATTACH_LINKS %d" % (P, len(arows)))
    w("static const int vgo_%s_attach_coarse[] = {%s};" % (name, ", ".join(str(r[0]) for r in arows) or "0"))
    w("static const int vgo_%s_attach_start[] = {%s};" % (name, ", ".join(str(r[1]) for r in arows + [(0, len(afine), 0)])))
    w("static const int vgo_%s_attach_fine[] = {%s};" % (name, ", ".join(map(str, afine)) or "0"))
    w("#define VGO_%s_SELF_CHECKS %d" % (P, len(model["self_checks"])))
    w("static const int vgo_%s_self_coarse[] = {%s};" % (name, ", ".join(map(str, self_coarse)) or "0"))
    w("static const int vgo_%s_self_start[] = {%s};" % (name, ", ".join(map(str, self_start))))
    w("static const int vgo_%s_self_fine[] = {%s};" % (name, ", ".join(map(str, self_fine)) or "0"))
    w("")

    for tgt, ty, sc in (("c32", "float", "vgo_sincos_ref"), ("c64", "double", None)):
        em = Emitter(tgt, SNAP32 if tgt == "c32" else 0.0)
        if tgt == "c32":
            scf = lambda x, s, c: f"float {s}, {c}; vgo_sincos_ref({x}, &{s}, &{c});"
        else:
            scf = lambda x, s, c: f"const double {s} = sin({x}), {c} = cos({x});"
        fr = emit_frames(kin, em, "q", sc_fn=scf)
        body = list(em.lines)
        for i, (link, p, r) in enumerate(slots):
            em.lines = []
            x, y, z = emit_centre(em, fr, kin, link, p, f"s{i}_")
            body += em.lines
            rr = lit32(r) if tgt == "c32" else lit64(f32(r))
            body.append(f"out[{4 * i}] = {em.ref(x)}; out[{4 * i + 1}] = {em.ref(y)}; out[{4 * i + 2}] = {em.ref(z)}; out[{4 * i + 3}] = {rr};")
        suffix = "f32" if tgt == "c32" else "f64"
        if tgt == "c32":
            em2 = Emitter(tgt, SNAP32)
            fr2 = emit_frames(kin, em2, "q", sc_fn=scf)
            vals = emit_ee_pose(em2, fr2, kin, model["end_effector"])
            w(f"/* Transform of {model['end_effector']} (fkcc_attach's attachment frame): R row-major, then t. */")
            w(f"static void vgo_{name}_ee_pose_f32(const float *q, float *T)")
            w("{")
            for l in em2.lines:
                w("    " + l)
            w("    " + " ".join(f"T[{i}] = {em2.ref(v)};" for i, v in enumerate(vals)))
            w("}")
            w("")
        w(f"/* Every sphere slot (fine, then coarse), {ty}: out[4 * slot + (x, y, z, r)]. */")
        w(f"static void vgo_{name}_spheres_{suffix}(const {ty} *q, {ty} *out)")
        w("{")
        for l in body:
            w("    " + l)
        w("}")
        w("")
    return "\n".join(lines) + "\n"


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("robots", nargs="*", default=["panda", "ur5", "fetch", "baxter"])
    a = ap.parse_args()
    CUDA_OUT.mkdir(parents=True, exist_ok=True)
    C_OUT.mkdir(parents=True, exist_ok=True)
    for r in a.robots:
        model = json.loads((MODELS / f"{r}.json").read_text())
        (CUDA_OUT / f"{r}.cuh").write_text(gen_cuda(model))
        (C_OUT / f"{r}.h").write_text(gen_c(model))
        print(r, "ok")


if __name__ == "__main__":
    main()
