"""Host-side models of the tensor-memory kernels' producer / converter / MMA / epilogue pipelines.

The kernels (hidet_b200/csrc: qlinear_prefill.cu is `Pipeline`, qlinear_pair.cu and qlinear_mid.cu are `TensorMemoryPipeline`) synchronise their
warps with mbarriers waited on by phase parity.  A parity wait cannot tell a phase from the one two steps away, so the protocol is only correct if
no waiter can ever be two phases off.  The models restate the protocol (which barrier each role waits on,
with which parity, and what it signals), run it under randomly interleaved schedules in which copies land
out of order and late, and check that every role only ever touches the data it means to touch and that
nothing stalls.  Ring depths and group counts are read from the kernel source.

Test infrastructure only.
"""
from __future__ import annotations

import os
import random
import re
from dataclasses import dataclass
from typing import Callable, Dict, Generator, List, Optional, Tuple

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'hidet_b200', 'csrc')
KERNEL_SOURCE = os.path.join(KERNELS, 'qlinear_prefill.cu')


class ProtocolError(AssertionError):
    pass


@dataclass
class PipelineConfig:
    stages: int          # f16 weight + activation ring
    raw_slots: int       # int8 ring
    conv_groups: int     # converter groups taking stages in turn
    group_warps: int
    raw_period: int      # stages after which a (slot, group) pair recurs
    per_group_barriers: bool = True   # one "landed" barrier per (slot, group); False = one per slot
    drain_on_exit: bool = True        # producer / MMA lane wait for what they have in flight before the CTA retires
    epilogue_agrees: bool = True      # the warps that meet at a named barrier decide together whether their wait gave up


def _ternary(text: str, name: str, tm: int) -> int:
    m = re.search(r'static constexpr int %s = TM == 256 \? (\d+) : (\d+);' % name, text)
    if m is None:
        raise ProtocolError('cannot find {} in the kernel source'.format(name))
    return int(m.group(1) if tm == 256 else m.group(2))


def _epilogue_agrees(text: str) -> bool:
    """Whether the wait for the accumulator is decided by all warps of an epilogue group together."""
    waits = re.findall(r'if \(!(.*)wait\(smem_u32\(&acc_full', text)
    if len(waits) != 1:
        raise ProtocolError('cannot find the wait for the accumulator in the kernel source')
    return waits[0].startswith('all_of_128(')


def config_from_source(tm: int) -> PipelineConfig:
    text = open(KERNEL_SOURCE).read()
    conv_warps = int(re.search(r'constexpr int CONV_WARPS = (\d+);', text).group(1))
    groups = _ternary(text, 'CONV_GROUPS', tm)
    return PipelineConfig(stages=_ternary(text, 'STAGES', tm), raw_slots=_ternary(text, 'RAW_SLOTS', tm), conv_groups=groups,
                          group_warps=conv_warps // groups, raw_period=_ternary(text, 'RAW_PERIOD', tm),
                          epilogue_agrees=_epilogue_agrees(text))


class Barrier:
    """mbarrier: a phase completes when the expected arrivals have come and no copy bytes are outstanding."""

    def __init__(self, name: str, count: int):
        self.name, self.count = name, count
        self.arrived = 0
        self.tx = 0
        self.phases_done = 0

    def _settle(self):
        if self.arrived == self.count and self.tx == 0:
            self.arrived = 0
            self.phases_done += 1

    def arrive(self):
        if self.arrived >= self.count:
            raise ProtocolError('{}: more arrivals than the phase expects'.format(self.name))
        self.arrived += 1
        self._settle()

    def arrive_expect_tx(self, n: int):
        if self.arrived >= self.count:
            raise ProtocolError('{}: a second copy armed on a phase that is still pending'.format(self.name))
        self.tx += n
        self.arrived += 1

    def complete_tx(self, n: int):
        self.tx -= n
        self._settle()

    def test(self, parity: int) -> bool:
        """try_wait.parity: true when the phase of that parity is not the one in progress."""
        return (self.phases_done & 1) != (parity & 1)


class Meeting:
    """A barrier of `count` roles at which nobody's wait gives up; it hands everyone the AND of what they bring."""

    def __init__(self, count: int):
        self.count, self.answers, self.results = count, [], []

    def come(self, answer: bool = True):
        """The wait of the role that comes; the answer is in `results` under the number returned with it."""
        number = len(self.results)
        self.answers.append(answer)
        if len(self.answers) == self.count:
            self.results.append(all(self.answers))
            self.answers = []
        return number, ('meeting', lambda: len(self.results) > number)


Wait = Optional[Callable[[], bool]]


class Aborted(Exception):
    """Raised inside a role when the CTA-wide abort flag ends one of its waits."""


def stays(wait: Callable[[], bool], group: Optional[Meeting]):
    """A wait that may give up; false then.  With `group`, the answer of all its roles."""
    ok = True
    try:
        yield wait
    except Aborted:
        ok = False
    if group is None:
        return ok
    number, meeting = group.come(ok)
    yield meeting
    return group.results[number]


class Scheduler:
    """Runs the roles of one or two CTAs under a random schedule."""

    def __init__(self, rng: random.Random, ctas: int = 1):
        self.rng = rng
        self.copies: List[Callable[[], None]] = []      # copies in flight: may land in any order
        self.commits: List[Callable[[], None]] = []     # tensor-core commits: land in order
        self.abort = [False] * ctas                     # the flag a role raises in its CTA when its own wait runs out
        self.expire: Optional[Tuple[int, int]] = None   # (agent, n): that agent's n-th blocked wait "runs out"
        self.retired_dirty: Optional[str] = None

    def cta_of(self, agent: int) -> int:
        return 0

    def run(self, copy_delay: float = 0.5, max_steps: int = 2_000_000) -> int:
        """Runs all roles to completion under a random schedule; returns the number of steps taken.
        `copy_delay` is the chance that a step is not spent on landing a copy even though one is in flight."""
        agents = self.roles()
        waits: List = [None] * len(agents)
        alive = [True] * len(agents)
        blocked_count = [0] * len(agents)
        steps = 0

        def ready(k: int) -> bool:
            w = waits[k]
            if w is None:
                return True
            if isinstance(w, tuple):          # a teardown wait: not cut short by the abort flag
                return w[1]()
            if w():
                return True
            if self.abort[self.cta_of(k)]:
                return True                   # the wait ends; the role sees the flag and leaves
            return False

        while any(alive) or self.copies or self.commits:
            steps += 1
            if steps > max_steps:
                raise ProtocolError('no end after {} steps'.format(max_steps))
            if not any(alive) and (self.copies or self.commits) and self.retired_dirty is None:
                self.retired_dirty = '{} copies and {} commits in flight'.format(len(self.copies), len(self.commits))
            # a blocked wait of the chosen agent "runs out": that role raises the flag
            if self.expire is not None and not any(self.abort):
                k, n = self.expire
                if alive[k] and waits[k] is not None and not isinstance(waits[k], tuple) and not waits[k]():
                    blocked_count[k] += 1
                    if blocked_count[k] >= n:
                        self.abort[self.cta_of(k)] = True
            runnable = [k for k in range(len(agents)) if alive[k] and ready(k)]
            choices: List[Tuple[str, int]] = [('agent', k) for k in runnable]
            if self.commits:
                choices.append(('commit', 0))
            if self.copies and (not choices or self.rng.random() > copy_delay):
                choices.append(('copy', self.rng.randrange(len(self.copies))))
            if not choices and any(self.abort) and not all(self.abort):
                self.abort = [True] * len(self.abort)   # the waits of the other CTA run out in their turn
                continue
            if not choices:
                stuck = [k for k in range(len(agents)) if alive[k]]
                raise ProtocolError('deadlock: roles {} wait and nothing is in flight'.format(stuck))
            kind, k = self.rng.choice(choices)
            if kind == 'copy':
                self.copies.pop(k)()
            elif kind == 'commit':
                self.commits.pop(0)()
            else:
                try:
                    w = waits[k]
                    if w is not None and not isinstance(w, tuple) and self.abort[self.cta_of(k)] and not w():
                        waits[k] = agents[k].throw(Aborted())   # the wait ended because of the flag
                    else:
                        waits[k] = next(agents[k])
                except StopIteration:
                    alive[k] = False
        if self.retired_dirty is not None:
            raise ProtocolError('the kernel retired with ' + self.retired_dirty)
        return steps


class Pipeline(Scheduler):
    def __init__(self, cfg: PipelineConfig, tiles: int, k_blocks: int, rng: random.Random):
        super().__init__(rng)
        self.cfg, self.tiles, self.k_blocks = cfg, tiles, k_blocks
        c = cfg
        if c.per_group_barriers:
            self.raw_full = [[Barrier('raw_full[{}][{}]'.format(r, g), 1) for g in range(c.conv_groups)] for r in range(c.raw_slots)]
        else:
            shared = [Barrier('raw_full[{}]'.format(r), 1) for r in range(c.raw_slots)]
            self.raw_full = [[shared[r]] * c.conv_groups for r in range(c.raw_slots)]
        self.raw_empty = [Barrier('raw_empty[{}]'.format(r), c.group_warps) for r in range(c.raw_slots)]
        self.act_full = [Barrier('act_full[{}]'.format(s), 1) for s in range(c.stages)]
        self.conv_full = [Barrier('conv_full[{}]'.format(s), c.group_warps) for s in range(c.stages)]
        self.slot_free = [Barrier('slot_free[{}]'.format(s), 1) for s in range(c.stages)]
        self.acc_full = [Barrier('acc_full[{}]'.format(b), 1) for b in range(2)]
        self.acc_empty = [Barrier('acc_empty[{}]'.format(b), 4) for b in range(2)]
        # what each buffer holds: the stage index (or tile index) whose data is in it
        self.raw_content: List[Optional[int]] = [None] * c.raw_slots
        self.act_content: List[Optional[int]] = [None] * c.stages
        self.conv_content: List[Dict[int, int]] = [dict() for _ in range(c.stages)]   # warp -> stage index it wrote
        self.acc_content: List[Optional[Tuple[str, int]]] = [None, None]
        self.mma_reading: Dict[int, int] = {}           # stage slot -> stage index the tensor core still reads
        self.epilogue_barrier = Meeting(4)

    # ---- roles ----
    def producer(self) -> Generator[Wait, None, None]:
        try:
            yield from self._producer_loop()
        except Aborted:
            pass
        if self.cfg.drain_on_exit:
            # teardown: every copy armed by this lane must have landed (copies land without anyone's help)
            yield ('drain', lambda: not self.copies)

    def _producer_loop(self) -> Generator[Wait, None, None]:
        c = self.cfg
        i = 0
        for _tile in range(self.tiles):
            for _kb in range(self.k_blocks):
                r, use_r = i % c.raw_slots, i // c.raw_slots
                if use_r >= 1:
                    yield lambda r=r, p=(use_r - 1) & 1: self.raw_empty[r].test(p)
                bar = self.raw_full[r][i % c.conv_groups]
                bar.arrive_expect_tx(1)

                def land_raw(r=r, i=i, bar=bar):
                    self.raw_content[r] = i
                    bar.complete_tx(1)

                self.copies.append(land_raw)
                yield None
                s, use = i % c.stages, i // c.stages
                if use >= 1:
                    yield lambda s=s, p=(use - 1) & 1: self.slot_free[s].test(p)
                self.act_full[s].arrive_expect_tx(1)

                def land_act(s=s, i=i):
                    if s in self.mma_reading:
                        raise ProtocolError('activation tile {} lands in a slot the tensor core still reads'.format(i))
                    self.act_content[s] = i
                    self.act_full[s].complete_tx(1)

                self.copies.append(land_act)
                yield None
                i += 1

    def converter(self, group: int, warp: int) -> Generator[Wait, None, None]:
        try:
            yield from self._converter_loop(group, warp)
        except Aborted:
            pass

    def _converter_loop(self, group: int, warp: int) -> Generator[Wait, None, None]:
        c = self.cfg
        for i in range(self.tiles * self.k_blocks):
            if i % c.conv_groups != group:
                continue
            r, use_r = i % c.raw_slots, i // c.raw_slots
            s, use = i % c.stages, i // c.stages
            parity = (i // c.raw_period) & 1 if c.per_group_barriers else use_r & 1
            yield lambda r=r, p=parity: self.raw_full[r][group].test(p)
            if use >= 1:
                yield lambda s=s, p=(use - 1) & 1: self.slot_free[s].test(p)
            if self.raw_content[r] != i:
                raise ProtocolError('converter group {} reads slot {} for stage {} but it holds {}'.format(group, r, i, self.raw_content[r]))
            yield None
            self.raw_empty[r].arrive()
            yield None
            if s in self.mma_reading:
                raise ProtocolError('converter writes stage slot {} while the tensor core reads it'.format(s))
            self.conv_content[s][warp] = i
            self.conv_full[s].arrive()
            yield None

    def mma(self) -> Generator[Wait, None, None]:
        try:
            yield from self._mma_loop()
        except Aborted:
            pass
        if self.cfg.drain_on_exit:
            # teardown: a final commit; it arrives when every MMA issued so far has completed
            yield ('drain', lambda: not self.commits)

    def _mma_loop(self) -> Generator[Wait, None, None]:
        c = self.cfg
        i = 0
        for t in range(self.tiles):
            buf, acc_use = t & 1, t >> 1
            if acc_use >= 1:
                yield lambda buf=buf, p=(acc_use - 1) & 1: self.acc_empty[buf].test(p)
            self.acc_content[buf] = ('writing', t)
            for _kb in range(self.k_blocks):
                s, use = i % c.stages, i // c.stages
                yield lambda s=s, p=use & 1: self.act_full[s].test(p)
                yield lambda s=s, p=use & 1: self.conv_full[s].test(p)
                wrote = self.conv_content[s]
                if self.act_content[s] != i or len(wrote) != c.group_warps or any(v != i for v in wrote.values()):
                    raise ProtocolError('MMA of stage {} finds activations {} and weights {}'.format(i, self.act_content[s], wrote))
                self.mma_reading[s] = i

                def done(s=s, i=i):
                    if self.act_content[s] != i:
                        raise ProtocolError('stage {} was overwritten under the tensor core'.format(i))
                    del self.mma_reading[s]
                    self.conv_content[s] = dict()
                    self.slot_free[s].arrive()

                self.commits.append(done)
                yield None
                i += 1

            def finished(buf=buf, t=t):
                self.acc_content[buf] = ('done', t)
                self.acc_full[buf].arrive()

            self.commits.append(finished)
            yield None

    def epilogue(self, _warp: int) -> Generator[Wait, None, None]:
        for t in range(self.tiles):
            buf, acc_use = t & 1, t >> 1
            ok = yield from stays(lambda buf=buf, p=acc_use & 1: self.acc_full[buf].test(p), self.epilogue_barrier if self.cfg.epilogue_agrees else None)
            if not ok:
                return
            if self.acc_content[buf] != ('done', t):
                raise ProtocolError('epilogue of tile {} reads an accumulator holding {}'.format(t, self.acc_content[buf]))
            yield None
            for _ in range(2):   # a block is complete; its staging buffer may be overwritten
                yield self.epilogue_barrier.come()[1]
            if self.acc_content[buf] != ('done', t):
                raise ProtocolError('accumulator of tile {} was overwritten while being read'.format(t))
            self.acc_empty[buf].arrive()
            yield None

    def roles(self):
        c = self.cfg
        agents: List[Generator[Wait, None, None]] = [self.producer(), self.mma()]
        agents += [self.converter(g, w) for g in range(c.conv_groups) for w in range(c.group_warps)]
        agents += [self.epilogue(w) for w in range(4)]
        return agents


@dataclass
class TensorMemoryConfig:
    """The kernel on SM pairs (ctas = 2) or the mid-M kernel (ctas = 1), whose weight stands in tensor memory."""
    ctas: int
    raw_slots: int
    act_slots: int
    w_slots: int
    n_acc: int
    conv_groups: int
    group_warps: int
    epi_groups: int               # 0: no epilogue warps, every role waits for the one accumulator at the end
    epilogue_agrees: bool = True
    drain_on_exit: bool = True


def _constants(text: str) -> Dict[str, int]:
    """The kernel's integer constants, each an expression of the ones above it."""
    known: Dict[str, int] = {}
    for group in re.findall(r'^constexpr (?:int|uint32_t) ([^;]+);', text, re.M):
        for name, value in re.findall(r'(\w+) = ([^,]+)', group):
            try:
                known[name] = int(eval(value.replace('/', '//'), {}, known))
            except NameError:
                pass
    return known


def pair_config_from_source(tm: int) -> TensorMemoryConfig:
    """As launch_pair sets the kernel up for tiles of `tm` rows."""
    text = open(os.path.join(KERNELS, 'qlinear_pair.cu')).read()
    k = _constants(text)
    n_acc = 2 if 2 * tm + 4 * 32 <= k['TMEM_COLS'] else 1
    return TensorMemoryConfig(ctas=2, raw_slots=k['RAW_SLOTS'], act_slots=min(k['ACT_RING_BYTES'] // (tm // 2 * k['BK'] * 2), k['MAX_SLOTS']) & ~1,
                              w_slots=min((k['TMEM_COLS'] - n_acc * tm) // 32, k['MAX_W_SLOTS']) & ~1, n_acc=n_acc, conv_groups=k['CONV_GROUPS'],
                              group_warps=k['GROUP_WARPS'], epi_groups=k['EPI_GROUPS'], epilogue_agrees=_epilogue_agrees(text))


def mid_config_from_source(tm: int) -> TensorMemoryConfig:
    """As launch_mid sets the kernel up for tiles of `tm` rows."""
    k = _constants(open(os.path.join(KERNELS, 'qlinear_mid.cu')).read())
    act_slots = (k['CTA_SMEM'] - 1024 - k['RAW_SLOTS'] * k['RAW_BYTES']) // (tm * k['BK'] * 2)
    return TensorMemoryConfig(ctas=1, raw_slots=k['RAW_SLOTS'], act_slots=min(act_slots, k['MAX_SLOTS']), w_slots=k['W_SLOTS'], n_acc=1, conv_groups=k['CONV_GROUPS'],
                              group_warps=k['GROUP_WARPS'], epi_groups=0)


class TensorMemoryPipeline(Scheduler):
    def __init__(self, cfg: TensorMemoryConfig, tiles: int, k_blocks: int, rng: random.Random):
        super().__init__(rng, cfg.ctas)
        self.cfg, self.tiles, self.stages, self.k_blocks = cfg, tiles, tiles * k_blocks, k_blocks
        c, n = cfg, range(cfg.ctas)

        def ring(name, slots, count):
            return [[Barrier('{}{}[{}]'.format(name, cta, s), count) for s in range(slots)] for cta in n]

        self.raw_full, self.raw_empty = ring('raw_full', c.raw_slots, 1), ring('raw_empty', c.raw_slots, c.group_warps)
        self.act_full, self.act_empty = ring('act_full', c.act_slots, 1), ring('act_empty', c.act_slots, 1)
        self.done, self.acc_full = ring('done', c.w_slots, 1), ring('acc_full', c.n_acc, 1)
        self.ready = ring('ready', c.w_slots, c.ctas * c.group_warps)[0]                    # of the first CTA
        self.acc_empty = ring('acc_empty', c.n_acc, c.ctas * 4 * c.epi_groups)[0]
        self.raw_content = [[None] * c.raw_slots for _ in n]
        self.act_content = [[None] * c.act_slots for _ in n]
        self.w_content = [[{} for _ in range(c.w_slots)] for _ in n]                        # warp -> stage it wrote
        self.acc_content: List = [[None] * c.n_acc for _ in n]
        self.reading: Dict[Tuple[str, int], int] = {}                                       # what the tensor core still reads
        self.group_barriers = [[Meeting(4) for _ in range(c.epi_groups)] for _ in n]
        self.agents: List[Tuple[int, Generator]] = [(0, self.mma())]
        for cta in n:
            self.agents += [(cta, self.producer(cta, 'raw')), (cta, self.producer(cta, 'act'))]
            self.agents += [(cta, self.converter(cta, g, w)) for g in range(c.conv_groups) for w in range(c.group_warps)]
            self.agents += [(cta, self.epilogue(cta, g, w)) for g in range(c.epi_groups) for w in range(4)]
        self.exit = Meeting(len(self.agents))   # the cluster barrier (of one CTA: the CTA's) in front of the teardown
        self.agents = [(cta, self.whole(role)) for cta, role in self.agents]

    def roles(self):
        return [role for _, role in self.agents]

    def cta_of(self, agent: int) -> int:
        return self.agents[agent][0]

    def whole(self, role):
        try:
            yield from role
        except Aborted:
            pass
        if self.cfg.epi_groups == 0:
            yield ('drain', lambda: self.acc_full[0][0].phases_done > 0)   # all MMAs issued have completed
        yield self.exit.come()[1]

    def producer(self, cta: int, what: str):
        full, empty, content = getattr(self, what + '_full')[cta], getattr(self, what + '_empty')[cta], getattr(self, what + '_content')[cta]
        in_flight = [0]
        try:
            for i in range(self.stages):
                s, use = i % len(full), i // len(full)
                if use >= 1:
                    yield lambda s=s, p=(use - 1) & 1: empty[s].test(p)
                full[s].arrive_expect_tx(1)
                in_flight[0] += 1

                def land(s=s, i=i):
                    if what == 'act' and ('act', s) in self.reading:
                        raise ProtocolError('activation tile {} lands in a slot the tensor core still reads'.format(i))
                    content[s] = i
                    in_flight[0] -= 1
                    full[s].complete_tx(1)

                self.copies.append(land)
                yield None
        except Aborted:
            pass
        if self.cfg.drain_on_exit:
            yield ('drain', lambda: in_flight[0] == 0)

    def converter(self, cta: int, group: int, warp: int):
        c = self.cfg
        for i in range(group, self.stages, c.conv_groups):
            r, s, w = i % c.raw_slots, i % c.act_slots, i % c.w_slots
            yield lambda r=r, p=(i // c.raw_slots) & 1: self.raw_full[cta][r].test(p)
            if self.raw_content[cta][r] != i:
                raise ProtocolError('converter group {} reads slot {} for stage {} but it holds {}'.format(group, r, i, self.raw_content[cta][r]))
            yield None
            self.raw_empty[cta][r].arrive()
            if i >= c.w_slots:
                yield lambda w=w, p=(i // c.w_slots - 1) & 1: self.done[cta][w].test(p)
            if ('w', w) in self.reading:
                raise ProtocolError('converter writes weight slot {} while the tensor core reads it'.format(w))
            self.w_content[cta][w][warp] = i
            yield None
            if c.ctas == 2 and warp == 0:   # answers for this CTA's activations
                yield lambda s=s, p=(i // c.act_slots) & 1: self.act_full[cta][s].test(p)
                if self.act_content[cta][s] != i:
                    raise ProtocolError('stage {} is reported with activations {}'.format(i, self.act_content[cta][s]))
            self.ready[w].arrive()
            yield None

    def mma(self):
        try:
            yield from self._mma_loop()
        except Aborted:
            pass
        if self.cfg.epi_groups == 0:
            self.commits.append(self.acc_full[0][0].arrive)
        elif self.cfg.drain_on_exit:
            yield ('drain', lambda: not self.commits)

    def _mma_loop(self):
        c = self.cfg
        for t in range(self.tiles):
            buf, acc_use = t % c.n_acc, t // c.n_acc
            if acc_use >= 1:
                yield lambda buf=buf, p=(acc_use - 1) & 1: self.acc_empty[buf].test(p)
            for cta in range(c.ctas):
                self.acc_content[cta][buf] = ('writing', t)
            for i in range(t * self.k_blocks, (t + 1) * self.k_blocks):
                s, w = i % c.act_slots, i % c.w_slots
                if c.ctas == 1:
                    yield lambda s=s, p=(i // c.act_slots) & 1: self.act_full[0][s].test(p)
                yield lambda w=w, p=(i // c.w_slots) & 1: self.ready[w].test(p)
                for cta in range(c.ctas):
                    if self.act_content[cta][s] != i or self.w_content[cta][w] != {q: i for q in range(c.group_warps)}:
                        raise ProtocolError('MMA of stage {} finds activations {} and weights {}'.format(i, self.act_content[cta][s], self.w_content[cta][w]))
                self.reading[('w', w)] = self.reading[('act', s)] = i

                def finished(s=s, w=w, i=i):
                    if any(content[s] != i for content in self.act_content):
                        raise ProtocolError('stage {} was overwritten under the tensor core'.format(i))
                    del self.reading[('w', w)], self.reading[('act', s)]
                    for cta in range(c.ctas):
                        self.w_content[cta][w] = {}
                        self.done[cta][w].arrive()
                        self.act_empty[cta][s].arrive()

                self.commits.append(finished)
                yield None
            if c.epi_groups > 0:
                def tile_finished(buf=buf, t=t):
                    for cta in range(c.ctas):
                        self.acc_content[cta][buf] = ('done', t)
                        self.acc_full[cta][buf].arrive()

                self.commits.append(tile_finished)
                yield None

    def epilogue(self, cta: int, group: int, _warp: int):
        c, barrier = self.cfg, self.group_barriers[cta][group]
        for t in range(self.tiles):
            buf, acc_use = t % c.n_acc, t // c.n_acc
            ok = yield from stays(lambda buf=buf, p=acc_use & 1: self.acc_full[cta][buf].test(p), barrier if c.epilogue_agrees else None)
            if not ok:
                return
            if self.acc_content[cta][buf] != ('done', t):
                raise ProtocolError('epilogue of tile {} reads an accumulator holding {}'.format(t, self.acc_content[cta][buf]))
            yield None
            if self.acc_content[cta][buf] != ('done', t):
                raise ProtocolError('accumulator of tile {} was overwritten while being read'.format(t))
            self.acc_empty[buf].arrive()
            yield barrier.come()[1]   # the block stands in the staging buffer
