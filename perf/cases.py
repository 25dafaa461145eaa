"""What users of this framework have it compute, as measured cases.

Every case goes through a public entry point on inputs of the shapes and
distributions that the framework's benchmark, tests and synthetic data use:
Gaussian-mixture cells in a local PCA space, negative-binomial log1p(CP10k)
expression, lognormal growth, the reference's default solver keys.

``listed()`` holds the named cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare`` makes what a program holds before the call, ``run`` is the
call, ``work`` its unavoidable traffic and arithmetic, ``exact`` the FP64 result
by plain torch and numpy.
"""
import math

import numpy as np
import torch

import wot_gb300 as wot
from wot_gb300.ot import device as D
from wot_gb300.ot.adjoint import ot_objective
from wot_gb300.ot.batch import prepare_pair, solve_batched
from wot_gb300.ot.implicit import ImplicitCoupling

# The reference's solver defaults (OTModel's ot_config).
SOLVER = {'growth_iters': 1, 'epsilon': 0.05, 'lambda1': 1, 'lambda2': 50, 'epsilon0': 1, 'tau': 10000,
          'scaling_iter': 3000, 'inner_iter_max': 50, 'tolerance': 1e-8, 'max_iter': 1e7, 'batch_size': 5,
          'extra_iter': 1000}


def listed():
    return [
        # A user's own small cost matrix (a few clones or clusters of cells) through the reference's
        # drop-in function, host arrays in and out: launches, waits and copies are all there is.
        {'name': 'user_cost_tiny', 'kind': 'user_cost', 'I': 120, 'J': 150, 'd': 10, 'epsilon': 0.05,
         'lambda1': 1.0, 'growth_iters': 1},
        # The same call at the size of one small day pair, with odd sizes.
        {'name': 'user_cost_ragged', 'kind': 'user_cost', 'I': 1237, 'J': 1511, 'd': 30, 'epsilon': 0.05,
         'lambda1': 1.0, 'growth_iters': 1},
        # A day pair from the host expression matrix to the host map: selection, local PCA, cost, solve, copies.
        {'name': 'expression_pair', 'kind': 'expression', 'I': 2000, 'J': 2500, 'genes': 1000, 'epsilon': 0.05},
        # A day pair of an ordinary experiment, cells already in PCA space on the device.
        {'name': 'points_ordinary', 'kind': 'points', 'I': 5003, 'J': 6007, 'd': 30, 'epsilon': 0.05,
         'lambda1': 1.0, 'growth_iters': 1},
        # The benchmark's own pair: 20000 x 25000 cells, three growth iterations, dense FP64 map.
        {'name': 'points_large', 'kind': 'points', 'I': 20000, 'J': 25000, 'd': 30, 'epsilon': 0.05,
         'lambda1': 1.0, 'growth_iters': 3},
        # No local PCA (local_pca=0): the cost of raw gene space, beyond the tensor-core form's dimensions.
        {'name': 'genes_materialised', 'kind': 'points', 'I': 4001, 'J': 5003, 'd': 200, 'epsilon': 0.05,
         'lambda1': 1.0, 'growth_iters': 1},
        # OTModel's other solver, solver='fixed_iters' with its default iteration counts.
        {'name': 'fixed_iters', 'kind': 'fixed', 'I': 803, 'J': 1001, 'd': 30, 'epsilon': 0.05},
        # A short time course under a parameter sweep in one batched solve, maps kept as potentials.
        {'name': 'course_sweep', 'kind': 'sweep', 'days': 4, 'low': 900, 'high': 2500, 'd': 30, 'items': 5},
        # Ancestors and descendants of 8 cell sets through a large map held as potentials (50 dimensions).
        {'name': 'populations_implicit', 'kind': 'implicit', 'I': 22001, 'J': 30011, 'd': 50, 'k': 8,
         'epsilon': 0.05},
        # The same question asked of dense maps kept on the device, over two day steps each way.
        {'name': 'populations_dense', 'kind': 'dense', 'A': 5003, 'B': 7001, 'C': 6007, 'k': 8},
        # A long-range coupling chained from two day-pair maps in host memory.
        {'name': 'chained_map', 'kind': 'chain', 'A': 2003, 'B': 2500, 'C': 3001},
        # The differentiable objective with respect to both point sets and the growth, forward and backward.
        {'name': 'objective_gradient', 'kind': 'gradient', 'I': 3001, 'J': 3507, 'd': 30, 'epsilon': 0.05},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed kinds: cell numbers spread over their logarithm, any parity."""
    kind = rng.choice(['user_cost', 'expression', 'points', 'points', 'points', 'fixed', 'sweep', 'implicit',
                       'dense', 'chain', 'gradient'])
    eps = rng.choice([0.025, 0.05, 0.075, 0.1])
    if kind == 'user_cost':
        n = _size(rng, 60, 2500)
        return {'kind': kind, 'I': n, 'J': int(n * rng.uniform(0.6, 1.4)), 'd': rng.randint(5, 50), 'epsilon': eps,
                'lambda1': rng.choice([0.3, 1.0, 3.0]), 'growth_iters': rng.randint(1, 2)}
    if kind == 'expression':
        n = _size(rng, 900, 3500)
        return {'kind': kind, 'I': n, 'J': int(n * rng.uniform(0.7, 1.3)), 'genes': rng.randint(800, 1500),
                'epsilon': rng.choice([0.05, 0.075, 0.1])}
    if kind == 'points':
        n = _size(rng, 200, 16000)
        d = rng.choice([rng.randint(5, 30), rng.randint(31, 62), rng.randint(63, 250)])
        return {'kind': kind, 'I': n, 'J': int(n * rng.uniform(0.7, 1.4)), 'd': d, 'epsilon': max(0.05, eps),
                'lambda1': rng.choice([0.3, 1.0, 3.0]), 'growth_iters': 1}
    if kind == 'fixed':
        n = _size(rng, 300, 2500)
        return {'kind': kind, 'I': n, 'J': int(n * rng.uniform(0.7, 1.3)), 'd': rng.randint(5, 50), 'epsilon': eps}
    if kind == 'sweep':
        lo = _size(rng, 300, 1200)
        return {'kind': kind, 'days': rng.randint(3, 5), 'low': lo, 'high': 2 * lo + rng.randint(0, 200),
                'd': rng.randint(10, 50), 'items': rng.randint(2, 5)}
    if kind == 'implicit':
        n = _size(rng, 2000, 25000)
        return {'kind': kind, 'I': n, 'J': int(n * rng.uniform(0.7, 1.3)), 'd': rng.randint(10, 62),
                'k': rng.randint(1, 12), 'epsilon': max(0.05, eps)}
    if kind == 'dense':
        return {'kind': kind, 'A': _size(rng, 400, 7000), 'B': _size(rng, 400, 7000), 'C': _size(rng, 400, 7000),
                'k': rng.randint(1, 20)}
    if kind == 'chain':
        return {'kind': kind, 'A': _size(rng, 200, 3000), 'B': _size(rng, 200, 3000), 'C': _size(rng, 200, 3000)}
    n = _size(rng, 600, 4000)
    return {'kind': kind, 'I': n, 'J': int(n * rng.uniform(0.8, 1.2)), 'd': rng.randint(10, 50), 'epsilon': 0.05}


# --- inputs ---------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _cells(g, sizes, d):
    """FP32 cells of consecutive days: one Gaussian mixture of 10 clusters whose centres drift a little."""
    centres = torch.randn((10, d), generator=g, device='cuda')
    out = []
    for n in sizes:
        k = torch.randint(0, 10, (n,), generator=g, device='cuda')
        out.append(centres[k] + 0.3 * torch.randn((n, d), generator=g, device='cuda'))
        centres = centres + 0.1 * torch.randn((10, d), generator=g, device='cuda')
    return out


def _growth(g, n):
    return torch.exp(0.3 * torch.randn(n, generator=g, device='cuda', dtype=torch.float64))


def _cost64(x, y):
    """Median-normalised squared-Euclidean cost in FP64."""
    x, y = x.double(), y.double()
    C = x.square().sum(1)[:, None] + y.square().sum(1)[None, :] - 2.0 * (x @ y.T)
    C.clamp_(min=0.0)
    return C.div_(_median64(C))


def _median64(C):
    """Mean of the two middle entries, by bisection on counts (no sort of a large matrix)."""
    n = C.numel()
    if n <= 1 << 24:
        s = torch.sort(C.reshape(-1)).values
        return float(0.5 * (s[(n - 1) // 2] + s[n // 2]))

    def kth(k):
        lo, hi = float(C.min()), float(C.max())
        for _ in range(40):
            mid = 0.5 * (lo + hi)
            if int((C <= mid).sum()) > k:
                hi = mid
            else:
                lo = mid
            if hi - lo <= 1e-13 * hi:
                break
        return hi

    return 0.5 * (kth((n - 1) // 2) + kth(n // 2))


def _expression(g, n, genes, clusters=6):
    """log1p(CP10k) of negative-binomial counts (size 2), about 90 % zeros, cells around cluster profiles."""
    log_mu = torch.randn((clusters, genes), generator=g, device='cuda', dtype=torch.float64)
    out = []
    for size in n:
        k = torch.randint(0, clusters, (size,), generator=g, device='cuda')
        mu = 0.035 * torch.exp(log_mu[k] + 0.25 * torch.randn((size, genes), generator=g, device='cuda',
                                                              dtype=torch.float64))
        u = torch.rand((2, size, genes), generator=g, device='cuda', dtype=torch.float64).clamp_(min=1e-300)
        counts = torch.poisson(mu * 0.5 * (-torch.log(u[0]) - torch.log(u[1])), generator=g)
        total = counts.sum(1, keepdim=True).clamp(min=1.0)
        out.append(torch.log1p(counts / total * 1e4))
        log_mu = log_mu + 0.1 * torch.randn((clusters, genes), generator=g, device='cuda', dtype=torch.float64)
    return out


def _dense_map(g, x, y):
    """An FP64 coupling between two days: the entropic kernel at epsilon 0.05 with rows scaled to the growth."""
    T = torch.exp(_cost64(x, y).mul_(-1.0 / 0.05))
    T *= (_growth(g, x.shape[0]) / T.sum(1) / y.shape[0])[:, None]
    return T


def _config(case):
    return dict(SOLVER, **{k: case[k] for k in ('epsilon', 'lambda1', 'growth_iters') if k in case})


def _sweep_items(case):
    """(day pair, configuration) items: the corners and the middle of the epsilon x lambda1 grid."""
    grid = [(0.05, 1.0), (0.025, 0.3), (0.1, 3.0), (0.025, 3.0), (0.1, 0.3)][:case['items']]
    return [(p, dict(SOLVER, epsilon=e, lambda1=l)) for p in range(case['days'] - 1) for e, l in grid]


def _inputs(case, seed):
    """The raw inputs of a case, from the seed alone."""
    g = _gen(seed)
    kind = case['kind']
    if kind == 'expression':
        x, y = _expression(g, (case['I'], case['J']), case['genes'])
        return {'x': x, 'y': y, 'growth': _growth(g, case['I'] + case['J'])}
    if kind == 'sweep':
        last = case['days'] - 1
        sizes = [int(case['low'] * (case['high'] / case['low']) ** (t / last)) for t in range(case['days'])]
        days = _cells(g, sizes, case['d'])
        return {'days': days, 'growth': [_growth(g, n) for n in sizes[:-1]]}
    if kind in ('dense', 'chain'):
        a, b, c = _cells(g, (case['A'], case['B'], case['C']), 30)
        out = {'T0': _dense_map(g, a, b), 'T1': _dense_map(g, b, c)}
        if kind == 'dense':
            k = case['k']
            out['pa'] = (torch.rand((k, case['A']), generator=g, device='cuda') < 0.05).double().cpu().numpy()
            out['pc'] = (torch.rand((k, case['C']), generator=g, device='cuda') < 0.05).double().cpu().numpy()
            out['pa'][:, 0] = out['pc'][:, 0] = 1.0
        else:
            out['order'] = torch.randperm(case['B'], generator=g, device='cuda')
        return out
    x, y = _cells(g, (case['I'], case['J']), case['d'])
    out = {'x': x, 'y': y, 'growth': _growth(g, case['I'])}
    if kind in ('user_cost', 'fixed'):
        out['C'] = _cost64(x, y)
    if kind == 'gradient':
        out['log_g'] = torch.log(out['growth'])
    if kind == 'implicit':
        # Potentials of a coupling whose rows carry the growth and whose columns are already reweighted.
        eps, k = case['epsilon'], case['k']
        s = 1.0 / _median64(_cost64(x[:4000], y[:4000]))
        v = eps * 0.3 * torch.randn(case['J'], generator=g, device='cuda', dtype=torch.float64)
        u = torch.cat([-eps * torch.logsumexp(v / eps - (s / eps) * _sq(xb, y), dim=1) for xb in x.split(2048)])
        out.update(s=s, v=v, u=u + eps * torch.log(out['growth'] * case['J']),
                   pj=(torch.rand((k, case['J']), generator=g, device='cuda') < 0.02).double(),
                   pi=(torch.rand((k, case['I']), generator=g, device='cuda') < 0.02).double())
        out['pj'][:, 0] = out['pi'][:, 0] = 1.0
    return out


def _sq(x, y):
    """Squared distances in FP64."""
    x, y = x.double(), y.double()
    return (x.square().sum(1)[:, None] + y.square().sum(1)[None, :] - 2.0 * (x @ y.T)).clamp_(min=0.0)


# --- prepare and run ----------------------------------------------------------------

def prepare(case, seed):
    data = _inputs(case, seed)
    kind = case['kind']
    state = {'case': case, 'config': _config(case)}
    if kind in ('user_cost', 'fixed'):
        state.update(C=data['C'].cpu().numpy(), G=data['growth'].cpu().numpy())
    elif kind == 'expression':
        X = torch.cat([data['x'], data['y']]).cpu().numpy()
        obs = wot.Frame({'day': np.repeat([0.0, 1.0], [case['I'], case['J']]),
                         'cell_growth_rate': data['growth'].cpu().numpy()},
                        index=np.array(['c%d' % i for i in range(X.shape[0])]))
        state['model'] = wot.OTModel(wot.Dataset(X, obs), epsilon=case['epsilon'])
    elif kind == 'points':
        state.update(x=data['x'], y=data['y'], G=data['growth'])
    elif kind == 'sweep':
        pairs = [prepare_pair(D.default_cost(a, b), G)
                 for a, b, G in zip(data['days'][:-1], data['days'][1:], data['growth'])]
        state.update(pairs=pairs, items=_sweep_items(case))
    elif kind == 'implicit':
        state.update(map=ImplicitCoupling(data['u'], data['v'], case['epsilon'], data['s'], -math.log(case['J']),
                                          X=data['x'], Y=data['y']), pi=data['pi'], pj=data['pj'])
    elif kind in ('dense', 'chain'):
        names = [['%s%d' % (c, i) for i in range(case[c])] for c in 'ABC']
        T0, T1 = data['T0'], data['T1']
        if kind == 'chain':
            # maps read from files: the second one lists the shared day's cells in its own order
            order = data['order']
            T0, T1 = T0.cpu().numpy(), T1[order].cpu().numpy()
            rows1 = [names[1][i] for i in order.tolist()]
        else:
            rows1 = names[1]
        maps = {(0.0, 1.0): wot.Dataset(T0, wot.Frame(index=names[0]), wot.Frame(index=names[1])),
                (1.0, 2.0): wot.Dataset(T1, wot.Frame(index=rows1), wot.Frame(index=names[2]))}
        meta = wot.Frame({'day': np.repeat([0.0, 1.0, 2.0], [case[c] for c in 'ABC'])},
                         index=np.array([c for n in names for c in n]))
        state['model'] = wot.TransportMapModel(maps, meta)
        if kind == 'dense':
            state.update(start=[wot.Population(0.0, p) for p in data['pa']],
                         end=[wot.Population(2.0, p) for p in data['pc']])
    else:
        state.update(x=data['x'].requires_grad_(), y=data['y'].requires_grad_(),
                     log_g=data['log_g'].requires_grad_())
    return state


def run(state):
    case, cfg = state['case'], state['config']
    kind = case['kind']
    if kind == 'user_cost':
        tmap, learned = wot.ot.compute_transport_matrix(wot.ot.optimal_transport_duality_gap, C=state['C'],
                                                        G=state['G'], **cfg)
        return {'tmap': tmap, 'learned': learned}
    if kind == 'fixed':
        return wot.ot.transport_stablev2(state['C'], G=state['G'], **cfg)
    if kind == 'expression':
        tmap = state['model'].compute_transport_map(0.0, 1.0)
        return {'tmap': tmap.X, 'growth': [tmap.obs[c] for c in sorted(tmap.obs.columns)]}
    if kind == 'points':
        res = D.solve(D.default_cost(state['x'], state['y']), state['G'], cfg, form='auto')
        return {'tmap': res.tmap, 'learned': res.learned_growth, 'row_sums': res.row_sums}
    if kind == 'sweep':
        return [[m.u_bar, m.v_bar, m.row_sums] for m in solve_batched(state['pairs'], state['items'])]
    if kind == 'implicit':
        return {'back': state['map'].pull_back(state['pj']), 'forward': state['map'].push_forward(state['pi'])}
    if kind == 'dense':
        back = state['model'].pull_back(*state['end'], to_time=0.0, as_list=True)
        forward = state['model'].push_forward(*state['start'], to_time=2.0, as_list=True)
        return {'back': np.stack([p.p for p in back]), 'forward': np.stack([p.p for p in forward])}
    if kind == 'chain':
        return state['model'].get_coupling(0.0, 2.0).X
    leaves = [state['x'], state['y'], state['log_g']]
    objective = ot_objective(*leaves, epsilon=case['epsilon'])
    return [objective.detach(), *torch.autograd.grad(objective, leaves)]


# --- work ---------------------------------------------------------------------------

def _iterations(case):
    """Sinkhorn iterations of one duality-gap solve, as they come out at the default tolerance."""
    return 450.0 * (0.05 / case.get('epsilon', 0.05)) * (0.5 + 0.5 * min(3.0, case.get('lambda1', 1.0)))


def work(case):
    """Each input read and each output written once; per Sinkhorn iteration two half-steps, each a multiply-add,
    an exponential and a sum per cost entry (a fixed solve's counts, else the usual ones)."""
    kind = case['kind']
    if kind in ('dense', 'chain'):
        a, b, c = case['A'], case['B'], case['C']
        if kind == 'chain':
            return {'bytes': 8.0 * (a * b + b * c + a * c), 'flops': 2.0 * a * b * c}
        k = case['k']
        return {'bytes': 2 * 8.0 * (a * b + b * c) + 32.0 * k * (a + b + c), 'flops': 4.0 * k * (a * b + b * c)}
    if kind == 'sweep':
        n = math.sqrt(case['low'] * case['high'])
        maps = (case['days'] - 1) * case['items']
        return {'bytes': (case['days'] - 1) * 4.0 * n * n + maps * 24.0 * n, 'flops': maps * 900.0 * 2 * 4 * n * n}
    I, J = case['I'], case['J']
    d = case.get('d', 30)
    if kind == 'implicit':
        return {'bytes': 2 * (4.0 * d * (I + J) + 8.0 * (I + J) + 8.0 * case['k'] * (I + J)),
                'flops': 2.0 * I * J * (2 * d + 2 + 2 * case['k'])}
    if kind == 'fixed':
        return {'bytes': 16.0 * I * J + 8.0 * I, 'flops': 4000.0 * 2 * 4 * I * J}
    if kind == 'user_cost':
        return {'bytes': 16.0 * I * J + 16.0 * I, 'flops': case['growth_iters'] * _iterations(case) * 2 * 4 * I * J}
    if kind == 'expression':
        return {'bytes': 8.0 * (I + J) * case['genes'] + 8.0 * I * J,
                'flops': _iterations(case) * 2 * 4 * I * J + 17 * 2 * 40 * 0.1 * (I + J) * case['genes']}
    if kind == 'points':
        return {'bytes': 4.0 * d * (I + J) + 8.0 * I + 8.0 * I * J,
                'flops': 2.0 * d * I * J + case['growth_iters'] * _iterations(case) * 2 * 4 * I * J}
    return {'bytes': 12.0 * d * (I + J) + 24.0 * I,
            'flops': 2.0 * d * I * J + (_iterations(case) + 400) * 2 * 4 * I * J + 2 * (4.0 * d + 8) * I * J}


# --- the FP64 result -------------------------------------------------------------------

class _Sinkhorn64:
    """The reference's stabilised unbalanced Sinkhorn on a dense FP64 cost."""

    def __init__(self, C, G, cfg):
        self.C, self.p, self.cfg = C, G, cfg
        self.I, self.J = C.shape
        self.q = G.mean()
        self.u, self.v = torch.zeros_like(G), torch.zeros(self.J, dtype=torch.float64, device=C.device)
        self.a, self.b = torch.ones_like(self.u), torch.ones_like(self.v)
        self.K = torch.empty_like(C)

    def kernel(self):
        torch.sub(self.u[:, None], self.C, out=self.K)
        self.K.add_(self.v[None, :]).mul_(1.0 / self.eps).exp_()

    def set_epsilon(self, old, eps):
        self.absorb(old)
        self.eps = eps
        self.kernel()

    def absorb(self, eps):
        self.u, self.v = self.u + eps * torch.log(self.a), self.v + eps * torch.log(self.b)
        self.a, self.b = torch.ones_like(self.a), torch.ones_like(self.b)

    def step(self, check=True):
        l1, l2, eps = self.cfg['lambda1'], self.cfg['lambda2'], self.eps
        self.old = (self.a, self.b)
        self.a = (self.p / (self.K @ (self.b / self.J))) ** (l1 / (l1 + eps)) * torch.exp(-self.u / (l1 + eps))
        self.b = (self.q / (self.K.T @ (self.a / self.I))) ** (l2 / (l2 + eps)) * torch.exp(-self.v / (l2 + eps))
        if check and float(torch.maximum(self.a.max(), self.b.max())) > self.cfg['tau']:
            self.absorb(eps)
            self.kernel()

    def gap(self, sum_k0):
        """Relative duality gap, the entropy taken over the marginals (R log R = R (u + v - C) / eps)."""
        l1, l2, eps = self.cfg['lambda1'], self.cfg['lambda2'], self.eps
        x, y = self.a * (self.K @ (self.b / self.J)), self.b * (self.K.T @ (self.a / self.I))
        ub, vb = self.u + eps * torch.log(self.a), self.v + eps * torch.log(self.b)
        fx = (x * torch.log(x / self.p) - x + self.p).mean() * l1
        fy = (y * torch.log(y / self.q) - y + self.q).mean() * l2
        gx = (self.p * (torch.exp(-ub / l1) - 1)).mean() * l1
        gy = (self.q * (torch.exp(-vb / l2) - 1)).mean() * l2
        lin = (ub * x).mean() + (vb * y).mean()
        primal = fx + fy + lin + eps * (sum_k0 / (self.I * self.J) - x.mean())
        return float((fx + fy + lin + gx + gy) / primal.abs())

    def solve(self):
        cfg = self.cfg
        factor = math.exp(-math.log(cfg['epsilon']) / 5)
        eps = cfg['epsilon0'] * factor
        for stage in range(6):
            old, eps = eps, eps / factor
            self.set_epsilon(old, eps)
            gap = math.inf
            if stage == 5:
                sum_k0 = sum(float(torch.exp(c * (-1.0 / eps)).sum()) for c in self.C.split(1024))
            while gap > (cfg['tolerance'] if stage == 5 else 1e-6):
                for _ in range(cfg['batch_size'] if stage == 5 else 5):
                    self.step()
                if stage == 5:
                    gap = self.gap(sum_k0)
                else:
                    eu, ev = torch.exp(self.u / eps), torch.exp(self.v / eps)
                    gap = max(float(torch.linalg.norm((n - o) * e) / (1 + torch.linalg.norm(n * e)))
                              for n, o, e in ((self.a, self.old[0], eu), (self.b, self.old[1], ev)))
        return self

    def fixed(self):
        cfg = self.cfg
        eps = cfg['epsilon0']
        self.set_epsilon(0.0, eps)
        since = index = 0
        for _ in range(cfg['scaling_iter']):
            self.step()
            since += 1
            if since == cfg['inner_iter_max']:
                index, since = index + 1, 0
                old, eps = eps, (cfg['epsilon0'] - cfg['epsilon']) * math.exp(-index) + cfg['epsilon']
                self.set_epsilon(old, eps)
        for _ in range(cfg['extra_iter']):
            self.step(check=False)
        return self

    def potentials(self):
        return self.u + self.eps * torch.log(self.a), self.v + self.eps * torch.log(self.b)

    def map(self):
        """The returned coupling, in place of K."""
        return self.K.mul_(self.a[:, None]).mul_(self.b[None, :] / self.J)


def _maps64(C, G, cfg):
    """(map, the growth each iteration started from) of the growth-iteration driver."""
    learned = []
    for _ in range(cfg['growth_iters']):
        learned.append(G)
        T = _Sinkhorn64(C, G, cfg).solve().map()
        G = T.sum(1)
    return T, learned


def _pca64(x, y):
    """30 singular-value-scaled coordinates of two days: the randomized range finder of the reference's PCA
    (seed 58951, 10 extra directions) on the double-centred cells x genes matrix, by Householder QR."""
    k, n1 = 30, x.shape[0]
    T = torch.cat([x, y])
    T = T - T.mean(0)[None, :]
    T = T - T.mean(1)[:, None]
    n, p = T.shape
    M = T if p < n else T.T
    Q = torch.as_tensor(np.random.RandomState(58951).normal(size=(min(n, p), k + 10)), device='cuda')
    for _ in range(7 if k < 0.1 * min(n, p) else 4):
        Q = torch.linalg.qr(M @ Q)[0]
        Q = torch.linalg.qr(M.T @ Q)[0]
    Q = torch.linalg.qr(M @ Q)[0]
    U, s, Vt = torch.linalg.svd(Q.T @ M, full_matrices=False)
    comp = (Q @ U)[:, :k] if p < n else Vt[:k].T
    comp = comp * s[:k][None, :]
    return comp[:n1], comp[n1:]


def exact(case, seed):
    data = _inputs(case, seed)
    kind, cfg = case['kind'], _config(case)
    if kind == 'user_cost':
        T, learned = _maps64(data['C'], data['growth'], cfg)
        return {'tmap': T, 'learned': learned}
    if kind == 'fixed':
        return _Sinkhorn64(data['C'], data['growth'], cfg).fixed().map()
    if kind == 'expression':
        T, learned = _maps64(_cost64(*_pca64(data['x'], data['y'])), data['growth'][:case['I']], cfg)
        return {'tmap': T, 'growth': learned + [T.sum(1)]}
    if kind == 'points':
        T, learned = _maps64(_cost64(data['x'], data['y']), data['growth'], cfg)
        return {'tmap': T, 'learned': learned, 'row_sums': T.sum(1)}
    if kind == 'sweep':
        costs = [_cost64(a, b) for a, b in zip(data['days'][:-1], data['days'][1:])]
        out = []
        for p, conf in _sweep_items(case):
            s = _Sinkhorn64(costs[p], data['growth'][p], conf).solve()
            out.append([*s.potentials(), s.map().sum(1)])
        return out
    if kind == 'implicit':
        eps, s = case['epsilon'], data['s']

        def apply(P, src, tgt, a, b):
            rows = []
            for xb, ab in zip(src.split(2048), a.split(2048)):
                rows.append(torch.exp((ab[:, None] + b[None, :] - s * _sq(xb, tgt)) / eps) @ P.T)
            out = torch.cat(rows).T
            return out / out.sum(1, keepdim=True)

        return {'back': apply(data['pj'], data['x'], data['y'], data['u'], data['v']),
                'forward': apply(data['pi'], data['y'], data['x'], data['v'], data['u'])}
    if kind == 'dense':
        back = torch.as_tensor(data['pc'], device='cuda')
        forward = torch.as_tensor(data['pa'], device='cuda')
        for T in (data['T1'], data['T0']):
            back = back @ T.T
            back = back / back.sum(1, keepdim=True)
        for T in (data['T0'], data['T1']):
            forward = forward @ T
            forward = forward / forward.sum(1, keepdim=True)
        return {'back': back, 'forward': forward}
    if kind == 'chain':
        return data['T0'] @ data['T1']
    # the envelope gradient at the potentials of the solve and 400 further iterations
    x, y, p = data['x'].double(), data['y'].double(), data['growth']
    cfg = dict(cfg, growth_iters=1)
    C = _sq(x, y)
    scale = 1.0 / _median64(C)
    C.mul_(scale)
    s = _Sinkhorn64(C, p, cfg).solve()
    s.set_epsilon(s.eps, s.eps)
    for _ in range(400):
        s.step()
    u, v = s.potentials()
    I, J, eps = s.I, s.J, s.eps
    l1, l2 = cfg['lambda1'], cfg['lambda2']
    W = torch.exp((u[:, None] + v[None, :] - C) / eps) - torch.exp(-C / eps)
    gx = 2 * scale / (I * J) * (x * W.sum(1)[:, None] - W @ y)
    gy = 2 * scale / (I * J) * (y * W.sum(0)[:, None] - W.T @ x)
    eu, ev = torch.exp(-u / l1) - 1, torch.exp(-v / l2) - 1
    objective = -l1 * (p * eu).mean() - l2 * s.q * ev.mean() - eps * W.sum() / (I * J)
    gp = -l1 * eu / I - l2 * ev.mean() / I
    return [objective, gx, gy, gp * p]
