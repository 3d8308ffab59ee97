"""Workloads of the K-FAC framework, for timing and for comparing results.

A case is a dict of plain values.  ``prepare`` makes what a training program
holds before the call (model, optimizer, plans, inputs), ``run`` is one pass
through the public entry points:

``step``     ``KFAC.update(lossfun, x, t)``: forward, backward, factors,
             inverses, preconditioned update of a whole network;
``block``    the per-layer interface (hooks, ``update_cov_emas``,
             ``update_invs``, ``update_kfgrads``) of one layer, as a program
             with its own loop or a single curvature layer drives it;
``factors``  the grouped build of all factors of a network from its
             activations and output gradients (``ops.factor_group``,
             ``ops.bn_sample_grads_group``), running average included;
``pairs``    damped inverses of prebuilt factor pairs and the preconditioned
             momentum update (``ops.InversePlanSet``, ``ops.precondition``);
``wire``     packing gradients and factors into the exchange buffer and
             unpacking the sum of two ranks' buffers.
"""

import functools
import math

import torch
from torch import nn
import torch.nn.functional as F

import chainerkfac_b200 as ck
from chainerkfac_b200 import links
from chainerkfac_b200 import ops
from chainerkfac_b200.optimizers import fisher_blocks as FB

DEVICE = 'cuda'
MOMENTUM = 0.9
# The very end of a decaying schedule: passes are repeated on the same batch
# and results are compared, and a deep network with TF32 convolutions answers
# a change in the last bit of a weight with gradients that differ by percents.
LR = 1e-12


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # smallest calls: the per-layer interface on a classifier's last
        # layer, where launches and host work are everything
        dict(name='block_linear_small', kind='block', layer='linear',
             cin=84, cout=10, batch=64, bias=True, damping=1e-3),
        # an odd-sized convolution with bias through the same interface
        dict(name='block_conv_odd', kind='block', layer='conv', cin=37,
             cout=53, k=3, stride=1, pad=1, image=15, batch=33, bias=True,
             channels_last=False, damping=1e-2),
        # the fully connected network of the MNIST example
        dict(name='step_mlp', kind='step', net='mlp', image=784,
             widths='1000-1000', classes=10, batch=128, acc=1, decay=0.99,
             damping=1e-3, channels_last=False),
        # a small convolutional network with odd widths and image
        dict(name='step_cnn_odd', kind='step', net='cnn', image=29,
             widths='21-45-187', classes=10, batch=100, acc=1, decay=0.95,
             damping=1e-2, channels_last=False),
        # CIFAR ResNet-18, BatchNormalization blocks dense (the batch is as
        # large as the layers are wide)
        dict(name='step_resnet18_cifar', kind='step', net='resnet18',
             image=32, widths='64', classes=10, batch=128, acc=1, decay=0.99,
             damping=1e-2, channels_last=False),
        # ResNet-50 at 32 images per GPU, the framework's headline network
        dict(name='step_resnet50', kind='step', net='resnet50', image=224,
             widths='64', classes=1000, batch=32, acc=1, decay=0.9,
             damping=2.5e-4, channels_last=True),
        # gradient and factor accumulation: four micro-steps per update
        dict(name='accumulate_resnet18', kind='step', net='resnet18',
             image=32, widths='64', classes=10, batch=32, acc=4, decay=0.9,
             damping=1e-2, channels_last=True),
        # factor build of every layer of ResNet-50, NCHW
        dict(name='factors_resnet50', kind='factors', net='resnet50',
             image=224, widths='64', classes=1000, batch=32, decay=0.9,
             channels_last=False),
        # the 54 factor pairs of ResNet-50: inverse and precondition alone
        dict(name='pairs_resnet50', kind='pairs', net='resnet50', image=224,
             widths='64', classes=1000, damping=2.5e-4),
        # one owner's share at 8 GPUs: a single largest 3x3 layer
        dict(name='pairs_largest_layer', kind='pairs', dims='4608x512',
             damping=2.5e-4),
        # many small odd layers (widths that are no multiple of a tile)
        dict(name='pairs_small_odd', kind='pairs',
             dims='27x33,298x33,298x47,424x61,550x61,550x95,856x95,96x33,'
                  '62x129,130x211,212x10,785x301,302x77,78x10',
             damping=1e-3),
        # exchange buffers of ResNet-50, as the communicators move them
        dict(name='wire_resnet50', kind='wire', net='resnet50', image=224,
             widths='64', classes=1000, wire='float32', ranks=2),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['block', 'step', 'step', 'step', 'factors', 'pairs',
                       'pairs', 'wire'])
    if kind == 'block':
        layer = rng.choice(['linear', 'conv', 'bn'])
        c = dict(kind=kind, layer=layer, bias=rng.random() < 0.5,
                 damping=rng.choice([1e-3, 1e-2]))
        if layer == 'linear':
            c.update(cin=_between(rng, 10, 2048), cout=_between(rng, 10, 1000),
                     batch=_between(rng, 8, 512))
        else:
            c.update(cout=_between(rng, 8, 512), image=_between(rng, 5, 56),
                     batch=_between(rng, 4, 64),
                     channels_last=rng.random() < 0.5)
        if layer == 'conv':
            k = rng.choice([1, 3, 3, 5])
            c.update(cin=_between(rng, 3, 256), k=k, pad=k // 2,
                     stride=rng.choice([1, 1, 2]))
        return c
    if kind == 'pairs' and rng.random() < 0.75:
        top = rng.choice([300, 1200, 4608])
        dims, cost = [], 0.0
        for _ in range(_between(rng, 1, 54)):
            a, g = _between(rng, 10, top), _between(rng, 10, min(top, 2048))
            cost += a ** 3 + g ** 3
            if dims and cost > 3e11:
                break
            dims.append('%dx%d' % (a, g))
        return dict(kind=kind, dims=','.join(dims),
                    damping=rng.choice([2.5e-4, 1e-3, 1e-2]))
    c = dict(kind=kind, classes=rng.choice([10, 100, 1000]))
    net = rng.choice(['mlp', 'cnn', 'resnet18', 'resnet50'])
    c['net'] = net
    if net == 'mlp':
        c.update(image=_between(rng, 20, 2000), batch=_between(rng, 8, 1024),
                 widths='-'.join(str(_between(rng, 30, 2000))
                                 for _ in range(rng.randint(1, 3))))
    elif net == 'cnn':
        c.update(image=rng.randint(16, 64), batch=_between(rng, 8, 256),
                 widths='%d-%d-%d' % (rng.randint(8, 96), rng.randint(16, 128),
                                      _between(rng, 32, 512)))
    elif net == 'resnet18':
        c.update(image=rng.randint(24, 40), batch=_between(rng, 16, 128),
                 widths=str(rng.choice([16, 24, 32, 48, 64])))
    else:
        c.update(image=rng.randint(64, 224), batch=_between(rng, 4, 32),
                 widths=rng.choice(['32', '48', '64']))
    if kind in ('step', 'factors'):
        c.update(decay=rng.choice([0.9, 0.95, 0.99]),
                 channels_last=net != 'mlp' and rng.random() < 0.5)
    if kind == 'step':
        c.update(acc=rng.choice([1, 1, 1, 2]) if net != 'resnet50' else 1,
                 damping=rng.choice([1e-3, 1e-2]) if net == 'mlp' else 1e-2)
    elif kind == 'pairs':
        c.pop('batch')
        c['damping'] = rng.choice([2.5e-4, 1e-3])
    elif kind == 'wire':
        c.pop('batch')
        c.update(ranks=rng.choice([1, 2, 4]),
                 wire=rng.choice(['float32', 'float32', 'bfloat16',
                                  'float16']))
    return c


# --------------------------------------------------------------- the networks

class Residual(nn.Module):
    """Basic (two 3x3) or bottleneck (1x1, 3x3, 1x1) block with
    BatchNormalization after every convolution."""

    def __init__(self, cin, mid, stride, bottleneck):
        super().__init__()
        cout = mid * 4 if bottleneck else mid
        geo = [(cin, mid, 1, 1), (mid, mid, 3, stride), (mid, cout, 1, 1)] \
            if bottleneck else [(cin, mid, 3, stride), (mid, mid, 3, 1)]
        self.conv = nn.ModuleList(
            nn.Conv2d(a, b, k, s, k // 2, bias=False) for a, b, k, s in geo)
        self.bn = nn.ModuleList(nn.BatchNorm2d(g[1]) for g in geo)
        self.short = None
        if stride != 1 or cin != cout:
            self.short = nn.Sequential(
                nn.Conv2d(cin, cout, 1, stride, bias=False),
                nn.BatchNorm2d(cout))

    def forward(self, x):
        h = x
        for i, (conv, bn) in enumerate(zip(self.conv, self.bn)):
            h = bn(conv(h))
            if i + 1 < len(self.conv):
                h = F.relu(h)
        return F.relu(h + (x if self.short is None else self.short(x)))


def network(case):
    w = [int(v) for v in case['widths'].split('-')]
    if case['net'] == 'mlp':
        seq, d = [], case['image']
        for v in w:
            seq += [nn.Linear(d, v), nn.ReLU()]
            d = v
        return nn.Sequential(*seq, nn.Linear(d, case['classes']))
    if case['net'] == 'cnn':
        return nn.Sequential(
            nn.Conv2d(1, w[0], 5, padding=2), nn.ReLU(), nn.MaxPool2d(2),
            nn.Conv2d(w[0], w[1], 3, padding=1), nn.BatchNorm2d(w[1]),
            nn.ReLU(), nn.AdaptiveAvgPool2d(4), nn.Flatten(),
            nn.Linear(w[1] * 16, w[2]), nn.ReLU(),
            nn.Linear(w[2], case['classes']))
    bottleneck = case['net'] == 'resnet50'
    if bottleneck:
        stem = [nn.Conv2d(3, w[0], 7, 2, 3), nn.BatchNorm2d(w[0]), nn.ReLU(),
                nn.MaxPool2d(3, 2, 1)]
        depth = (3, 4, 6, 3)
    else:
        stem = [nn.Conv2d(3, w[0], 3, 1, 1, bias=False),
                nn.BatchNorm2d(w[0]), nn.ReLU()]
        depth = (2, 2, 2, 2)
    body, cin = [], w[0]
    for stage, blocks in enumerate(depth):
        mid = w[0] << stage
        for b in range(blocks):
            body.append(Residual(cin, mid, 2 if b == 0 and stage else 1,
                                 bottleneck))
            cin = mid * 4 if bottleneck else mid
    return nn.Sequential(*stem, *body, nn.AdaptiveAvgPool2d(1), nn.Flatten(),
                         nn.Linear(cin, case['classes']))


def _input_shape(case, batch):
    if case['net'] == 'mlp':
        return (batch, case['image'])
    c = 1 if case['net'] == 'cnn' else 3
    return (batch, c, case['image'], case['image'])


@functools.lru_cache(maxsize=64)
def _trace(net, image, widths, classes, batch):
    """Layer table of a network: shapes only, nothing is computed."""
    case = dict(net=net, image=image, widths=widths, classes=classes)
    model, table = network(case).to('meta'), []

    def hook(m, inp, out):
        x = tuple(inp[0].shape)
        if isinstance(m, nn.Conv2d):
            k = m.kernel_size[0]
            table.append(dict(
                kind='conv', x=x, gy=tuple(out.shape), k=k,
                stride=m.stride[0], pad=m.padding[0],
                bias=m.bias is not None,
                dA=x[1] * k * k + int(m.bias is not None),
                dG=out.shape[1], rows=x[0] * out.shape[2] * out.shape[3]))
        elif isinstance(m, nn.Linear):
            table.append(dict(
                kind='linear', x=x, gy=tuple(out.shape), bias=True,
                dA=x[1] + 1, dG=out.shape[1], rows=x[0]))
        elif isinstance(m, nn.BatchNorm2d):
            table.append(dict(kind='bn', x=x, gy=x, c=x[1], rows=x[0],
                              bias=True))
    for m in model.modules():
        m.register_forward_hook(hook)
    model(torch.empty(_input_shape(case, batch), device='meta'))
    return table


def table_of(case):
    return _trace(case['net'], case['image'], case['widths'],
                  case['classes'], case.get('batch', 2))


def pair_dims(case):
    if 'dims' in case:
        return [tuple(int(v) for v in p.split('x'))
                for p in case['dims'].split(',')]
    return [(l['dA'], l['dG']) for l in table_of(case) if l['kind'] != 'bn']


# ------------------------------------------------------------------- helpers

def _flat_views(shapes):
    """One buffer and views of it with the given shapes (256-byte steps)."""
    sizes = [math.prod(s) for s in shapes]
    step = [-(-n // 64) * 64 for n in sizes]
    flat = torch.zeros(max(sum(step), 1), device=DEVICE)
    views, o = [], 0
    for s, n, st in zip(shapes, sizes, step):
        views.append(flat[o:o + n].view(s))
        o += st
    return flat, views


def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _layout(t, case):
    return t.contiguous(memory_format=torch.channels_last) \
        if case.get('channels_last') and t.dim() == 4 else t


# ------------------------------------------------------------------- prepare

def prepare(case, seed):
    return dict(step=_prepare_step, block=_prepare_block,
                factors=_prepare_factors, pairs=_prepare_pairs,
                wire=_prepare_wire)[case['kind']](case, seed)


def _prepare_step(case, seed):
    g = _gen(seed)
    with torch.random.fork_rng(devices=[torch.cuda.current_device()]):
        torch.manual_seed(seed)
        with torch.device(DEVICE):
            model = network(case)
    model.train()
    # weights, preconditioned gradients and velocities: one buffer each
    params = list(model.parameters())
    flat, views = _flat_views([tuple(p.shape) for p in params])
    for p, v in zip(params, views):
        v.copy_(p.data)
        p.data = v
    opt = ck.KFAC(lr=LR, momentum=MOMENTUM, cov_ema_decay=case['decay'],
                  damping=case['damping'], acc_iters=case['acc'])
    opt.setup(model)
    kflat, kviews = _flat_views([p.shape for p in opt.target.params()])
    for p, v in zip(opt.target.params(), kviews):
        p.kfgrad = v
    batches = []
    for _ in range(case['acc']):
        shape = _input_shape(case, case['batch'])
        x = torch.rand(shape, device=DEVICE, generator=g) \
            if case['net'] == 'mlp' else \
            torch.randn(shape, device=DEVICE, generator=g)
        batches.append((_layout(x, case), torch.randint(
            0, case['classes'], (case['batch'],), device=DEVICE,
            generator=g)))

    def lossfun(x, t):
        return F.cross_entropy(model(x), t)
    state = dict(kind='step', opt=opt, lossfun=lossfun, batches=batches,
                 params=flat, kfgrad=kflat)
    _run_step(state)
    vflat, vviews = _flat_views([p.shape for p in opt.target.params()])
    for p, v in zip(opt.target.params(), vviews):
        p.update_rule.state['v'] = v.copy_(p.update_rule.state['v'])
    state['velocity'] = vflat
    for _ in range(2):      # running averages and plans of a running program
        _run_step(state)
    return state


def _prepare_block(case, seed):
    g = _gen(seed)
    n, layer = case['batch'], case['layer']
    if layer == 'linear':
        module = nn.Linear(case['cin'], case['cout'], bias=case['bias'])
        xs, gs = (n, case['cin']), (n, case['cout'])
        ctor = FB.FisherBlockLinear
    elif layer == 'conv':
        module = nn.Conv2d(case['cin'], case['cout'], case['k'],
                           case['stride'], case['pad'], bias=case['bias'])
        ho = (case['image'] + 2 * case['pad'] - case['k']) // \
            case['stride'] + 1
        xs = (n, case['cin'], case['image'], case['image'])
        gs = (n, case['cout'], ho, ho)
        ctor = FB.FisherBlockConvolution2D
    else:
        module = nn.BatchNorm2d(case['cout'])
        xs = gs = (n, case['cout'], case['image'], case['image'])
        ctor = FB.FisherBlockBatchNormalization
    link = links.wrap(module.to(DEVICE))
    fb = ctor('/layer', link, 0.95, case['damping'])
    x = torch.randn(xs, device=DEVICE, generator=g)
    if layer != 'bn':
        x = x.clamp_(min=0)
    # gradients of a mean loss (BatchNormalization sums them over positions)
    gy = torch.randn(gs, device=DEVICE, generator=g) / (
        n * case['image'] if layer == 'bn' else n)
    params = list(link.params())
    for p in params:
        p.grad = torch.randn(p.shape, device=DEVICE, generator=g) * 1e-2
    state = dict(kind='block', fb=fb, params=params,
                 in_data=(_layout(x, case),) + tuple(p.data for p in params),
                 gy=_layout(gy, case))
    for _ in range(2):
        _run_block(state)
    return state


def _prepare_factors(case, seed):
    g, table = _gen(seed), table_of(case)
    shapes, bn_shapes = [], []
    for l in table:
        if l['kind'] == 'bn':
            bn_shapes.append((l['rows'], 2 * l['c']))
        else:
            shapes += [(l['dA'], l['dA']), (l['dG'], l['dG'])]
    flat, outs = _flat_views(shapes)
    bflat, bouts = _flat_views(bn_shapes)
    layers, o, b = [], 0, 0
    for i, l in enumerate(table):
        n = l['x'][0]
        x = torch.randn(l['x'], device=DEVICE, generator=g)
        if i > 0 and l['kind'] != 'bn':
            x.clamp_(min=0)          # behind a ReLU
        gy = torch.randn(l['gy'], device=DEVICE, generator=g).div_(n)
        e = dict(l, x=_layout(x, case), gy=_layout(gy, case), n=n)
        if l['kind'] == 'bn':
            e['out'], b = bouts[b], b + 1
            e['stats'] = torch.empty(2 * l['c'] + 4 * n * l['c'],
                                     device=DEVICE)
        else:
            e['A'], e['G'], o = outs[o], outs[o + 1], o + 2
        layers.append(e)
    return dict(kind='factors', layers=layers, factors=flat, bn=bflat,
                decay=case['decay'])


def _prepare_pairs(case, seed):
    g, dims = _gen(seed), pair_dims(case)
    sides = [(d, d) for p in dims for d in p]
    _, factors = _flat_views(sides)
    inv_flat, inverses = _flat_views(sides)
    grads, velocity = [], []
    kf_flat, kf = _flat_views([(b, a) for a, b in dims])
    w_flat, weights = _flat_views([(b, a) for a, b in dims])
    for f in factors:
        d = f.shape[0]
        rows = max(2 * d, 256)
        x = torch.randn((rows, d), device=DEVICE, generator=g)
        torch.mm(x.t(), x, out=f)
        f.div_(rows).diagonal().add_(1e-3)
        f.copy_((f + f.t()) / 2)
    for a, b in dims:
        grads.append(torch.randn((b, a), device=DEVICE, generator=g) * 1e-2)
        velocity.append(torch.zeros((b, a), device=DEVICE))
    for w in weights:
        w.copy_(torch.randn(w.shape, device=DEVICE, generator=g))
    k = len(dims)
    plan = ops.InversePlanSet(
        factors, inverses, [i ^ 1 for i in range(2 * k)], [0, 1] * k)
    state = dict(kind='pairs', plan=plan, inverses=inverses, grads=grads,
                 kf=kf, weights=weights, velocity=velocity,
                 damping=case['damping'], out=(inv_flat, kf_flat, w_flat))
    for _ in range(2):
        _run_pairs(state)
    return state


def _prepare_wire(case, seed):
    g = _gen(seed)
    shapes, tri = [], []
    for l in table_of(case):
        if l['kind'] == 'bn':
            shapes += [(l['c'],), (l['c'],)]
            tri += [False, False]
        else:
            shapes += [(l['dG'], l['dA']), (l['dA'], l['dA']),
                       (l['dG'], l['dG'])]
            tri += [False, True, True]
    src_flat, src = _flat_views(shapes)
    dst_flat, dst = _flat_views(shapes)
    src_flat.normal_(generator=g)
    for t, is_tri in zip(src, tri):
        if is_tri:
            t.copy_((t + t.t()) / 2)
    dtype = getattr(torch, case['wire'])
    n = ops.wire_nelems(src, tri)
    wire = torch.zeros(n, dtype=dtype, device=DEVICE)
    # the buffers the other ranks have packed
    others = [torch.randn(n, device=DEVICE, generator=g).to(dtype)
              for _ in range(case['ranks'] - 1)]
    return dict(kind='wire', src=src, dst=dst, tri=tri, wire=wire,
                others=others, dst_flat=dst_flat)


# ----------------------------------------------------------------------- run

def run(state):
    return dict(step=_run_step, block=_run_block, factors=_run_factors,
                pairs=_run_pairs, wire=_run_wire)[state['kind']](state)


def _run_step(s):
    opt = s['opt']
    for x, t in s['batches']:
        opt.update(s['lossfun'], x, t)
    out = dict(loss=opt.loss, params=s['params'], kfgrad=s['kfgrad'],
               velocity=s.get('velocity'))
    conn = [fb for fb in opt.fblocks
            if isinstance(fb, FB.FisherBlockLinear) or
            isinstance(fb, FB.FisherBlockConvolution2D)]
    if len(conn) <= 25:
        out['factors'] = [fb.cov_emas for fb in conn]
    return out


def _run_block(s):
    fb, in_data = s['fb'], s['in_data']
    func = fb.funcclass()
    fb.forward_postprocess(func, in_data)
    fb.backward_preprocess(func, in_data, (s['gy'],))
    fb.update_cov_emas()
    fb.update_invs()
    fb.update_kfgrads()
    return dict(factors=fb.cov_emas, inverses=fb.invs,
                kfgrad=[p.kfgrad for p in s['params']])


def _run_factors(s):
    r = s['decay']
    items, bn = [], []
    for l in s['layers']:
        n = l['n']
        if l['kind'] == 'bn':
            bn.append(ops.bn_item(l['x'], l['gy'], 1e-5, float(n), l['out'],
                                  l['stats']))
        elif l['kind'] == 'conv':
            ho, wo = l['gy'].shape[2:]
            items.append(ops.conv_input_item(
                l['x'], l['k'], l['stride'], l['pad'], l['bias'], r / n,
                1.0 - r, l['A']))
            items.append(ops.conv_grad_item(
                l['gy'], r * n / float(ho * wo), 1.0 - r, l['G']))
        else:
            items.append(ops.dense_item(l['x'], l['bias'], r / n, 1.0 - r,
                                        l['A']))
            items.append(ops.dense_item(l['gy'], False, r * n, 1.0 - r,
                                        l['G']))
    ops.bn_sample_grads_group(bn)
    ops.factor_group(items, s['factors'].device)
    return dict(factors=s['factors'], bn=s['bn'])


def _run_pairs(s):
    plan, inv = s['plan'], s['inverses']
    classes = plan.classes()

    def after(c):
        own = sorted({i // 2 for i in classes[c]})
        none = [None] * len(own)
        w = [s['weights'][i] for i in own]
        v = [s['velocity'][i] for i in own]
        ops.precondition(
            [inv[2 * i + 1] for i in own], [inv[2 * i] for i in own],
            [s['grads'][i] for i in own], none, [s['kf'][i] for i in own],
            none, w, none, v, none, lr=LR, momentum=MOMENTUM, ws_key=c)
    plan.run(s['damping'], True, after_class=after)
    return s['out']


def _run_wire(s):
    ops.wire_pack(s['src'], s['tri'], s['wire'])
    wires = [s['wire']] + s['others']
    ops.wire_unpack_sum(s['dst'], s['tri'], [w.data_ptr() for w in wires],
                        scale=1.0 / len(wires), wire_dtype=s['wire'].dtype)
    return s['wire'], s['dst_flat']


# ------------------------------------------------------ work and tolerance

def work(case):
    """Bytes and operations of one pass: every input read once, every result
    written once; one triangle of a symmetric product; d^3 per inverse."""
    kind, nbytes, flops = case['kind'], 0.0, 0.0
    if kind == 'pairs':
        for a, b in pair_dims(case):
            flops += a ** 3 + b ** 3 + 2.0 * a * b * (a + b)
            # factor triangles, inverses, gradient, kf, weight and velocity
            nbytes += 4.0 * (1.5 * (a * a + b * b) + 6 * a * b)
        return dict(bytes=nbytes, flops=flops)
    if kind == 'wire':
        size = 4 if case['wire'] == 'float32' else 2
        for l in table_of(case):
            if l['kind'] == 'bn':
                full = tri = 2 * l['c']
            else:
                a, b = l['dA'], l['dG']
                full = a * b + a * a + b * b
                tri = a * b + (a * (a + 1) + b * (b + 1)) // 2
            nbytes += 4.0 * (tri + full) + size * tri * (1 + case['ranks'])
        return dict(bytes=nbytes, flops=0.0)
    if kind == 'block':
        table = [_block_layer(case)]
    else:
        table = table_of(case)
    acc = case.get('acc', 1)
    for l in table:
        act = 4.0 * (math.prod(l['x']) + math.prod(l['gy']))
        if l['kind'] == 'bn':
            d, rows = 2 * l['c'], l['rows']
            nbytes += acc * (act + 4.0 * rows * d)
            flops += acc * 6.0 * math.prod(l['x'])
            if kind != 'factors':
                # the block's damped solve in its cheaper form
                m = min(d, 8 * rows) if case.get('acc', 1) == 1 else d
                flops += 2.0 * m * m * d + m ** 3 + 2.0 * m * d
                nbytes += 4.0 * (m * d + 6 * d)
            continue
        a, b, rows = l['dA'], l['dG'], l['rows']
        flops += acc * float(rows) * (a * (a + 1) + b * (b + 1))
        nbytes += acc * act + 8.0 * (a * a + b * b)
        if kind != 'factors':
            flops += a ** 3 + b ** 3 + 2.0 * a * b * (a + b)
            nbytes += 4.0 * (a * a + b * b + 6 * a * b)
        if kind == 'step':      # forward and backward of the layer itself
            flops += acc * 6.0 * rows * a * b
            nbytes += acc * 3.0 * act
    return dict(bytes=nbytes, flops=flops)


def _block_layer(case):
    n = case['batch']
    if case['layer'] == 'linear':
        a, b = case['cin'] + int(case['bias']), case['cout']
        return dict(kind='linear', x=(n, case['cin']), gy=(n, b), dA=a, dG=b,
                    rows=n)
    if case['layer'] == 'bn':
        s = (n, case['cout'], case['image'], case['image'])
        return dict(kind='bn', x=s, gy=s, c=case['cout'], rows=n)
    ho = (case['image'] + 2 * case['pad'] - case['k']) // case['stride'] + 1
    return dict(kind='conv',
                x=(n, case['cin'], case['image'], case['image']),
                gy=(n, case['cout'], ho, ho),
                dA=case['cin'] * case['k'] ** 2 + int(case['bias']),
                dG=case['cout'], rows=n * ho * ho)


def tolerance(case):
    """Factors are products of fp32 values held as two 16-bit terms (5e-6; up
    to 5e-5 for the longest sums), inverses and preconditioned gradients
    amplify that by the conditioning the damping leaves: up to about 1e-4 in
    a network's step and on prebuilt factors, 1e-3 for a single layer with
    fewer rows than columns."""
    kind = case['kind']
    if kind == 'wire':
        return dict(rel=1e-6, max=1e-5)
    if kind == 'factors':
        return dict(rel=1e-4, max=5e-3)
    if kind == 'pairs':
        return dict(rel=2e-4, max=1e-2)
    if kind == 'block':
        return dict(rel=2e-3, max=5e-2)
    return dict(rel=1e-3, max=2e-2)
