// adjoint_api.cu -- C ABI of the variational equations and the adjoint (FP64): state transition
// matrices, vector-Jacobian products of the propagation, and the gradient of the closest-approach
// miss distance of listed pairs with respect to both objects' initial states.
#include "common.cuh"
#include "context.h"
#include "variational.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

using namespace gpop;

namespace {

struct ScopedBufs {
    DevBuf b[12];
    explicit ScopedBufs(const gpop_ctx* ctx)
    {
        for (DevBuf& x : b)
            x.use(ctx->pool, true);
    }
    ~ScopedBufs()
    {
        for (DevBuf& x : b)
            x.release();
    }
};

bool valid_start(const gpop_time* t)
{
    return t && t->month >= 1 && t->month <= 12 && t->day >= 1 && t->day <= 31 && std::isfinite(t->sec);
}

gpop_status check_common(gpop_ctx* ctx, const gpop_time* start, double h, int32_t steps, int64_t n,
    const void* r_in, const void* v_in)
{
    if (!valid_start(start) || !(h > 0.0) || !std::isfinite(h) || steps < 0 || n <= 0 || !r_in || !v_in)
        return fail(ctx, GPOP_ERR_INVALID_ARG, "invalid propagation arguments");
    if (n > (int64_t)1 << 24)
        return fail(ctx, GPOP_ERR_INVALID_ARG, "too many objects");
    const int64_t bad = first_bad_state(static_cast<const double*>(r_in), static_cast<const double*>(v_in), n, true);
    if (bad >= 0)
        return bad_state(ctx, bad, "object");
    if (ctx->cfg.n_corrections < 1)
        return fail(ctx, GPOP_ERR_UNSUPPORTED, "the adjoint needs at least one corrector pass");
    cudaError_t e = cudaSetDevice(ctx->cfg.device);
    if (e != cudaSuccess)
        return cuda_fail(ctx, e, "cudaSetDevice");
    return GPOP_OK;
}

gpop_status upload(gpop_ctx* ctx, DevBuf& d, const double* host, size_t count, cudaStream_t s)
{
    cudaError_t e = d.ensure(count * sizeof(double));
    if (e != cudaSuccess)
        return fail(ctx, GPOP_ERR_NOMEM, std::string("device buffer: ") + cudaGetErrorString(e));
    if ((e = cudaMemcpyAsync(d.p, host, count * sizeof(double), cudaMemcpyHostToDevice, s)) != cudaSuccess)
        return cuda_fail(ctx, e, "upload");
    return GPOP_OK;
}

constexpr int64_t kVarObjects = 65536; // objects whose startup tangents are held at once
constexpr size_t kWindowBytes = (size_t)512 << 20; // Jacobians held at once

gpop_status nomem(gpop_ctx* ctx, const char* what, cudaError_t e)
{
    return fail(ctx, GPOP_ERR_NOMEM, std::string(what) + ": " + cudaGetErrorString(e));
}

// A fresh FP64 propagation of n objects (device AoS r, v in place).
gpop_status begin(gpop_ctx* ctx, gpop_propagator& p, const gpop_time* start, double h, int32_t steps, int64_t n,
    double* r, double* v, cudaStream_t s)
{
    p.ctx = ctx;
    p.kind = GPOP_FORCE_GRAVITY;
    p.start = *start;
    p.h = h;
    p.ncorr = ctx->cfg.n_corrections;
    p.max_steps = steps;
    p.n = n;
    p.r = r;
    p.v = v;
    p.mixed = false;
    for (DevBuf* b : { &p.own_state, &p.own_gen, &p.own_prop })
        b->use(ctx->pool, true);
    return propagator_init(&p, s);
}

constexpr size_t kPassBytes = (size_t)64 << 20; // Jacobians of plain startup passes held at once

// Positions of the startup's stages and columns, their Jacobians and the startup tangents.
struct StartupTangents {
    DevBuf stage_pos, col_pos, pass_pos, stage_jac, col_jac, pass_jac, out;
    int window = 1; // plain passes whose Jacobians are held at once
    explicit StartupTangents(const gpop_ctx* ctx)
    {
        for (DevBuf* b : { &stage_pos, &col_pos, &pass_pos, &stage_jac, &col_jac, &pass_jac, &out })
            b->use(ctx->pool, true);
    }
    ~StartupTangents()
    {
        for (DevBuf* b : { &stage_pos, &col_pos, &pass_pos, &stage_jac, &col_jac, &pass_jac, &out })
            b->release();
    }
    gpop_status reserve(gpop_ctx* ctx, gpop_propagator& p)
    {
        const size_t n = (size_t)p.n;
        window = (int)std::min<size_t>(p.ncorr, std::max<size_t>(1, kPassBytes / (81 * n * 8)));
        cudaError_t e;
        if ((e = stage_pos.ensure(240 * n * 8)) != cudaSuccess || (e = col_pos.ensure(27 * n * 8)) != cudaSuccess
            || (e = pass_pos.ensure((size_t)p.ncorr * 27 * n * 8)) != cudaSuccess
            || (e = pass_jac.ensure((size_t)window * 81 * n * 8)) != cudaSuccess
            || (e = stage_jac.ensure(720 * n * 8)) != cudaSuccess || (e = col_jac.ensure(81 * n * 8)) != cudaSuccess
            || (e = out.ensure((size_t)kStartupTangents * 6 * n * 8)) != cudaSuccess)
            return nomem(ctx, "startup tangents", e);
        p.stage_pos = stage_pos.as<double>();
        p.col_pos = col_pos.as<double>();
        p.pass_pos = pass_pos.as<double>();
        return GPOP_OK;
    }
    // after the startup of p has run
    gpop_status make(gpop_ctx* ctx, const gpop_propagator& p, cudaStream_t s)
    {
        JacPoints j;
        j.n = j.width = p.n;
        j.err = ctx->err_word.as<unsigned>();
        j.pos = stage_pos.as<double>();
        j.M = p.gen_m->as<double>();
        j.items = 80;
        j.total = 80 * p.n;
        j.jac = stage_jac.as<double>();
        cudaError_t e = launch_jac_points(ctx->table(false), j, ctx->num_sms, s);
        j.pos = col_pos.as<double>();
        j.M = p.prop_m->as<double>();
        j.items = 9;
        j.total = 9 * p.n;
        j.jac = col_jac.as<double>();
        if (e == cudaSuccess)
            e = launch_jac_points(ctx->table(false), j, ctx->num_sms, s);
        StartupTangentArgs t;
        t.n = p.n;
        t.h = p.h;
        t.ncorr = p.ncorr;
        t.stage_jac = stage_jac.as<double>();
        t.col_jac = col_jac.as<double>();
        t.out = out.as<double>();
        if (e == cudaSuccess)
            e = launch_rk8_tangents(t, s);
        ctx->launches += 3;
        t.mark = pass_pos.as<double>();
        t.pass_jac = pass_jac.as<double>();
        j.frames = 9;
        j.mark = t.mark;
        j.jac = pass_jac.as<double>();
        for (; t.pass_lo < p.ncorr && e == cudaSuccess; t.pass_lo = t.pass_hi) {
            t.pass_hi = std::min(p.ncorr, t.pass_lo + window);
            j.pos = pass_pos.as<double>() + (size_t)t.pass_lo * 27 * p.n;
            j.items = 9 * (t.pass_hi - t.pass_lo);
            j.total = j.items * p.n;
            if ((e = launch_jac_points(ctx->table(false), j, ctx->num_sms, s)) == cudaSuccess)
                e = launch_pass_tangents(t, s);
            ctx->launches += 2;
        }
        if (e == cudaSuccess)
            e = launch_corrector_tangents(t, s);
        ctx->launches++;
        if (e != cudaSuccess)
            return cuda_fail(ctx, e, "startup tangents");
        return GPOP_OK;
    }
};

// Forward run of the adjoint: the whole trajectory's positions and accelerations in traj_r and traj_a (and v when
// asked for), or, with traj_r NULL, the GJ8 state after the startup and after every 64th step in ckpt.
gpop_status forward_run(gpop_ctx* ctx, gpop_propagator& p, int32_t steps, double* traj_r, double* traj_v,
    double* traj_a, DevBuf& ckpt, cudaStream_t s)
{
    if (traj_r)
        return propagator_step(&p, steps, traj_r, traj_v, traj_a, s);
    const int64_t n = p.n;
    const int nseg = (steps - 1) / kCheckpointSteps + 1;
    const size_t ck_elems = (size_t)kCheckpointArrays * n;
    cudaError_t e = ckpt.ensure(std::max(1, nseg) * ck_elems * sizeof(double));
    if (e != cudaSuccess)
        return nomem(ctx, "checkpoints", e);
    const double* state_ck = p.state->as<double>() + (size_t)kSs * n;
    gpop_status st;
    int done = std::min(steps, 4); // startup + the replayed steps: the GJ8 state is final here
    if ((st = propagator_step(&p, done, nullptr, nullptr, nullptr, s)) != GPOP_OK)
        return st;
    for (int seg = 0;; ++seg) {
        if ((e = cudaMemcpyAsync(ckpt.as<double>() + (size_t)seg * ck_elems, state_ck, ck_elems * sizeof(double),
                 cudaMemcpyDeviceToDevice, s))
            != cudaSuccess)
            return cuda_fail(ctx, e, "checkpoint copy");
        if (seg + 1 >= nseg)
            return GPOP_OK; // the last segment is run by the reverse sweep alone
        const int target = (seg + 1) * kCheckpointSteps;
        if ((st = propagator_step(&p, target - done, nullptr, nullptr, nullptr, s)) != GPOP_OK)
            return st;
        done = target;
    }
}

// Reverse sweep over a forward run. step0: host copy of the units' first seeded step, obj_host of their
// objects. Device: unit_obj, seed_step0, seeds, grad.
gpop_status run_adjoint(gpop_ctx* ctx, gpop_propagator& p, int32_t steps, const double* r0, const double* v0,
    const double* traj_r, const double* traj_a, const DevBuf& ckpt, StartupTangents& tan, const std::vector<int>& step0,
    const std::vector<int>& obj_host, const int* unit_obj, const int* seed_step0, const double* seeds, double* grad,
    cudaStream_t s)
{
    const int64_t U = (int64_t)step0.size(), n = p.n;
    struct Bufs {
        DevBuf rank, sweep, jac, offset, pos;
        explicit Bufs(const gpop_ctx* ctx)
        {
            for (DevBuf* b : { &rank, &sweep, &jac, &offset, &pos })
                b->use(ctx->pool, true);
        }
        ~Bufs()
        {
            for (DevBuf* b : { &rank, &sweep, &jac, &offset, &pos })
                b->release();
        }
    } B(ctx);
    // ranks: units by their last seeded step, latest first
    std::vector<int> rank(2 * U); // unit, then object of each rank
    for (int64_t u = 0; u < U; ++u)
        rank[u] = (int)u;
    auto last = [&](int u) { return std::min(step0[u] + 2, steps); };
    std::stable_sort(rank.begin(), rank.begin() + U, [&](int a, int b) { return last(a) > last(b); });
    for (int64_t u = 0; u < U; ++u)
        rank[U + u] = obj_host[rank[u]];
    cudaError_t e;
    if ((e = B.rank.ensure(2 * U * sizeof(int))) != cudaSuccess
        || (e = B.sweep.ensure((size_t)kAdjSweep * U * sizeof(double))) != cudaSuccess)
        return nomem(ctx, "adjoint buffers", e);
    if ((e = cudaMemcpyAsync(B.rank.p, rank.data(), 2 * U * sizeof(int), cudaMemcpyHostToDevice, s)) != cudaSuccess)
        return cuda_fail(ctx, e, "unit ranks");
    AdjSweepArgs a;
    a.n_units = U;
    a.unit = B.rank.as<int>();
    a.seed_step0 = seed_step0;
    a.seeds = seeds;
    a.steps = steps;
    a.h = p.h;
    a.ncorr = ctx->cfg.n_corrections;
    a.sweep = B.sweep.as<double>();
    a.first = true;
    int hi = U > 0 ? last(rank[0]) : 0;
    int64_t cnt = 0; // ranks that take part at the present step
    if (hi < 5) { // nothing to sweep: zero adjoints
        if ((e = launch_adjoint_sweep(a, s)) != cudaSuccess)
            return cuda_fail(ctx, e, "adjoint kernel");
        ctx->launches++;
    }
    size_t limit = std::max<size_t>(kWindowBytes / 72, (size_t)U);
    int held = -1; // segment whose positions and accelerations, `rows` doubles each, are in B.pos
    size_t rows = 0;
    while (hi >= 5) {
        const int floor_step = traj_r ? 5 : std::max(5, (hi - 1) / kCheckpointSteps * kCheckpointSteps + 1);
        // ranks per step from hi down, as many steps as the Jacobians' budget takes
        std::vector<int64_t> width;
        size_t total = 0;
        int lo = hi + 1;
        int64_t c = cnt;
        while (lo > floor_step) {
            while (c < U && last(rank[c]) >= lo - 1)
                ++c;
            if (total > 0 && total + (size_t)c > limit)
                break;
            total += (size_t)c;
            width.push_back(c);
            --lo;
        }
        std::vector<int64_t> offset(width.size()); // ascending steps
        int64_t at = 0;
        for (size_t i = 0; i < width.size(); ++i) {
            offset[i] = at;
            at += width[width.size() - 1 - i];
        }
        e = B.jac.ensure(9 * total * sizeof(double));
        if (e == cudaErrorMemoryAllocation && width.size() > 1) { // fewer steps at once
            cudaGetLastError();
            limit = total / 2;
            continue;
        }
        cnt = width.back();
        if (e != cudaSuccess || (e = B.offset.ensure(offset.size() * sizeof(int64_t))) != cudaSuccess)
            return nomem(ctx, "adjoint Jacobians", e);
        if ((e = cudaMemcpyAsync(B.offset.p, offset.data(), offset.size() * sizeof(int64_t), cudaMemcpyHostToDevice, s))
            != cudaSuccess)
            return cuda_fail(ctx, e, "adjoint window");
        const double* pos = traj_r ? traj_r + (size_t)(lo - 1) * 3 * n : nullptr;
        const double* acc = traj_r ? traj_a + (size_t)(lo - 1) * 3 * n : nullptr;
        if (!traj_r) {
            const int seg = (lo - 1) / kCheckpointSteps, from = std::max(5, seg * kCheckpointSteps + 1);
            if (seg != held) { // its first window, which ends where the segment does: run it from its checkpoint
                rows = (size_t)(hi - from + 1) * 3 * n;
                if ((e = B.pos.ensure(2 * rows * sizeof(double))) != cudaSuccess)
                    return nomem(ctx, "adjoint segment", e);
                const size_t ck = (size_t)kCheckpointArrays * n;
                if ((e = cudaMemcpyAsync(p.state->as<double>() + (size_t)kSs * n,
                         ckpt.as<double>() + (size_t)seg * ck, ck * sizeof(double), cudaMemcpyDeviceToDevice, s))
                    != cudaSuccess)
                    return cuda_fail(ctx, e, "checkpoint restore");
                p.done = from - 1;
                const gpop_status st
                    = propagator_step(&p, hi - from + 1, B.pos.as<double>(), nullptr, B.pos.as<double>() + rows, s);
                if (st != GPOP_OK)
                    return st;
                held = seg;
            }
            pos = B.pos.as<double>() + (size_t)(lo - from) * 3 * n;
            acc = pos + rows;
        }
        JacPoints j;
        j.n = n;
        j.pos = pos;
        j.acc = acc;
        j.M = p.prop_m->as<double>() + (size_t)(lo + 4) * 9;
        j.items = (int)offset.size();
        j.offset = B.offset.as<int64_t>();
        j.obj = B.rank.as<int>() + U;
        j.total = (int64_t)total;
        j.jac = B.jac.as<double>();
        j.err = ctx->err_word.as<unsigned>();
        a.step_lo = lo;
        a.step_hi = hi;
        a.jac = j.jac;
        a.offset = j.offset;
        a.total = j.total;
        if ((e = launch_jac_points(ctx->table(false), j, ctx->num_sms, s)) != cudaSuccess
            || (e = launch_adjoint_sweep(a, s)) != cudaSuccess)
            return cuda_fail(ctx, e, "adjoint kernel");
        ctx->launches += 2;
        a.first = false;
        hi = lo - 1;
    }
    // the startup's part, for the objects whose tangents are at hand, or piece by piece
    AdjFinishArgs f;
    f.n_units = U;
    f.unit = a.unit;
    f.unit_obj = unit_obj;
    f.seed_step0 = seed_step0;
    f.seeds = seeds;
    f.steps = steps;
    f.flags = ctx->cfg.flags;
    f.sweep = a.sweep;
    f.grad = grad;
    for (int64_t lo = 0; lo < n; lo += kVarObjects) {
        f.obj_lo = lo;
        f.n = std::min(kVarObjects, n - lo);
        gpop_status st;
        if (n <= kVarObjects) {
            if ((st = tan.make(ctx, p, s)) != GPOP_OK)
                return st;
        } else {
            gpop_propagator q;
            DevBuf rv;
            struct Free {
                DevBuf& b;
                ~Free() { b.release(); }
            } free_rv { rv };
            const size_t bytes = (size_t)f.n * 3 * sizeof(double);
            rv.use(ctx->pool, true);
            q.own_state.use(ctx->pool, true);
            if ((e = rv.ensure(2 * bytes)) != cudaSuccess || (e = q.own_state.ensure(state_bytes(f.n))) != cudaSuccess)
                return nomem(ctx, "startup tangents", e);
            q.ctx = ctx;
            q.start = p.start;
            q.h = p.h;
            q.ncorr = p.ncorr;
            q.max_steps = 1;
            q.n = f.n;
            q.r = rv.as<double>();
            q.v = q.r + 3 * f.n;
            q.gen_m = p.gen_m;
            q.prop_m = p.prop_m;
            if ((e = cudaMemcpyAsync(q.r, r0 + 3 * lo, bytes, cudaMemcpyDeviceToDevice, s)) != cudaSuccess
                || (e = cudaMemcpyAsync(q.v, v0 + 3 * lo, bytes, cudaMemcpyDeviceToDevice, s)) != cudaSuccess)
                return cuda_fail(ctx, e, "startup tangents");
            if ((st = tan.reserve(ctx, q)) != GPOP_OK || (st = propagator_step(&q, 1, nullptr, nullptr, nullptr, s)) != GPOP_OK
                || (st = tan.make(ctx, q, s)) != GPOP_OK)
                return st;
        }
        f.startup = tan.out.as<double>();
        if ((e = launch_adjoint_finish(f, s)) != cudaSuccess)
            return cuda_fail(ctx, e, "adjoint kernel");
        ctx->launches++;
        if (n > kVarObjects && (e = cudaStreamSynchronize(s)) != cudaSuccess) // the piece's buffers are used again
            return cuda_fail(ctx, e, "adjoint kernel");
    }
    return check_device_errors(ctx, s);
}

// The vector-Jacobian product of checked arguments, from the stored trajectory or from checkpoints.
gpop_status run_vjp(gpop_ctx* ctx, const gpop_time* start, double h, int32_t steps, int64_t n, const double* r_in,
    const double* v_in, const double* r_bar, const double* v_bar, bool store, double* grad_r0, double* grad_v0)
{
    cudaStream_t s = nullptr;
    gpop_status st;
    cudaError_t e;
    ScopedBufs B(ctx);
    DevBuf &dr = B.b[0], &dv = B.b[1], &dr0 = B.b[2], &dv0 = B.b[3], &ck = B.b[4], &traj = B.b[5],
           &dobj = B.b[6], &dstep = B.b[7], &dseed = B.b[8], &dgrad = B.b[9];
    StartupTangents tan(ctx);
    if ((st = upload(ctx, dr, r_in, 3 * n, s)) != GPOP_OK || (st = upload(ctx, dv, v_in, 3 * n, s)) != GPOP_OK
        || (st = upload(ctx, dr0, r_in, 3 * n, s)) != GPOP_OK || (st = upload(ctx, dv0, v_in, 3 * n, s)) != GPOP_OK)
        return st;
    const size_t rows = (size_t)steps * 3 * n;
    if (store && (e = traj.ensure(2 * rows * sizeof(double))) != cudaSuccess)
        return nomem(ctx, "trajectory", e);
    gpop_propagator p;
    if ((st = begin(ctx, p, start, h, steps, n, dr.as<double>(), dv.as<double>(), s)) != GPOP_OK
        || (n <= kVarObjects && (st = tan.reserve(ctx, p)) != GPOP_OK)
        || (st = forward_run(ctx, p, steps, store ? traj.as<double>() : nullptr, nullptr,
                store ? traj.as<double>() + rows : nullptr, ck, s))
            != GPOP_OK)
        return st;
    // seeds on the final state: node 0 at the last step
    std::vector<int> obj(n), step0(n, steps);
    std::vector<double> seeds((size_t)n * 27, 0.0);
    for (int64_t o = 0; o < n; ++o) {
        obj[o] = (int)o;
        for (int j = 0; j < 3; ++j) {
            seeds[o * 27 + j] = r_bar ? r_bar[o * 3 + j] : 0.0;
            seeds[o * 27 + 3 + j] = v_bar ? v_bar[o * 3 + j] : 0.0;
        }
    }
    if ((e = dobj.ensure(n * sizeof(int))) != cudaSuccess || (e = dstep.ensure(n * sizeof(int))) != cudaSuccess
        || (e = dgrad.ensure(6 * n * sizeof(double))) != cudaSuccess)
        return fail(ctx, GPOP_ERR_NOMEM, std::string("adjoint buffers: ") + cudaGetErrorString(e));
    if ((st = upload(ctx, dseed, seeds.data(), seeds.size(), s)) != GPOP_OK)
        return st;
    if ((e = cudaMemcpyAsync(dobj.p, obj.data(), n * sizeof(int), cudaMemcpyHostToDevice, s)) != cudaSuccess
        || (e = cudaMemcpyAsync(dstep.p, step0.data(), n * sizeof(int), cudaMemcpyHostToDevice, s)) != cudaSuccess)
        return cuda_fail(ctx, e, "seed upload");
    if ((st = run_adjoint(ctx, p, steps, dr0.as<double>(), dv0.as<double>(), store ? traj.as<double>() : nullptr,
             store ? traj.as<double>() + rows : nullptr, ck, tan, step0, obj, dobj.as<int>(),
             dstep.as<int>(), dseed.as<double>(), dgrad.as<double>(), s))
        != GPOP_OK)
        return st;
    std::vector<double> g(6 * n);
    if ((e = cudaMemcpy(g.data(), dgrad.p, 6 * n * sizeof(double), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cuda_fail(ctx, e, "gradient download");
    for (int64_t o = 0; o < n; ++o)
        for (int j = 0; j < 3; ++j) {
            grad_r0[o * 3 + j] = g[o * 6 + j];
            grad_v0[o * 3 + j] = g[o * 6 + 3 + j];
        }
    return GPOP_OK;
}

} // namespace

extern "C" {

gpop_status gpop_gravity_jacobian(gpop_ctx* ctx, int64_t n, const double* r_dev, const double* frame9_dev,
    double* a_dev, double* jac_dev, void* stream)
{
    if (!ctx)
        return GPOP_ERR_INVALID_ARG;
    if (n < 0 || (n > 0 && (!r_dev || !jac_dev)))
        return fail(ctx, GPOP_ERR_INVALID_ARG, "invalid Jacobian arguments");
    cudaError_t e = cudaSetDevice(ctx->cfg.device);
    if (e != cudaSuccess)
        return cuda_fail(ctx, e, "cudaSetDevice");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if ((e = launch_jacobian(ctx->table(false), ctx->lane_table(false), n, r_dev, frame9_dev, a_dev, jac_dev,
             ctx->err_word.as<unsigned>(), ctx->num_sms, s))
        != cudaSuccess)
        return cuda_fail(ctx, e, "Jacobian kernel");
    ctx->launches++;
    return check_device_errors(ctx, s);
}

gpop_status gpop_stm(gpop_ctx* ctx, const gpop_time* start, double h, int32_t steps, int64_t n,
    const double* r_in, const double* v_in, double* r_out, double* v_out, double* stm_out)
{
    if (!ctx)
        return GPOP_ERR_INVALID_ARG;
    gpop_status st = check_common(ctx, start, h, steps, n, r_in, v_in);
    if (st != GPOP_OK)
        return st;
    if (!stm_out)
        return fail(ctx, GPOP_ERR_INVALID_ARG, "missing STM output");
    if (steps == 0) {
        for (int64_t o = 0; o < n; ++o)
            for (int i = 0; i < 6; ++i)
                for (int j = 0; j < 6; ++j)
                    stm_out[(o * 6 + i) * 6 + j] = i == j ? 1.0 : 0.0;
        if (r_out)
            std::copy(r_in, r_in + 3 * n, r_out);
        if (v_out)
            std::copy(v_in, v_in + 3 * n, v_out);
        return GPOP_OK;
    }
    cudaStream_t s = nullptr;
    for (int64_t lo = 0; lo < n; lo += kVarObjects) {
        const int64_t m = std::min(kVarObjects, n - lo);
        ScopedBufs B(ctx);
        DevBuf &dr = B.b[0], &dv = B.b[1], &dphi = B.b[2], &pos = B.b[3], &jac = B.b[4], &sweep = B.b[5];
        StartupTangents tan(ctx);
        gpop_propagator p;
        if ((st = upload(ctx, dr, r_in + 3 * lo, 3 * m, s)) != GPOP_OK || (st = upload(ctx, dv, v_in + 3 * lo, 3 * m, s)) != GPOP_OK
            || (st = begin(ctx, p, start, h, steps, m, dr.as<double>(), dv.as<double>(), s)) != GPOP_OK
            || (st = tan.reserve(ctx, p)) != GPOP_OK)
            return st;
        int window = (int)std::min<int64_t>(steps, std::max<int64_t>(1, (int64_t)(kWindowBytes / 120) / m));
        cudaError_t e;
        if ((e = dphi.ensure(36 * m * sizeof(double))) != cudaSuccess
            || (e = sweep.ensure((size_t)kStmSweep * 6 * m * sizeof(double))) != cudaSuccess)
            return nomem(ctx, "STM buffers", e);
        while ((e = pos.ensure((size_t)window * 6 * m * sizeof(double))) != cudaSuccess
            || (e = jac.ensure((size_t)window * 9 * m * sizeof(double))) != cudaSuccess) {
            if (e != cudaErrorMemoryAllocation || window == 1)
                return nomem(ctx, "STM buffers", e);
            cudaGetLastError(); // fewer steps at once
            window /= 2;
        }
        int done = std::min(steps, 4);
        if ((st = propagator_step(&p, done, nullptr, nullptr, nullptr, s)) != GPOP_OK || (st = tan.make(ctx, p, s)) != GPOP_OK)
            return st;
        StmArgs a;
        a.n = m;
        a.steps = steps;
        a.h = h;
        a.ncorr = ctx->cfg.n_corrections;
        a.first = true;
        a.startup = tan.out.as<double>();
        a.sweep = sweep.as<double>();
        a.phi = dphi.as<double>();
        do {
            const int w = std::min(window, steps - done);
            a.step_lo = done + 1;
            a.step_hi = done + w;
            a.last = a.step_hi >= steps;
            if (w > 0) {
                double* acc = pos.as<double>() + (size_t)window * 3 * m;
                if ((st = propagator_step(&p, w, pos.as<double>(), nullptr, acc, s)) != GPOP_OK)
                    return st;
                JacPoints j;
                j.n = j.width = m;
                j.pos = pos.as<double>();
                j.acc = acc;
                j.M = p.prop_m->as<double>() + (size_t)(a.step_lo + 4) * 9;
                j.items = w;
                j.total = (int64_t)w * m;
                j.jac = jac.as<double>();
                j.err = ctx->err_word.as<unsigned>();
                if ((e = launch_jac_points(ctx->table(false), j, ctx->num_sms, s)) != cudaSuccess)
                    return cuda_fail(ctx, e, "STM Jacobians");
                a.jac = j.jac;
                ctx->launches++;
            }
            if ((e = launch_stm_sweep(a, s)) != cudaSuccess)
                return cuda_fail(ctx, e, "STM kernel");
            ctx->launches++;
            a.first = false;
            done += w;
        } while (done < steps);
        if ((e = cudaMemcpyAsync(stm_out + 36 * lo, dphi.p, 36 * m * sizeof(double), cudaMemcpyDeviceToHost, s)) != cudaSuccess
            || (r_out && (e = cudaMemcpyAsync(r_out + 3 * lo, dr.p, 3 * m * sizeof(double), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
            || (v_out && (e = cudaMemcpyAsync(v_out + 3 * lo, dv.p, 3 * m * sizeof(double), cudaMemcpyDeviceToHost, s)) != cudaSuccess))
            return cuda_fail(ctx, e, "STM download");
        if ((st = check_device_errors(ctx, s)) != GPOP_OK)
            return st;
    }
    return GPOP_OK;
}

gpop_status gpop_propagate_vjp(gpop_ctx* ctx, const gpop_time* start, double h, int32_t steps, int64_t n,
    const double* r_in, const double* v_in, const double* r_bar, const double* v_bar, double* grad_r0,
    double* grad_v0)
{
    if (!ctx)
        return GPOP_ERR_INVALID_ARG;
    gpop_status st = check_common(ctx, start, h, steps, n, r_in, v_in);
    if (st != GPOP_OK)
        return st;
    if (!grad_r0 || !grad_v0)
        return fail(ctx, GPOP_ERR_INVALID_ARG, "missing gradient outputs");
    if (steps == 0) {
        for (int64_t i = 0; i < 3 * n; ++i) {
            grad_r0[i] = r_bar ? r_bar[i] : 0.0;
            grad_v0[i] = v_bar ? v_bar[i] : 0.0;
        }
        return GPOP_OK;
    }
    // the positions and accelerations of every step when they fit, else checkpoints: also where memory runs out
    // behind them
    const size_t traj_bytes = (size_t)6 * steps * n * sizeof(double);
    st = GPOP_ERR_NOMEM;
    if (traj_bytes <= ctx->adjoint_store)
        st = run_vjp(ctx, start, h, steps, n, r_in, v_in, r_bar, v_bar, true, grad_r0, grad_v0);
    if (st == GPOP_ERR_NOMEM) {
        cudaGetLastError();
        st = run_vjp(ctx, start, h, steps, n, r_in, v_in, r_bar, v_bar, false, grad_r0, grad_v0);
    }
    return st;
}

gpop_status gpop_miss_gradient(gpop_ctx* ctx, const gpop_time* start, double h, int32_t steps, int64_t n,
    const double* r_in, const double* v_in, int64_t n_pairs, const int32_t* pairs, double* tca,
    double* miss, double* grad)
{
    if (!ctx)
        return GPOP_ERR_INVALID_ARG;
    gpop_status st = check_common(ctx, start, h, steps, n, r_in, v_in);
    if (st != GPOP_OK)
        return st;
    if (steps < 1 || n_pairs <= 0 || !pairs || !tca || !miss || !grad)
        return fail(ctx, GPOP_ERR_INVALID_ARG, "invalid pair arguments");
    if (n_pairs > (int64_t)1 << 24)
        return fail(ctx, GPOP_ERR_INVALID_ARG, "too many pairs");
    for (int64_t i = 0; i < n_pairs; ++i) {
        const int32_t a = pairs[2 * i], b = pairs[2 * i + 1];
        if (a < 0 || b < 0 || a >= n || b >= n || a == b)
            return fail(ctx, GPOP_ERR_INVALID_ARG, "invalid pair " + std::to_string(i));
    }
    const size_t traj_bytes = (size_t)steps * 3 * n * sizeof(double);
    cudaStream_t s = nullptr;
    ScopedBufs B(ctx);
    StartupTangents tan(ctx);
    DevBuf &dr = B.b[0], &dv = B.b[1], &dr0 = B.b[2], &dv0 = B.b[3], &ck = B.b[4],
           &traj = B.b[6], &dpairs = B.b[7], &units = B.b[8], &dseed = B.b[9], &out = B.b[10],
           &dgrad = B.b[11];
    if ((st = upload(ctx, dr, r_in, 3 * n, s)) != GPOP_OK || (st = upload(ctx, dv, v_in, 3 * n, s)) != GPOP_OK
        || (st = upload(ctx, dr0, r_in, 3 * n, s)) != GPOP_OK || (st = upload(ctx, dv0, v_in, 3 * n, s)) != GPOP_OK)
        return st;
    cudaError_t e;
    const int64_t U = 2 * n_pairs;
    if ((e = traj.ensure(3 * traj_bytes)) != cudaSuccess
        || (e = dpairs.ensure(2 * n_pairs * sizeof(int32_t))) != cudaSuccess
        || (e = units.ensure(2 * U * sizeof(int))) != cudaSuccess
        || (e = dseed.ensure(27 * U * sizeof(double))) != cudaSuccess
        || (e = out.ensure(n_pairs * (2 * sizeof(double) + sizeof(int)))) != cudaSuccess
        || (e = dgrad.ensure(6 * U * sizeof(double))) != cudaSuccess)
        return fail(ctx, GPOP_ERR_NOMEM, std::string("pair buffers: ") + cudaGetErrorString(e));
    double* tr = traj.as<double>();
    const size_t tn = (size_t)steps * 3 * n;
    gpop_propagator p;
    if ((st = begin(ctx, p, start, h, steps, n, dr.as<double>(), dv.as<double>(), s)) != GPOP_OK
        || (n <= kVarObjects && (st = tan.reserve(ctx, p)) != GPOP_OK)
        || (st = forward_run(ctx, p, steps, tr, tr + tn, tr + 2 * tn, ck, s)) != GPOP_OK)
        return st;
    if ((e = cudaMemcpyAsync(dpairs.p, pairs, 2 * n_pairs * sizeof(int32_t), cudaMemcpyHostToDevice, s)) != cudaSuccess)
        return cuda_fail(ctx, e, "pair upload");
    PairArgs pa;
    pa.n_obj = n;
    pa.n_pairs = n_pairs;
    pa.pairs = dpairs.as<int>();
    pa.steps = steps;
    pa.h = h;
    pa.traj_r = tr;
    pa.traj_v = tr + tn;
    pa.traj_a = tr + 2 * tn;
    pa.tca = out.as<double>();
    pa.miss = out.as<double>() + n_pairs;
    pa.closest = reinterpret_cast<int*>(out.as<double>() + 2 * n_pairs);
    pa.unit_obj = units.as<int>();
    pa.seed_step0 = units.as<int>() + U;
    pa.seeds = dseed.as<double>();
    if ((e = launch_pair_approach(pa, s)) != cudaSuccess)
        return cuda_fail(ctx, e, "pair approach kernel");
    ctx->launches++;
    std::vector<int> step0(U), obj(U);
    if ((e = cudaMemcpy(step0.data(), pa.seed_step0, U * sizeof(int), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cuda_fail(ctx, e, "pair approach kernel");
    std::copy(pairs, pairs + U, obj.begin());
    if ((st = run_adjoint(ctx, p, steps, dr0.as<double>(), dv0.as<double>(), tr, tr + 2 * tn, ck, tan, step0, obj, pa.unit_obj,
             pa.seed_step0, pa.seeds, dgrad.as<double>(), s))
        != GPOP_OK)
        return st;
    std::vector<double> g(6 * U);
    if ((e = cudaMemcpy(g.data(), dgrad.p, 6 * U * sizeof(double), cudaMemcpyDeviceToHost)) != cudaSuccess
        || (e = cudaMemcpy(tca, pa.tca, n_pairs * sizeof(double), cudaMemcpyDeviceToHost)) != cudaSuccess
        || (e = cudaMemcpy(miss, pa.miss, n_pairs * sizeof(double), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cuda_fail(ctx, e, "result download");
    std::copy(g.begin(), g.end(), grad); // [pair][object a: r0 3, v0 3 | object b: r0 3, v0 3]
    return GPOP_OK;
}

} // extern "C"
