// Device pieces shared by the kernels of the agent loop: the location lists,
// the movement decision, the histogram and sums, the draws of one agent.
#pragma once
#include "psim_device.cuh"

namespace psim {

// An error flag: in device memory for the kernels, and the host's word, which
// the host looks at after it has waited for the stream (no copy per call).
__device__ __forceinline__ void raise_error(const KArgs& k, uint32_t bits) {
    atomicOr(k.err, bits);
    *(volatile uint32_t*)k.err_host = 1u;
}

// Atomics nobody reads the result of, as the instructions.  With the atomic
// functions the decisions ran as many instructions but waited longer for
// memory (12.9 against 10.8 warps stalled on it per issue): 0.43 against 0.37
// ms of decisions a day at 2M agents and 4.16 against 3.69 at 20M.
__device__ __forceinline__ void red_add(uint32_t* p, uint32_t x) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(x) : "memory");
}
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long x) {
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(x) : "memory");
}
__device__ __forceinline__ void red_or(uint32_t* p, uint32_t x) {
    asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(x) : "memory");
}
__device__ __forceinline__ void red_and(uint32_t* p, uint32_t x) {
    asm volatile("red.relaxed.gpu.global.and.b32 [%0], %1;" ::"l"(p), "r"(x) : "memory");
}

__device__ __forceinline__ uint32_t wb_of(const KArgs& k, uint32_t i) {
    return k.m.state_wb[(uint8_t)k.a.state[i]];
}
__device__ __forceinline__ bool infected_of(const KArgs& k, uint32_t i) {
    return k.m.state_infected[(uint8_t)k.a.state[i]] != 0;
}
__device__ __forceinline__ uint8_t loc_open(const KArgs& k, uint32_t l) { return l < k.l.n ? k.l.open[l] : 0; }
__device__ __forceinline__ uint32_t loc_closed_until(const KArgs& k, uint32_t l) {
    return l < k.l.n ? k.l.closed_until[l] : 0u;
}
__device__ __forceinline__ uint32_t loc_qu(const KArgs& k, uint32_t l) { return l < k.l.n ? k.l.quarantine_until[l] : 0u; }
__device__ __forceinline__ uint32_t loc_type(const KArgs& k, uint32_t l) { return l < k.l.n ? k.l.type[l] : NONE; }

// Entry j of the per-agent location lists: x = location, y = its type.
__device__ __forceinline__ uint2 poss_entry(const KArgs& k, uint32_t j) {
    if (k.a.poss4) {
        const uint32_t v = k.a.poss4[j];
        return make_uint2(v & 0x3FFFFFFu, v >> 26);
    }
    return k.a.poss[j];
}

// RealMovementOps::findActualLocationForType, movementPolicies.h:69-122.
// f0, f1, f2: the types resolved by first match (home, school, work except in
// the plan helpers, movementPolicies.h:1073-1080, :1144, :1209-1214).
// [b, e): the agent's entries in the per-agent location list.
static __device__ uint32_t find_location_range(const KArgs& k, uint32_t b, uint32_t e, uint32_t lt, int retry,
                                        psim_stream* rng, uint32_t f0, uint32_t f1, uint32_t f2) {
    if (lt == f0 || lt == f1 || lt == f2) {
        for (uint32_t j = b; j < e; ++j) {
            const uint2 en = poss_entry(k, j);
            if (lt == en.y) return en.x;
        }
        return NONE;
    }
    uint32_t counter = 0, pos = 0, first = NONE;
    for (uint32_t j = b; j < e; ++j) {
        const uint2 en = poss_entry(k, j);
        if (lt == en.y) {
            if (counter == 0) {
                pos = j;
                first = en.x;
            }
            counter++;
        }
    }
    if (counter == 1) return first;
    if (counter > 1) {
        uint32_t counter2 = counter, rand_idx = counter2;
        // the reference loops until the pick is open or its one retry is
        // spent: a second pass always ends (retry is 0 by then)
        for (int pass = 0; pass < 2; ++pass) {
            while (rand_idx == counter2) rand_idx = psim_below(rng, counter);
            counter2 = 0;
            for (uint32_t j = pos; j < e; ++j) {
                const uint2 en = poss_entry(k, j);
                if (lt == en.y) {
                    if (counter2 == rand_idx) {
                        if (retry && loc_open(k, en.x) == 0) {
                            retry = 0;
                            break;
                        }
                        return en.x;
                    }
                    counter2++;
                }
            }
        }
    }
    return NONE;
}

// The same for agent i by its list's layout; lb: the list's first entry.
__device__ __forceinline__ uint32_t find_location_at(const KArgs& k, uint32_t i, uint32_t layout, uint32_t lb,
                                                     uint32_t lt, int retry, psim_stream* rng, uint32_t f0,
                                                     uint32_t f1, uint32_t f2) {
    if (layout == 0) return find_location_range(k, lb, k.a.loc_offset[i + 1], lt, retry, rng, f0, f1, f2);
    if (lt >= LAYOUT_TYPES) return NONE;
    const uint32_t e = k.m.layout[layout * LAYOUT_TYPES + lt];
    const uint32_t count = e >> 8, first = lb + (e & 0xFFu);
    if (count == 0) return NONE;
    uint32_t pick = 0;
    const bool any = count > 1 && lt != f0 && lt != f1 && lt != f2;
    if (any) pick = psim_below(rng, count);
    uint32_t loc = k.a.poss4[first + pick] & 0x3FFFFFFu;
    if (any && retry && loc_open(k, loc) == 0) {
        // its one retry: another pick, open or not
        const uint32_t before = pick;
        while (pick == before) pick = psim_below(rng, count);
        loc = k.a.poss4[first + pick] & 0x3FFFFFFu;
    }
    return loc;
}

__device__ __forceinline__ uint32_t find_location3(const KArgs& k, uint32_t i, uint32_t lt, int retry, psim_stream* rng,
                                                   uint32_t f0, uint32_t f1, uint32_t f2) {
    return find_location_at(k, i, k.a.layout[i], k.a.loc_offset[i], lt, retry, rng, f0, f1, f2);
}

__device__ __forceinline__ uint32_t find_location(const KArgs& k, uint32_t i, uint32_t lt, int retry, psim_stream* rng) {
    return find_location3(k, i, lt, retry, rng, k.p.home_type, k.p.school_type, k.p.work_type);
}

// A location quarantine written by a decision at step t: merged into
// quarantine_until by the scan of step t (build[3] = the step whose decisions
// wrote; every writer of a step stores the same value).
__device__ __forceinline__ void qu_write(const KArgs& k, uint32_t loc, uint32_t until, uint32_t t) {
    if (loc < k.l.n) {
        atomicMax(&k.l.qu_pending[loc], until);
        k.l.build[3] = t;
        k.l.build[4] = 1u;
    }
}

// RealMovementOps::quarantineAgent, movementPolicies.h:176-245
// Returns whether the agent was quarantined (its flag set).  The stream is a
// copy: a decision that quarantines draws nothing after it.
template <int POL>
__device__ __forceinline__ bool quarantine_agent(const KArgs& k, uint32_t i, uint32_t t, uint32_t until,
                                              psim_stream rng_copy) {
    psim_stream* rng = &rng_copy;
    const psim_params& p = k.p;
    if (POL == 0 || p.quarantine_policy == 0) return false;
    if (k.a.st_diagnosed_ts[i] > 0 && !infected_of(k, i) && !p.quarantine_immune) return false;
    if (!k.a.diagnosed[i] && k.a.st_immunization_ts[i] > 0 && !p.quarantine_immune) return false;
    k.a.quarantined[i] = 1;
    k.a.st_quarantined_ts[i] = t;
    uint32_t prev_until = k.a.st_quarantined_until[i];
    k.a.st_quarantined_until[i] = until;
    k.a.st_days_in_quarantine[i] += (until - t) / (24u * 60u / p.time_step);
    if (k.a.diagnosed[i]) {
        uint32_t my_home = find_location(k, i, p.home_type, 0, rng);
        if (p.quarantine_policy > 1) qu_write(k, my_home, until, t);
        if (p.quarantine_policy > 2 && prev_until < t) {
            uint32_t classroom = find_location(k, i, p.classroom_type, 0, rng);
            uint32_t work = find_location(k, i, p.work_type, 0, rng);
            uint32_t to_close[2] = {classroom, work};
            for (int c = 0; c < 2; ++c) {
                uint32_t loc = to_close[c];
                if (loc != NONE && (loc_type(k, loc) == p.work_type || loc_type(k, loc) == p.classroom_type) &&
                    loc_qu(k, loc) < t && loc_open(k, loc) && loc_closed_until(k, loc) < t)
                    qu_write(k, loc, until, t);
            }
        }
    }
    return true;
}

// returns the decision word's flags of what it set
template <int POL>
__device__ __forceinline__ uint32_t diagnose_and_quarantine(const KArgs& k, uint32_t i, uint32_t t, uint32_t sum,
                                                         psim_stream rng) {
    const uint32_t dt = k.p.time_step;
    k.a.diagnosed[i] = 1;
    const uint32_t ts = sum == 24u * 60u / dt ? t + 1u : t;
    k.a.st_diagnosed_ts[i] = ts;
    return DW_DIAGNOSED | (ts > 0 ? DW_DIAG_TS : 0u) |
           (quarantine_agent<POL>(k, i, t, t + k.p.quarantine_length * 24u * 60u / dt, rng) ? DW_QUARANTINED : 0u);
}

// S: the agent's countdown (stepsUntilMove) as the decision just set it;
// cur: the agent's location as the decision left it
__device__ __forceinline__ void stayed_home_check(const KArgs& k, uint32_t i, uint32_t agent_home, uint32_t cur,
                                                  uint32_t S) {
    if (agent_home != NONE && cur != agent_home && S > k.hour_steps) k.a.stayed_home[i] = 0;
}

// The agent's decision word (DW_*) from its fields; t = the first timestep it
// is used at.
__device__ __forceinline__ uint32_t decision_word(const KArgs& k, uint32_t i, uint32_t t) {
    const uint32_t type = k.a.type[i], st = (uint8_t)k.a.state[i], age = k.a.age[i];
    const bool quar = k.a.quarantined[i] != 0, diag = k.a.diagnosed[i] != 0, no_work = k.a.no_work[i] != 0;
    const bool hosp = k.a.st_hospitalized_until[i] > t, diag_ts = k.a.st_diagnosed_ts[i] > 0;
    const bool inf = k.a.infectious[i] != 0.0f;
    return type | (uint32_t)k.m.state_wb[st] << DW_WB_SHIFT | (quar ? DW_QUARANTINED : 0u) | (hosp ? DW_HOSPITAL : 0u) |
           (diag ? DW_DIAGNOSED : 0u) | (diag_ts ? DW_DIAG_TS : 0u) | (inf ? DW_INFECTIOUS : 0u) |
           (no_work ? DW_NO_WORK : 0u) | (age >= k.p.school_age_restriction ? DW_TOO_OLD : 0u) |
           (uint32_t)k.a.layout[i] << DW_LAYOUT_SHIFT;
}

// What a decision reads of its agent, loaded together before it starts: the
// decision word, the current location, the agent's first entry in the
// per-agent location lists, the replica.
struct DecisionIn {
    uint32_t w, loc, lb, rep;
};
__device__ __forceinline__ void decision_in(const KArgs& k, uint32_t i, DecisionIn& d) {
    d.loc = k.a.location[i];
    d.lb = k.a.loc_offset[i];
    d.rep = k.r.n == 1 ? 0u : k.a.rep[i];
}

// A location's flag word (LF_*): the running day's, or from the location's
// fields (the per-phase entry points).  A location out of range is closed and
// of no type, as its fields read one by one would be.
template <bool DAY>
__device__ __forceinline__ uint32_t loc_flags(const KArgs& k, uint32_t loc, uint32_t t) {
    if (loc >= k.l.n) return LF_TYPE;
    if (DAY) return k.l.lflags[loc];
    return k.l.type[loc] | (k.l.open[loc] ? LF_OPEN : 0u) | (k.l.closed_until[loc] > t ? LF_CLOSED : 0u) |
           (k.l.quarantine_until[loc] > t ? LF_QUARANTINE : 0u);
}
// closed by its open flag or its closing time
__device__ __forceinline__ bool closed_at(const KArgs& k, uint32_t loc, uint32_t f, uint32_t t) {
    return !(f & LF_OPEN) || ((f & LF_CLOSED) && k.l.closed_until[loc] > t);
}
__device__ __forceinline__ bool quarantine_type(const KArgs& k, uint32_t ty) {
    return ty == k.p.home_type || ty == k.p.school_type || ty == k.p.classroom_type || ty == k.p.work_type;
}

// The full per-agent decision of doMovement once the countdown reached zero
// (movementPolicies.h:333-1040).  The curfew and countdown prologue is in
// move_agent.  S receives the agent's new countdown (stepsUntilMove after
// the step); the caller turns it into the absolute timestamp of the next
// decision, cur the agent's location after it (d.loc before).  Returns the
// agent's decision word after it.
//
// The decisions are bound by the chain of dependent loads (word, location
// list, window, chosen location's flags) and by instructions, not by bytes:
// the countdowns of every event at every step come from a table computed on
// the host (no divisions here), a location's flags are one word, the home is
// looked up once, and an entry of a location list is found by the list's
// layout.  22 us of decisions a step at 2M agents (17 now), against 25 without
// those; the rare quarantine out of line (its arguments through memory) took
// 26, and the location list in registers 23.6.
//
// POL: the policies compiled in: 0 neither quarantine nor curfew, 1 no curfew,
// 2 all (their code costs every decision registers and instructions).
template <bool DAY, int POL>
__device__ __forceinline__ uint32_t move_decide(const KArgs& k, uint32_t i, uint32_t t, uint32_t step, uint32_t day,
                                                uint32_t sum, psim_stream* rng, uint32_t& S, const DecisionIn& d,
                                                uint32_t& cur) {
    const psim_params& p = k.p;
    const bool qrule = POL > 0 && p.quarantine_policy > 1;
    const uint32_t f_now = qrule ? loc_flags<DAY>(k, d.loc, t) : 0u;
    // the quarantine end of a location whose quarantine sends home, else 0
    auto quarantine_end = [&](uint32_t loc, uint32_t f) {
        return (f & LF_QUARANTINE) && quarantine_type(k, f & LF_TYPE) ? k.l.quarantine_until[loc] : 0u;
    };
    auto fl = [&](uint32_t lt, int retry) {
        return find_location_at(k, i, d.w >> DW_LAYOUT_SHIFT, d.lb, lt, retry, rng, p.home_type, p.school_type,
                                p.work_type);
    };
    uint32_t w = d.w;
    if ((w & DW_QUARANTINED) && k.a.st_quarantined_until[i] <= t) {
        w &= ~DW_QUARANTINED;
        k.a.quarantined[i] = 0;
    }
    // quarantine_agent and the word's flag
    auto quarantine = [&](uint32_t until) {
        if (quarantine_agent<POL>(k, i, t, until, *rng)) w |= DW_QUARANTINED;
    };

    cur = d.loc;
    const uint32_t wb = (w >> DW_WB_SHIFT) & 7u;
    if (wb == WB_D) {
        S = NONE;
        cur = k.r.cemetery[d.rep];
        k.a.location[i] = cur;
        return w;
    }
    // the first match, no draw (find_location_range): the same at every use
    const uint32_t agent_home = fl(p.home_type, 0);

    // in hospital: for another disease, or severe
    uint32_t h_until = 0;
    if ((w & DW_HOSPITAL) && wb != WB_S) {
        h_until = k.a.st_hospitalized_until[i];
        if (k.a.st_hospitalized_ts[i] > t || h_until <= t) h_until = 0;
    }
    if (wb == WB_S || h_until) {
        S = h_until ? min(h_until - t - 1u, sum) : sum;
        cur = fl(p.hospital_type, 0);
        k.a.location[i] = cur;
        if ((w & (DW_DIAGNOSED | DW_INFECTIOUS)) == DW_INFECTIOUS) w |= diagnose_and_quarantine<POL>(k, i, t, sum, *rng);
        return w;
    }
    // sent home: by the quarantine of the current location, by the agent's own
    const uint32_t qu_now = quarantine_end(d.loc, f_now);
    if (t < qu_now) {
        if (!(w & DW_QUARANTINED)) quarantine(qu_now);
        if (w & DW_QUARANTINED) {
            S = min(qu_now - t - 1u, sum);
            if (agent_home != cur) k.a.location[i] = agent_home;
            cur = agent_home;
            return w;
        }
    }
    if (POL > 0 && p.quarantine_policy > 0 && (w & (DW_DIAGNOSED | DW_DIAG_TS | DW_QUARANTINED))) {
        const uint32_t ql = p.quarantine_length * 24u * 60u / p.time_step;
        if ((w & (DW_DIAGNOSED | DW_QUARANTINED)) || t - k.a.st_diagnosed_ts[i] < ql) {
            if (!(w & DW_QUARANTINED)) quarantine(t + ql);
            if (w & DW_QUARANTINED) {
                cur = agent_home;
                k.a.location[i] = cur;
                S = sum;
                return w;
            }
        }
    }

    // schedule window (AgentTypeList::getOffsetIndex, agentType.cpp:13-15;
    // the window of the slot at this step, movementPolicies.h:585-603, from
    // the table the host computed)
    const uint32_t agent_type = w & DW_TYPE;
    const uint4* wp = reinterpret_cast<const uint4*>(k.m.window + ((size_t)(7u * wb + day + agent_type * 28u) * k.spd + step));
    const uint4 win = wp[0];
    const uint4 first = wp[1];  // DecChoice
    uint32_t new_type = NONE;
    // the chosen location and its flag word
    uint32_t spec_loc = NONE, spec_f = 0u;
    if (win.x) {  // Case 2 and 4: an event is active
        uint32_t num_pot = win.x, picked = 0;
        uint32_t s_steps = first.y, s_draw = first.z;
        new_type = first.x;
        if (num_pot != 1) {
            // U > chance of the first event, in integers: U = K 2^-53 and
            // chance 2^53 (exact in float), so K > floor(chance 2^53); the
            // few that go on compare in double as the reference does
            const uint64_t K = psim_u53(rng);
            const float c0 = __uint_as_float(first.w);
            if (c0 < 0.0f || (c0 < 1.0f && K > __float2ull_rd(c0 * 9007199254740992.0f))) {
                const double rnd = (double)K * (1.0 / 9007199254740992.0);
                double thr = c0;
                uint32_t idx = 0;
                while (rnd > thr && idx < num_pot) {
                    idx++;
                    thr += k.m.ev_chance[win.y + idx];
                }
                if (idx == num_pot) idx--;
                picked = idx;
                const uint4 c = reinterpret_cast<const uint4*>(k.m.choice)[win.z + idx];
                new_type = c.x;
                s_steps = c.y;
                s_draw = c.z;
            }
        }
        if ((w & DW_NO_WORK) && new_type == p.work_type) {
            new_type = p.home_type;
            num_pot = 1;
            if (!(w & DW_QUARANTINED)) k.a.st_days_in_quarantine[i]++;
        }
        uint32_t new_loc = new_type == p.home_type ? agent_home : fl(new_type, num_pot == 1);
        const bool too_old = (w & DW_TOO_OLD) && (new_type == p.school_type || new_type == p.classroom_type);
        const bool barred = p.lockdown_nonvacc && k.a.st_immunization_ts[i] == 0;
        spec_loc = new_loc;
        spec_f = loc_flags<DAY>(k, new_loc, t);
        if (too_old || barred || (new_type != p.work_type && closed_at(k, new_loc, spec_f, t))) {
            if (num_pot > 1) {
                double rnd = psim_u01(rng) * 1.0;
                double pc = k.m.ev_chance[win.y + picked];
                double thr = (picked == 0) ? 0.0 : k.m.ev_chance[win.y] / (1.0 - pc);
                uint32_t idx = 0;
                while (rnd > thr && idx < num_pot) {
                    idx++;
                    thr += (picked == idx) ? 0.0 : k.m.ev_chance[win.y + idx] / (1.0 - pc);
                }
                if (idx == num_pot) idx--;
                const uint4 c = reinterpret_cast<const uint4*>(k.m.choice)[win.z + idx];
                new_type = c.x;
                s_steps = c.y;
                s_draw = c.z;
                new_loc = new_type == p.home_type ? agent_home : fl(new_type, 0);
                if (too_old || barred ||
                    (new_type != p.work_type && closed_at(k, new_loc, loc_flags<DAY>(k, new_loc, t), t)))
                    new_loc = agent_home;
            } else {
                new_loc = agent_home;
            }
        } else if (new_type == p.school_type) {
            uint32_t my_class = fl(p.classroom_type, 0);
            if (my_class != NONE && loc_closed_until(k, my_class) > t) new_loc = agent_home;
        }
        cur = new_loc;
        S = s_steps + psim_below(rng, s_draw);
        if (POL == 2 && agent_type + 1 == 7 && p.enable_curfew && (p.curfew_begin <= step || p.curfew_end > step)) {
            bool work_closed = new_type == p.work_type && (loc_open(k, new_loc) == 0 || loc_closed_until(k, new_loc) > t);
            if (work_closed || (new_type != p.work_type && new_type != p.home_type)) cur = agent_home;
        }
    } else if (win.w) {  // Case 3: the next event lies ahead
        S = first.y + psim_below(rng, first.z);
        if (S >= k.hour_steps) {
            new_type = p.home_type;
            cur = agent_home;
        } else if (S >= k.half_hour_steps) {
            new_type = p.public_type;
            cur = new_type == p.home_type ? agent_home : fl(new_type, 0);
        }
    } else {  // Case 1: no event for the rest of the day
        new_type = p.home_type;
        cur = agent_home;
        S = sum;
    }
    k.a.location[i] = cur;
    if (qrule) {
        const uint32_t f = cur == spec_loc ? spec_f : cur == d.loc ? f_now : loc_flags<DAY>(k, cur, t);
        const uint32_t qu = quarantine_end(cur, f);
        if (t < qu) {
            if (!(w & DW_QUARANTINED)) quarantine(qu);
            if (w & DW_QUARANTINED) {
                S = min(qu - t - 1u, sum);
                if (agent_home != cur) k.a.location[i] = agent_home;
                cur = agent_home;
                return w;
            }
        }
    }
    if ((w & (DW_DIAGNOSED | DW_INFECTIOUS)) == DW_INFECTIOUS &&
        (new_type == p.hospital_type || (new_type == p.doctor_type && psim_u01(rng) * 1.0 < 0.7)))
        w |= diagnose_and_quarantine<POL>(k, i, t, sum, *rng);
    stayed_home_check(k, i, agent_home, cur, S);
    S = S - 1u;
    return w;
}

// curfew prologue of doMovement (movementPolicies.h:267-326); returns true if
// the agent's step is finished (S, the countdown, then holds `sum`).
static __device__ bool curfew_prologue(const KArgs& k, uint32_t i, uint32_t t, uint32_t sum, psim_stream* rng, uint32_t& S) {
    const psim_params& p = k.p;
    uint32_t wb = wb_of(k, i);
    bool dead_or_hosp = (wb == WB_D || wb == WB_S);
    bool hosp_noncovid = (k.a.st_hospitalized_ts[i] <= t && k.a.st_hospitalized_until[i] > t);
    if (dead_or_hosp || hosp_noncovid) return false;
    if (k.a.type[i] + 1u == 7u) {
        uint32_t workplace = find_location(k, i, p.work_type, 0, rng);
        if (k.a.location[i] != workplace || workplace == NONE || loc_open(k, workplace) == 0) {
            k.a.location[i] = find_location(k, i, p.home_type, 0, rng);
            if (workplace == NONE || loc_open(k, workplace) == 0) {
                S = sum;
                return true;
            }
        }
        return false;
    }
    S = sum;
    k.a.location[i] = find_location(k, i, p.home_type, 0, rng);
    return true;
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---------------------------------------------------------------------------
// Per-agent pieces of a step.

struct StepClock {
    uint32_t t, step, day, sum;
    bool curfew_now;
};

__device__ __forceinline__ StepClock step_clock(const KArgs& k, uint32_t step) {
    StepClock c;
    c.t = k.clock->t0 + step;
    c.step = step;
    c.day = k.clock->day_of_week;
    c.sum = k.spd - step;  // the steps left of the day
    c.curfew_now = k.p.enable_curfew && k.p.curfew_begin == step;
    return c;
}

// The countdown of the reference (stepsUntilMove: decremented every step,
// a decision when it reaches zero) is kept as the absolute timestamp of the
// agent's next decision, move_at = t + 1 + stepsUntilMove after step t (u32
// arithmetic: the dead agents' NONE countdown wraps like the reference's).
// Before step t the countdown is move_at - t; only a decision or the curfew
// prologue writes move_at, so the steps in between touch nothing.  The
// library converts to and from countdowns at upload and download (time base
// t_next, psim_api.cu).
//
// Steps of the running day at which some agent decides: one bit per step in
// move_mask, set by whoever writes such a move_at (through a block-shared
// copy, one global atomic per word and block).  The day graph's kernels read
// it to skip the steps nobody decides at.
__device__ __forceinline__ void mask_clear_shared(uint32_t* s_mm) {
    for (uint32_t w = threadIdx.x; w < MOVE_MASK_WORDS; w += blockDim.x) s_mm[w] = 0u;
    __syncthreads();
}
__device__ __forceinline__ void mask_note(const KArgs& k, uint32_t* s_mm, uint32_t m) {
    const uint32_t s = m - k.clock->t0;
    if (s < k.spd) {
        // most deciders of a step land on a few steps: read before the
        // atomic, whose lanes on one word would queue
        const uint32_t bit = 1u << (s & 31u);
        if (!(s_mm[s >> 5] & bit)) atomicOr(&s_mm[s >> 5], bit);
    }
}
__device__ __forceinline__ void mask_flush(const KArgs& k, uint32_t* s_mm) {
    __syncthreads();
    for (uint32_t w = threadIdx.x; w < MOVE_MASK_WORDS; w += blockDim.x)
        if (s_mm[w]) atomicOr(&k.a.move_mask[w], s_mm[w]);
}

// doMovement for agent i at step c.t; s = its countdown before the step
// (move_at - c.t).  Writes move_at when the agent decides or the curfew
// prologue resets its countdown.  d: the decision's inputs.  Returns the
// agent's location after the step; w receives its decision word after it.
template <bool DAY, int POL>
__device__ __forceinline__ uint32_t move_agent(const KArgs& k, uint32_t i, const StepClock& c, uint32_t s,
                                               uint32_t* s_mm, DecisionIn d, uint32_t* w) {
    psim_stream rng;
    psim_stream_init(&rng, k.r.seed[d.rep], i - k.r.agent_off[d.rep], c.t, PSIM_PHASE_MOVE);
    bool done = false;
    uint32_t S = s;
    if (POL == 2 && c.curfew_now) {
        done = curfew_prologue(k, i, c.t, c.sum, &rng, S);
        d.loc = k.a.location[i];  // the prologue may have sent the agent home
    }
    uint32_t cur = d.loc;
    *w = d.w;
    if (!done) {
        if (S > 0)
            S = S - 1u;
        else
            *w = move_decide<DAY, POL>(k, i, c.t, c.step, c.day, c.sum, &rng, S, d, cur);
    }
    const uint32_t m = c.t + 1u + S;
    k.a.move_at[i] = m;
    mask_note(k, s_mm, m);
    return cur;
}

// Scan tiles: 256 threads x ITEMS locations (ITEMS = 2, 4 or 8, a tuning
// choice); the masks hold one 32-bit word per warp and item.
constexpr int SCAN_THREADS = 256;

// A location that receives an infectious term sets its hazard-mask bit at
// once, so the mask is always a superset of the locations with a nonzero sum
// (the day kernel's rebuild lists from it and clears the bits of zero sums;
// the per-phase scans recompute the bits of their dirty locations).
__device__ __forceinline__ void mark_hazardous(const KArgs& k, uint32_t loc) {
    red_or(&k.l.hmask[loc >> 5], 1u << (loc & 31u));
}

// The full pass of a day's first step (k_movement, after a reset of the
// sums): an agent whose location changed from loc0 to loc moves one count
// (two fire-and-forget reductions), and every infectious agent adds its term
// at its (new) location.  Returns whether the agent took a new location (its
// kernel then publishes the timestamp of the new locations, publish_moved).
__device__ __forceinline__ bool count_agent(const KArgs& k, bool act, uint32_t loc0, uint32_t loc, float inf,
                                            uint32_t variant) {
    const uint32_t L = k.l.n;
    if (act && loc >= L) {
        raise_error(k, ERR_LOCATION);
        loc = NONE;
    }
    const bool mv = act && loc != loc0;
    if (mv) {
        if (loc0 < L) red_add(&k.l.counts[loc0], 0u - 1u);
        if (loc != NONE) red_add(&k.l.counts[loc], 1u);
    }
    if (act && loc != NONE && inf > 0.0f) {
        const long long q = __float2ll_rn(inf * PSIM_FIX_SCALE_F);
        red_add(&k.l.sfix[(size_t)variant * L + loc], (unsigned long long)q);
        red_or(&k.l.smask[loc >> 5], 1u << (loc & 31u));
        mark_hazardous(k, loc);
    }
    return mv;
}

// Within a day the per-location sums persist: an agent changes them only
// when it moves or its infectiousness changes (a draw that infects).  The
// first step of a day (k_movement after a reset of the sums) adds every
// agent's term afresh.
// The agent went from (loc0, inf0, var0) to (loc, inf, var) in a day
// kernel's decision: its count moves, its fixed-point term leaves (loc0,
// var0) and joins (loc, var).  The day kernel computes every ratio from the
// sums, so it keeps no dirty marks (the day graph marks every location dirty
// at its start: a scan after it recomputes every ratio).  Returns whether the
// agent took a new location.
__device__ __forceinline__ bool count_agent_delta(const KArgs& k, bool act, uint32_t loc0, uint32_t loc, float inf0,
                                                  uint32_t var0, float inf, uint32_t var) {
    const uint32_t L = k.l.n;
    if (act && loc >= L) {
        raise_error(k, ERR_LOCATION);
        loc = NONE;
    }
    const bool mv = act && loc != loc0;
    if (mv) {
        if (loc0 < L) red_add(&k.l.counts[loc0], 0u - 1u);
        if (loc != NONE) red_add(&k.l.counts[loc], 1u);
    }
    if (act) {
        const long long q0 = (loc0 < L && inf0 > 0.0f) ? __float2ll_rn(inf0 * PSIM_FIX_SCALE_F) : 0ll;
        const long long q1 = (loc != NONE && inf > 0.0f) ? __float2ll_rn(inf * PSIM_FIX_SCALE_F) : 0ll;
        if (mv || q0 != q1 || var0 != var) {
            if (q0) red_add(&k.l.sfix[(size_t)var0 * L + loc0], (unsigned long long)(-q0));
            if (q1) {
                red_add(&k.l.sfix[(size_t)var * L + loc], (unsigned long long)q1);
                mark_hazardous(k, loc);
            }
        }
    }
    return mv;
}

// The full histogram of the current positions (after a reset of counts and sums).
__device__ __forceinline__ void count_full(const KArgs& k, bool act, uint32_t loc, float inf, uint32_t variant) {
    const uint32_t L = k.l.n;
    if (!act) return;
    if (loc >= L) {
        raise_error(k, ERR_LOCATION);
        return;
    }
    red_add(&k.l.counts[loc], 1u);
    if (inf > 0.0f) {
        const long long q = __float2ll_rn(inf * PSIM_FIX_SCALE_F);
        red_add(&k.l.sfix[(size_t)variant * L + loc], (unsigned long long)q);
        red_or(&k.l.smask[loc >> 5], 1u << (loc & 31u));
        mark_hazardous(k, loc);
    }
}

// CSR slot of an agent: a warp-aggregated returning atomic on the location's
// cursor, which the scan set to the location's first slot.  Warp-collective.
__device__ __forceinline__ uint32_t take_slot(const KArgs& k, bool ok, uint32_t loc) {
    if (!k.tune.agg_slot) return ok ? atomicAdd(&k.l.cursor[loc], 1u) : NONE;
    const unsigned valid = __ballot_sync(0xffffffffu, ok);
    uint32_t pos = NONE;
    if (ok) {
        const unsigned peers = __match_any_sync(valid, loc);
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(&k.l.cursor[loc], (uint32_t)__popc(peers));
        base = __shfl_sync(peers, base, leader);
        pos = base + (uint32_t)__popc(peers & lanemask_lt());
    }
    return pos;
}

__device__ __forceinline__ void store_slot(const KArgs& k, uint32_t pos, uint32_t i) {
    if (pos < k.a.n)
        k.l.csr_agents[pos] = i;
    else
        raise_error(k, ERR_LOCATION);
}

// Infection draws of agent i at location loc with hazard h0 of variant 0
// (LocationsList::infectAgents, locationList.h:233-310; DynamicPPState::gotInfected,
// dynamicPPState.cpp:235-244).  Returns the sum of min(1, p) over the draws.
// d p / d theta of one draw (p = r * s * sigma_band, r = 1 - exp(-x),
// x = k * S/n * w * season * dt), weighted by the replica's dL/dE, added to the
// block's FP64 accumulators
// x: the location's hazard argument k*S/n*w*season*dt for variant v; times:
// how many timesteps made this draw with the same p (negative: taken back)
static __device__ __noinline__ void adjoint_terms(const KArgs& k, uint32_t i, uint32_t loc, uint32_t v, uint32_t rep, float r,
                                           float su, float s_eff, double* s_grad, float x_f, int times) {
    const double g = k.adj.weight[rep] * (double)times;
    if (g == 0.0) return;
    const double x = (double)x_f;
    const double dpdx = (double)s_eff * (1.0 - (double)r);
    const double kf = (double)k.r.k_f[rep];
    if (kf != 0.0) atomicAdd(&s_grad[GRAD_K], g * dpdx * x / kf);
    const int slot = k.adj.type_slot[k.l.type[loc]];
    const double w = (double)k.l.infectiousness[loc];
    if (slot >= 0 && w != 0.0) atomicAdd(&s_grad[GRAD_W + slot], g * dpdx * x / w);
    atomicAdd(&s_grad[GRAD_SIGMA + k.a.band[i]], g * (double)r * (double)su);
}

__device__ __forceinline__ double draw_agent(const KArgs& k, uint32_t i, uint32_t loc, uint32_t t, float h0,
                                             double* s_grad) {
    const uint32_t N = k.a.n, L = k.l.n, V = k.m.n_variants;
    // the agent's fields load together (variant 0's susceptibility: a draw
    // that infects rewrites the later variants' before they are read)
    const uint32_t rep = k.a.rep[i];
    const float sigma = k.p.sigma_band[k.a.band[i]];
    const float su0 = k.a.susceptible[i];
    const unsigned long long seed = k.r.seed[rep];
    const uint32_t li = i - k.r.agent_off[rep];
    double term_sum = 0.0;
    for (uint32_t v = 0; v < V; ++v) {
        const float h = v == 0 ? h0 : k.l.hazard[(size_t)v * L + loc];
        if (!(h > 0.0f)) continue;
        if (!k.r.variant_active[rep * V + v]) continue;
        const float su = v == 0 ? su0 : k.a.susceptible[(size_t)v * N + i];
        const float s_eff = su * sigma;
        if (!(s_eff > 0.0f)) continue;
        const float pf = h * s_eff;
        term_sum += pf < 1.0f ? (double)pf : 1.0;
        if (k.adj.on && pf < 1.0f)
            adjoint_terms(k, i, loc, v, rep, h, su, s_eff, s_grad, k.l.hazard_x[(size_t)v * L + loc], 1);
        const double U = psim_u01_once(seed, li, t, PSIM_PHASE_INFECT + v);
        if (U < (double)pf) {
            k.a.state[i] = (int8_t)k.m.first_infected;
            k.a.variant[i] = (uint8_t)v;
            k.a.days[i] = -2;
            update_meta(k, i);
            k.a.st_infected_ts[i] = t;
            k.a.st_infected_count[i] = k.a.st_infected_count[i] + 1;
            k.a.st_infected_loc[i] = loc;
            k.a.st_worst_state[i] = (int8_t)k.m.first_infected;
            k.a.st_worst_ts[i] = t;
            k.a.st_variant_mask[i] |= 1u << v;
        }
    }
    return term_sum;
}

__device__ __forceinline__ void grad_begin(const KArgs& k, double* s_grad) {
    if (!k.adj.on) return;
    if (threadIdx.x < GRAD_N) s_grad[threadIdx.x] = 0.0;
    __syncthreads();
}

// one global atomic per block and parameter
__device__ __forceinline__ void grad_end(const KArgs& k, double* s_grad) {
    if (!k.adj.on) return;
    __syncthreads();
    if (threadIdx.x < GRAD_N && s_grad[threadIdx.x] != 0.0) atomicAdd(&k.adj.grad[threadIdx.x], s_grad[threadIdx.x]);
}

// expected-infection accumulation: one atomic per replica present in the warp
__device__ __forceinline__ void add_expected(const KArgs& k, bool act, uint32_t i, double term) {
    const unsigned am = __ballot_sync(0xffffffffu, act && term != 0.0);
    if (!(act && term != 0.0)) return;
    const uint32_t rep = k.a.rep[i];
    const unsigned peers = __match_any_sync(am, rep);
    const int leader = __ffs(peers) - 1;
    unsigned rest = peers;
    double tot = 0.0;
    while (rest) {
        const int src = __ffs(rest) - 1;
        tot += __shfl_sync(peers, term, src);
        rest &= rest - 1;
    }
    if ((int)(threadIdx.x & 31) == leader) atomicAdd(&k.r.expected[rep], tot);
}

// Timeline stamps of the profiled day graph (KArgs::prof): one atomic per
// block, from thread 0, on the global nanosecond timer.
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// the block's entry (no wait for the other threads)
__device__ __forceinline__ void prof_enter(const KArgs& k, uint32_t slot) {
    if (k.prof && threadIdx.x == 0) atomicMax(&k.prof[slot], ~global_ns());
}
// the block's threads are past this point (every thread calls it)
__device__ __forceinline__ void prof_mark(const KArgs& k, uint32_t slot) {
    if (!k.prof) return;
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&k.prof[slot], global_ns());
}

// Where a warp's lanes put the entries they flagged (bits of `flags`, one
// per agent of the lane) in a block's list: the first one's place (one
// shared-memory atomic per warp).
__device__ __forceinline__ uint32_t list_place(uint32_t flags, uint32_t* s_cnt) {
    const int lane = threadIdx.x & 31;
    const uint32_t mine = __popc(flags);
    uint32_t inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    uint32_t base = 0;
    if (lane == 31 && inc) base = atomicAdd(s_cnt, inc);
    return __shfl_sync(0xffffffffu, base, 31) + inc - mine;
}

}  // namespace psim
