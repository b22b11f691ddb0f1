// The packet walk of the forward solves and of the adjoint's replays.
//
// Replaces the reference's per-cycle generate + integrate launches
// (modules/particle/evolve/generate_par.h:51-62 -> ker_gen, then
// evolve/integrator.h:47-63 -> ker_itg running photon::cart_t::proc) by one
// persistent launch.  Each warp owns a pool of packets in global memory
// (48 MB at most together, of which the peel-off queue's stream evicts a part
// from L2: 3.1 GB written and 1.4 GB read per 1e7 packets of the clump) and
// works on it in three phases:
//   walk    the lanes take ready packets and march each to the end of its
//           flight: an interaction, the domain's boundary or a step limit;
//   events  the interactions, 32 together: albedo, peel-off ray, roulette,
//           scattering, new optical depth;
//   births  the ended packets: escape tallies and records; the slot takes the
//           next packet of the launch.
// The lists of ready, interacting and ended packets are in shared memory.  A
// flight that is still under way when its warp has better things to do goes
// back to the ready packets as it is.
//
// What bounded the walk before was its lanes: one packet per lane, phases
// scheduled by ballots, gave 14 lanes to a segment, 13 to an interaction and
// 11 to an instruction, all at 59% issue; and an interaction's rejection loop
// ran as long as its longest lane.  With the pools a segment has 18 to 21
// lanes, an interaction 29, and the spare lanes of a batch try the next draws
// of the others (scatter_warp).  Tried on the way: one pool per block of 256
// with a barrier between the phases (8.3 ms for 1e6 packets of the clump,
// half of the warps waiting at the barrier); packets as 128-byte records
// (6.9 ms: 72% of the L1's data pipe); the crossed axis by branches (6.1 ms;
// by selects, below, 5.6 ms).  Warp pools, fields in chunks of 32 and the
// interaction's packet read again for its second half: 4.2 ms, against 6.0 ms
// for the walk before.  With the extinction ahead (AHEAD, below), against the
// walk before: the clump 5.96 -> 3.99 ms per 1e6 packets, 1.85 -> 1.36 ms per
// 3e5, 0.56 -> 0.24 ms per 2000; the atmosphere 11.5 -> 8.5 ms per 1e6, 2.57 ->
// 1.15 ms per 1117; the large scene 11.5 -> 8.0 ms per 2e6; the adjoint's replay
// 4.49 -> 3.86 ms.
#include "kp_transport.cuh"

#include <algorithm>
#include <mutex>
#include <vector>

namespace kp
{

// 32 packets between phases, field by field: the lanes of a warp, which take
// any packets of its pool, touch one 128-byte line per chunk and word.  The
// words up to `stop` are what a flight needs, the rest what interactions,
// births and tallies use.
struct __align__( 128 ) pool_chunk_t
{
    double   x[ 3 ][ 32 ];
    float    tau[ 32 ];
    int      n_left[ 32 ];         // segments the packet may still walk in this launch
    int      b[ 32 ], c[ 3 ][ 32 ];
    float    d[ 3 ][ 32 ];
    int      stop[ 32 ];           // its segments so far plus n_left
    float    e1[ 3 ][ 32 ], S[ 3 ][ 32 ], w[ 32 ];
    int      n_scat[ 32 ];
    uint32_t k1[ 32 ], pid_lo[ 32 ], pid_hi[ 32 ], draw[ 32 ];
    int      link[ 32 ];           // TAPE: the packet's last task, ADJ1: its next
    int      si[ 32 ];             // scene of a batched launch
    union
    {
        int    batch[ 32 ];        // pid % n_batches
        double R[ 32 ];            // ADJ1: the score of the interactions ahead
    };
};
static_assert( sizeof( pool_chunk_t ) == 32 * 128, "pool chunk" );

namespace
{

// Scheduling, times for 1e6 packets of the clump and of the atmosphere (FETCH
// and PARK: of the clump and of the large scene's 2e6).
#ifndef KP_WALK_FETCH
#define KP_WALK_FETCH 8              // idle lanes that wait for a fetch batch (4 and 12:
                                     // within 1%; 16: 4.00 against 3.97 ms, 8.40
                                     // against 7.96)
#endif
#ifndef KP_WALK_HOP
#define KP_WALK_HOP 6                // lanes that wait for a block hand-off (8: 4.20
                                     // against 4.21 ms, 8.56 against 8.39)
#endif
#ifndef KP_WALK_ROUND
#define KP_WALK_ROUND 4              // segments per scheduling round (3: 4.27 against
                                     // 4.21 ms, 8.62 against 8.39)
#endif
#ifndef KP_WALK_PARK
#define KP_WALK_PARK 20              // flights under way that may be put back (8: 4.51
                                     // against 3.97 ms, 8.55 against 7.96; 14: 4.08
                                     // and 8.13; 26 and 32: within 1%)
#endif
#ifndef KP_WALK_MINB
#define KP_WALK_MINB 5               // resident blocks the registers allow (96 registers;
                                     // 6, with 80 and spills: 4.38 against 4.21 ms,
                                     // 9.06 against 8.39)
#endif

constexpr int WALK_WARPS = WALK_THREADS / 32;

// How a flight ended; a list entry of an ended packet is its slot and this.
enum end_kind { END_NONE = 0, END_ESCAPED = 1, END_LOST = 2, END_STEPS = 3, END_EVENT = 4 };
constexpr int SLOT_BITS = 12;
static_assert( KP_WALK_POOL <= 1 << SLOT_BITS, "pool slot in a list entry" );

struct walk_shared_t
{
    unsigned long long cnt[ KP_NCOUNTERS ];
    struct warp_t
    {
        unsigned short ready[ KP_WALK_POOL ], ev[ KP_WALK_POOL ], dead[ KP_WALK_POOL ];
        unsigned char  pend[ 32 ];
    } w[ WALK_WARPS ];
};

// Whether a warp with `ev` packets at their events and `ready` others runs an
// event batch: a full one, or, with few packets left, the larger part of them.
// (A walk phase left for events that are due is followed by their batch, so
// every pass makes progress.)
__device__ __forceinline__ bool events_due( const fwd_params_t & P, int ev, int ready )
{
    return ev >= P.ev_pool || ( ev > 0 && ev >= ready && ev + ready < P.ev_pool + 8 );
}

// phys::scatter for the lanes with `need`, the whole warp taking part: the
// trials of a lane are draws draw, draw + 1, ... of its own counter, so a lane
// that has been accepted (or has nothing to scatter) tries the next draws of
// one that has not.  Each lane keeps its first accepted trial, as the trials
// one after another would.  A batch of 32 needs about 3 rounds instead of the
// longest lane's 6 or 7 (a trial is accepted with probability about 0.52).
__device__ __forceinline__ void scatter_warp( const phys::phase_t & ph, phys::rng_t & rng,
                                              phys::v3 & d, phys::v3 & e1, phys::stokes_t & S,
                                              bool need, unsigned char * pend )
{
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    float mu = 0.0f, a = 1.0f, b = 0.0f;
    int   tried = 0;
    const bool had = need;
    for( ;; )
    {
        const unsigned m = __ballot_sync( FULL, need );
        if( m == 0u ) break;
        // trials of each lane this round: 2^k, as many as the warp has lanes for
        const int n = __popc( m ), k = 5 - ( 32 - __clz( n - 1 ) ), q = 1 << k;
        const int rank = __popc( m & ( ( 1u << lane ) - 1u ) );
        if( need ) pend[ rank ] = ( unsigned char ) lane;
        __syncwarp(  );
        const int grp = ( int ) lane >> k, sub = ( int ) lane & ( q - 1 );
        const int from = pend[ grp < n ? grp : 0 ];
        const float    Sq = __shfl_sync( FULL, S.q, from ), Su = __shfl_sync( FULL, S.u, from );
        const uint32_t k1 = __shfl_sync( FULL, rng.k1, from );
        const uint32_t lo = __shfl_sync( FULL, rng.pid_lo, from );
        const uint32_t hi = __shfl_sync( FULL, rng.pid_hi, from );
        const uint32_t dr = __shfl_sync( FULL, rng.draw, from );
        const int      tr = __shfl_sync( FULL, tried, from ) + sub;     // this trial's number
        float tmu, ta, tb;
        bool  ok = phys::scatter_trial( ph, phys::philox( phys::u4 { dr + sub, lo, hi, 0x4B50u }, rng.k0, k1 ),
                                        Sq, Su, tmu, ta, tb );
        ok = ( ok || tr == 63 ) && grp < n && tr < 64;   // the 64th is kept as it is
        const unsigned acc = __ballot_sync( FULL, ok );
        const unsigned mine = need ? ( acc >> ( rank << k ) ) & ( FULL >> ( 32 - q ) ) : 0u;
        const int first = __ffs( mine ) - 1;
        const int src = need ? ( rank << k ) + ( first < 0 ? 0 : first ) : 0;
        const float gmu = __shfl_sync( FULL, tmu, src ), ga = __shfl_sync( FULL, ta, src ),
                    gb = __shfl_sync( FULL, tb, src );
        if( need )
        {
            rng.draw += first < 0 ? q : first + 1;
            tried += q;
            if( first >= 0 ) { mu = gmu; a = ga; b = gb; need = false; }
        }
        __syncwarp(  );
    }
    if( had )
        phys::scatter_apply( ph, mu, a, b, __fadd_rn( __fmul_rn( a, a ), __fmul_rn( b, b ) ), d, e1, S );
}

// IMG: peel-off rays are queued for k_peel (when the queue is full they are
// marched at once by the lane; not in the adjoint's replay, which flags the
// packet).  TAPE: they are linked per packet.  FLUX: every segment adds
// w * dl / volume to its cell's flux tally, the path-length estimator of
// photon::cart_t::proc_phys (modules/particle/radiation/photon.h:73-83).
// RESUME: packets an earlier call suspended come first, and a packet that
// reaches its step budget is written to P.rs_out.
// KIND WALK_ADJ0, WALK_ADJ1: the adjoint's replays (kp_adjoint.cu).  The
// first queues the rays as a taped solve does and tallies nothing; the second
// deposits -R * length along the walk and R / sigma_sca at interactions, R
// the sum of the scores of the interactions ahead.
template< int TALLY, int KIND, bool IMG, bool TAPE, bool FLUX, bool RESUME >
__global__ void __launch_bounds__( WALK_THREADS, KP_WALK_MINB )
k_walk( const __grid_constant__ fwd_params_t P )
{
    constexpr bool ADJ = KIND == WALK_ADJ1, TALLIES = KIND == WALK_FORWARD;
    // AHEAD: the next cell's extinction is loaded before this cell's decides
    // whether the flight ends in it.  With rays to queue: the large scene's
    // walk, beyond L2, 8.80 -> 8.02 ms, 1e6 packets of the clump 4.14 -> 4.01,
    // the taped walk 3.16 -> 3.01.  Not where every segment deposits (the
    // replay 3.85 -> 4.35 ms, the flux walk 1.91 -> 2.08), nor in the walks
    // without an image (the atmosphere 8.5 -> 8.8, 64 scenes 3.35 -> 3.50).
    constexpr bool AHEAD = IMG && ! ADJ && ! FLUX;
    __shared__ walk_shared_t sh;
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u, below = ( 1u << lane ) - 1u;
    auto & L = sh.w[ threadIdx.x >> 5 ];
    pool_chunk_t * const pool = P.pool + ( ( size_t ) blockIdx.x * WALK_WARPS + ( threadIdx.x >> 5 ) )
                                         * ( ( P.pool_n + 31 ) >> 5 );
    const int nc0 = P.m.nc[ 0 ], nc1 = P.m.nc[ 1 ], nc2 = P.m.nc[ 2 ];
    unsigned n_steps_done = 0, n_peel_done = 0;
    const long long n_items = P.n_packets + ( RESUME ? P.rs_n_in : 0 );

    if( threadIdx.x < KP_NCOUNTERS ) sh.cnt[ threadIdx.x ] = 0;
    for( int k = lane; k < P.pool_n; k += 32 ) L.dead[ k ] = ( unsigned short ) k;
    __syncthreads(  );
    int n_ready = 0, n_ev = 0, n_dead = P.pool_n;      // the same in every lane of the warp

    auto load_packet = [ & ]( const pool_chunk_t & o, int i, packet_t & p )
    {
        #pragma unroll
        for( int a = 0; a < 3; ++ a ) { p.x[ a ] = o.x[ a ][ i ]; p.c[ a ] = o.c[ a ][ i ]; }
        p.tau = o.tau[ i ]; p.n_steps = o.stop[ i ] - o.n_left[ i ]; p.b = o.b[ i ];
        p.d = phys::v3 { o.d[ 0 ][ i ], o.d[ 1 ][ i ], o.d[ 2 ][ i ] };
        p.e1 = phys::v3 { o.e1[ 0 ][ i ], o.e1[ 1 ][ i ], o.e1[ 2 ][ i ] };
        p.S = phys::stokes_t { o.S[ 0 ][ i ], o.S[ 1 ][ i ], o.S[ 2 ][ i ] };
        p.w = o.w[ i ]; p.n_scat = o.n_scat[ i ];
        p.rng = phys::rng_t { P.seed, o.k1[ i ], o.pid_lo[ i ], o.pid_hi[ i ], o.draw[ i ] };
    };
    auto add_flux = [ & ]( size_t ic, double v )
    {
        if( TALLY == KP_TALLY_FLOAT && P.flux_sum )
            atomicAdd( P.flux_sum + ic, v );
        else
            add_grad< TALLY >( P.flux, P.c_flux, ic, v, P.flux_scale );
    };
    // RESUME: the packet leaves this launch unfinished
    auto suspend = [ & ]( const packet_t & p, int batch )
    {
        const unsigned long long k = atomicAdd( P.rs_count, 1ull );
        if( k >= ( unsigned long long ) P.rs_cap )
        {
            atomicOr( P.m.status, ST_QUEUE_FULL );
            return;
        }
        dd_walk_t & o = P.rs_out[ k ];
        for( int a = 0; a < 3; ++ a ) { o.x[ a ] = p.x[ a ]; o.c[ a ] = p.c[ a ]; }
        o.d[ 0 ] = p.d.x; o.d[ 1 ] = p.d.y; o.d[ 2 ] = p.d.z;
        o.e1[ 0 ] = p.e1.x; o.e1[ 1 ] = p.e1.y; o.e1[ 2 ] = p.e1.z;
        o.S[ 0 ] = p.S.q; o.S[ 1 ] = p.S.u; o.S[ 2 ] = p.S.v;
        o.w = p.w; o.tau = p.tau; o.b = p.b;
        o.n_scat = p.n_scat; o.n_steps = p.n_steps;
        o.k1 = p.rng.k1; o.pid_lo = p.rng.pid_lo; o.pid_hi = p.rng.pid_hi;
        o.draw = p.rng.draw; o.batch = batch;
    };
    // Queues the peel-off ray of vertex kv for the lanes with `want`, from x
    // in cell c of block b; false where the queue is full (and it is to be
    // marched here).  link: the packet's last task (-1 none, -2 flagged).
    auto queue_ray = [ & ]( bool want, const pool_chunk_t & o, int i, const double x[ 3 ], int b,
                            const int c[ 3 ], float w, int kv, int pix, int cpix, float I,
                            float Q, float U, float V, int & link ) -> bool
    {
        const unsigned m = __ballot_sync( FULL, want );
        if( m == 0u ) return true;
        unsigned long long base = 0;
        if( ( int ) lane == __ffs( m ) - 1 )
            base = atomicAdd( P.pq_count, ( unsigned long long ) __popc( m ) );
        base = __shfl_sync( FULL, base, __ffs( m ) - 1 );
        if( ! want ) return true;
        const unsigned long long k = base + __popc( m & below );
        const int lp = TAPE ? ( int ) ( ( long long ) ( ( unsigned long long ) o.pid_hi[ i ] << 32
                                                        | o.pid_lo[ i ] ) - P.pid0 ) : 0;
        if( k < ( unsigned long long ) P.pq_cap )
        {
            store_task( P.pq, k, x, b, c, w, I, Q, U, V, pix, cpix );
            if constexpr( TAPE )
            {
                P.pq_link[ k ] = peel_link_t { lp, kv, -1 };
                if( link >= 0 ) P.pq_link[ link ].next = ( int ) k;
                else P.adj_head[ lp ] = ( int ) k;
                link = ( int ) k;
            }
            return true;
        }
        if constexpr( TAPE )
            if( link != -2 )
            {   // the adjoint replays this packet with its rays inline
                link = -2;
                P.adj_flag[ lp ] = 1;
                P.adj_list[ atomicAdd( P.adj_list_n, 1ull ) ] = lp;
            }
        return ! TALLIES;
    };
    // A ray that found the queue full, marched by its lane.
    auto march_here = [ & ]( const double x[ 3 ], int b, const int c[ 3 ], float w, int pix, int cpix,
                             float I, float Q, float U, float V )
    {
        unsigned segs = 0, hops = 0;
        const float tau = oray_march( P, b, c, x, segs, hops );
        n_peel_done += segs;
        if( hops )
            atomicAdd( sh.cnt + KP_CNT_HOPS, ( unsigned long long ) hops );
        if( tau <= P.tau_cut )
        {
            const float att = __fmul_rn( w, ( float ) phys::kp_exp_neg( -( double ) tau ) );
            deposit_pixel< TALLY >( P, pix, cpix, __fmul_rn( att, I ), __fmul_rn( att, Q ),
                                    __fmul_rn( att, U ), __fmul_rn( att, V ) );
            count( sh, KP_CNT_DEPOSITS );
        }
    };

    for( bool start = true; ; start = false )
    {
        // ---- births: the whole pool at the start, then whole batches, or what
        // there is when nothing is ready ----
        while( n_dead >= 32 || ( n_dead > 0 && ( start || ( n_ready == 0 && n_ev == 0 ) ) ) )
        {
            const int take = min( n_dead, 32 );
            const bool act = ( int ) lane < take;
            const int entry = act ? L.dead[ n_dead - take + lane ] : 0;
            n_dead -= take;
            __syncwarp(  );
            const int slot = entry & ( ( 1 << SLOT_BITS ) - 1 ), kind = entry >> SLOT_BITS;
            pool_chunk_t & o = pool[ slot >> 5 ];
            const int i = slot & 31;
            packet_t p;
            if( act && kind != END_NONE )
            {
                load_packet( o, i, p );
                const int end = kind == END_ESCAPED ? PK_ESCAPED : kind == END_LOST ? PK_LOST : PK_STEP_CAP;
                if constexpr( TALLIES )
                    if( kind == END_ESCAPED
                        && tally_escape< TALLY >( P, ( char * ) P.mu_tally
                                                      + ( size_t ) o.si[ i ] * P.mu_scene_stride
                                                      * ( TALLY == KP_TALLY_FIXED ? 8 : 4 ),
                                                  P.c_mu, p, o.batch[ i ] ) )
                        count( sh, KP_CNT_DEPOSITS );
                if( RESUME && kind == END_STEPS && p.n_steps < P.max_steps )
                    suspend( p, o.batch[ i ] );
                else
                {
                    if constexpr( TALLIES ) write_record( P, p, end );
                    count( sh, end == PK_ESCAPED ? KP_CNT_ESCAPED
                             : ( end == PK_LOST ? KP_CNT_LOST : KP_CNT_CAPPED ) );
                }
            }
            // the launch's next packets
            unsigned long long item = 0;
            if( lane == 0 ) item = atomicAdd( P.work, ( unsigned long long ) take );
            item = __shfl_sync( FULL, item, 0 ) + lane;
            bool born = false, resumed = false;
            int  si = 0, lp = 0;
            float peel_I = 0.0f;                  // emission's intensity toward the observer
            if( act )
                for( ; item < ( unsigned long long ) n_items; item = atomicAdd( P.work, 1ull ) )
                {
                    long long idx = ( long long ) item;
                    if constexpr( RESUME )
                    {
                        if( idx < P.rs_n_in )
                        {   // a packet suspended by an earlier call goes on
                            const dd_walk_t & s = P.rs_in[ idx ];
                            for( int a = 0; a < 3; ++ a )
                            {
                                o.x[ a ][ i ] = s.x[ a ]; o.c[ a ][ i ] = s.c[ a ]; o.d[ a ][ i ] = s.d[ a ];
                                o.e1[ a ][ i ] = s.e1[ a ]; o.S[ a ][ i ] = s.S[ a ];
                            }
                            o.tau[ i ] = s.tau; o.b[ i ] = s.b; o.w[ i ] = s.w; o.n_scat[ i ] = s.n_scat;
                            o.k1[ i ] = s.k1; o.pid_lo[ i ] = s.pid_lo; o.pid_hi[ i ] = s.pid_hi; o.draw[ i ] = s.draw;
                            o.batch[ i ] = s.batch; o.si[ i ] = 0;
                            o.stop[ i ] = ( int ) min( P.max_steps, ( long long ) s.n_steps + P.rs_budget );
                            o.n_left[ i ] = o.stop[ i ] - s.n_steps;
                            resumed = true;
                            break;
                        }
                        idx -= P.rs_n_in;
                    }
                    if( TALLIES && P.n_scenes > 0 )
                    {   // batched launch: scene of this packet index, then its local id
                        int lo = 0, hi = P.n_scenes;
                        while( hi - lo > 1 )
                        {
                            const int mid = ( lo + hi ) >> 1;
                            if( idx >= P.scene_prefix[ mid ] ) lo = mid; else hi = mid;
                        }
                        si = lo;
                        born = emit_packet( P, P.pid0 + ( idx - P.scene_prefix[ si ] ), p,
                                            P.scenes[ si ].src, P.scenes[ si ].stream );
                    }
                    else
                    {
                        const long long l = source_major( idx, P.n_packets, P.n_src );
                        if constexpr( ADJ )
                        {
                            lp = ( int ) l;
                            if( P.adj_flag[ lp ] )
                                continue;                     // replayed by k_adjoint
                        }
                        born = emit_any( P, P.pid0 + l, p, peel_I );
                    }
                    if( born ) break;
                    atomicOr( P.m.status, ST_BAD_SOURCE );
                }
            int link = -1, batch = 0, pix = -1;
            if( born )
            {
                if constexpr( ! ADJ ) count( sh, KP_CNT_EMITTED );
                batch = ( int ) ( p.pid(  ) % P.n_batch );
                if constexpr( ADJ ) link = P.adj_head[ lp ];
                if( IMG && P.img_n > 0 && peel_I > 0.0f ) pix = image_pixel( P, p.x );
                o.tau[ i ] = sample_tau( p.rng );
                #pragma unroll
                for( int a = 0; a < 3; ++ a ) { o.x[ a ][ i ] = p.x[ a ]; o.c[ a ][ i ] = p.c[ a ]; }
                o.b[ i ] = p.b;
                o.d[ 0 ][ i ] = p.d.x; o.d[ 1 ][ i ] = p.d.y; o.d[ 2 ][ i ] = p.d.z;
                o.stop[ i ] = ( int ) ( RESUME ? min( P.max_steps, ( long long ) P.rs_budget ) : P.max_steps );
                o.n_left[ i ] = o.stop[ i ];
                o.e1[ 0 ][ i ] = p.e1.x; o.e1[ 1 ][ i ] = p.e1.y; o.e1[ 2 ][ i ] = p.e1.z;
                o.S[ 0 ][ i ] = p.S.q; o.S[ 1 ][ i ] = p.S.u; o.S[ 2 ][ i ] = p.S.v;
                o.w[ i ] = p.w; o.n_scat[ i ] = 0;
                o.k1[ i ] = p.rng.k1; o.pid_lo[ i ] = p.rng.pid_lo; o.pid_hi[ i ] = p.rng.pid_hi;
                o.draw[ i ] = p.rng.draw;
                o.si[ i ] = si;
                if constexpr( ADJ ) o.R[ i ] = P.adj_R0[ lp ];
                else o.batch[ i ] = batch;
            }
            if constexpr( IMG )
            {   // direct light of the emission (unpolarized)
                if constexpr( ADJ )
                {   // its ray is deposited by k_peel
                    if( pix >= 0 && link >= 0 ) link = P.pq_link[ link ].next;
                }
                else
                {
                    const int cpix = pix >= 0 ? coarse_pixel( P, pix, batch ) : 0;
                    if( ! queue_ray( pix >= 0, o, i, p.x, p.b, p.c, p.w, 0, pix, cpix, peel_I, 0.0f,
                                     0.0f, 0.0f, link ) )
                        march_here( p.x, p.b, p.c, p.w, pix, cpix, peel_I, 0.0f, 0.0f, 0.0f );
                }
                if( ( TAPE || ADJ ) && born ) o.link[ i ] = link;
            }
            const unsigned m = __ballot_sync( FULL, born || resumed );
            if( born || resumed ) L.ready[ n_ready + __popc( m & below ) ] = ( unsigned short ) slot;
            n_ready += __popc( m );
            __syncwarp(  );
        }
        if( n_ready == 0 && n_ev == 0 )
            break;                                // no slot is left dead either

        // ---- walk ----
        if( n_ready > 0 )
        {
            double x[ 3 ], dd[ 3 ], inv[ 3 ], fx[ 3 ];    // position, direction, 1 / dd, next faces
            float  tau = 0.0f, ext = 0.0f;        // optical depth left, the cell's extinction
            int    b = 0, c[ 3 ] = { 0, 0, 0 }, ci = 0, n_left = 0, slot = 0;
            int    kind = END_NONE, hop_ax = 0;   // of the flight that ended, of a pending hand-off
            double wv = 0.0;                      // FLUX: w / volume of the block; ADJ1: -R
            int    phase = PH_EMIT;
            const double * g = P.m.geo_d;         // the block's geometry
            const float  * eb = P.m.ext;          // ... and extinctions
            auto enter = [ & ](  )
            {
                g = P.m.geo_d + 16 * ( size_t ) b;
                #pragma unroll
                for( int a = 0; a < 3; ++ a )
                    fx[ a ] = dd[ a ] == 0.0 ? 1e300
                            : __fma_rn( ( double ) ( c[ a ] + ( dd[ a ] > 0.0 ? 1 : 0 ) ), g[ 3 + a ],
                                        g[ a ] );
                eb = P.m.ext + ( size_t ) b * P.m.cpb;
                ci = c[ 0 ] + nc0 * ( c[ 1 ] + nc1 * c[ 2 ] );
                if constexpr( AHEAD ) ext = eb[ ci ];
                if constexpr( FLUX )
                    wv = __ddiv_rn( ( double ) pool[ slot >> 5 ].w[ slot & 31 ], g[ 6 ] );
            };
            auto store_flight = [ & ](  )
            {
                pool_chunk_t & o = pool[ slot >> 5 ];
                const int i = slot & 31;
                #pragma unroll
                for( int a = 0; a < 3; ++ a ) { o.x[ a ][ i ] = x[ a ]; o.c[ a ][ i ] = c[ a ]; }
                o.tau[ i ] = tau; o.n_left[ i ] = n_left; o.b[ i ] = b;
                n_steps_done -= n_left;
            };
            for( ;; )
            {
                const unsigned m_idle = __ballot_sync( FULL, phase == PH_EMIT );
                const unsigned m_seg  = __ballot_sync( FULL, phase == PH_SEGMENT );
                const int n_idle = __popc( m_idle ), n_seg = __popc( m_seg ), n_hop = 32 - n_idle - n_seg;
                // once no packet is ready, the phase ends: when no flight is
                // left, or few flights and a batch of events (of a warp with
                // few packets, as many events as flights); a flight that
                // waits for its hand-off gets it first
                bool leave = false;
                if( n_ready == 0 )
                {
                    const int ev = n_ev + __popc( __ballot_sync( FULL, phase == PH_EMIT && kind == END_EVENT ) );
                    const int act = 32 - n_idle;
                    leave = act == 0 || ( act <= KP_WALK_PARK && events_due( P, ev, act ) );
                }
                const bool dry = leave && n_hop == 0;
                if( dry || ( n_ready > 0 && ( n_idle >= KP_WALK_FETCH || n_seg + n_hop == 0 ) ) )
                {
                    const bool ended = phase == PH_EMIT && kind != END_NONE;
                    const bool back = dry && phase != PH_EMIT;       // put back as it is
                    if( ended || back ) store_flight(  );
                    const unsigned m_ev   = __ballot_sync( FULL, ended && kind == END_EVENT );
                    const unsigned m_dead = __ballot_sync( FULL, ended && kind != END_EVENT );
                    if( ended )
                    {
                        if( kind == END_EVENT ) L.ev[ n_ev + __popc( m_ev & below ) ] = ( unsigned short ) slot;
                        else L.dead[ n_dead + __popc( m_dead & below ) ] = ( unsigned short ) ( slot | kind << SLOT_BITS );
                    }
                    n_ev += __popc( m_ev );
                    n_dead += __popc( m_dead );
                    kind = END_NONE;
                    if( dry )
                    {
                        const unsigned m_back = __ballot_sync( FULL, back );
                        if( back ) L.ready[ __popc( m_back & below ) ] = ( unsigned short ) slot;
                        n_ready = __popc( m_back );
                        __syncwarp(  );       // the lists and the pool, read by other lanes next
                        break;
                    }
                    const int take = min( n_ready, n_idle );
                    const int k = __popc( m_idle & below );
                    if( phase == PH_EMIT && k < take )
                    {
                        slot = L.ready[ n_ready - take + k ];
                        const pool_chunk_t & o = pool[ slot >> 5 ];
                        const int i = slot & 31;
                        #pragma unroll
                        for( int a = 0; a < 3; ++ a )
                        {
                            x[ a ] = o.x[ a ][ i ]; c[ a ] = o.c[ a ][ i ]; dd[ a ] = ( double ) o.d[ a ][ i ];
                            inv[ a ] = dd[ a ] != 0.0 ? __drcp_rn( dd[ a ] ) : 1.0;
                        }
                        tau = o.tau[ i ]; b = o.b[ i ];
                        n_left = o.n_left[ i ];
                        n_steps_done += n_left;
                        if constexpr( ADJ ) wv = - o.R[ i ];
                        enter(  );
                        phase = PH_SEGMENT;
                    }
                    n_ready -= take;
                    __syncwarp(  );
                    continue;
                }
                if( n_hop > 0 && ( n_hop >= KP_WALK_HOP || n_seg == 0 || leave ) )
                {
                    if( phase == PH_HOP )
                    {
                        const int b_old = b;
                        bool lost;
                        const bool left = ! hand_off( P.m, b, c, x, hop_ax,
                                                        ( hop_ax == 0 ? dd[ 0 ] : hop_ax == 1 ? dd[ 1 ] : dd[ 2 ] ) > 0.0,
                                                        lost );
                        if( ! left && b != b_old ) count( sh, KP_CNT_HOPS );
                        if( left || n_left <= 0 )
                        {
                            kind = left ? ( lost ? END_LOST : END_ESCAPED ) : END_STEPS;
                            phase = PH_EMIT;
                        }
                        else
                        {
                            enter(  );
                            phase = PH_SEGMENT;
                        }
                    }
                    __syncwarp(  );
                    continue;
                }
                if( phase == PH_SEGMENT )
                {
                    #pragma unroll 1
                    for( int it = 0; it < KP_WALK_ROUND; ++ it )
                    {
                        if constexpr( ! AHEAD ) ext = eb[ ci ];
                        // exit_cached: the nearest face, distances clamped at 0
                        // (the first axis wins ties; an axis without motion has
                        // its face at 1e300)
                        double ta[ 3 ];
                        #pragma unroll
                        for( int a = 0; a < 3; ++ a )
                            ta[ a ] = __dmul_rn( __dsub_rn( fx[ a ], x[ a ] ), inv[ a ] );
                        bool q1 = ta[ 1 ] < ta[ 0 ];
                        double t = q1 ? ta[ 1 ] : ta[ 0 ];
                        bool q2 = ta[ 2 ] < t;
                        t = q2 ? ta[ 2 ] : t;
                        if( t < 0.0 )
                        {   // a face behind x: every such distance is 0
                            #pragma unroll
                            for( int a = 0; a < 3; ++ a ) ta[ a ] = ta[ a ] < 0.0 ? 0.0 : ta[ a ];
                            q1 = ta[ 1 ] < ta[ 0 ];
                            q2 = ta[ 2 ] < ( q1 ? ta[ 1 ] : ta[ 0 ] );
                            t = 0.0;
                        }
                        // the next cell, across the nearest face
                        int ax, sgn, cn, cj;
                        bool in;
                        double g0, gd;
                        float ext_next = 0.0f;
                        auto next_cell = [ & ](  )
                        {
                            const int h = q2 ? __double2hiint( dd[ 2 ] ) : q1 ? __double2hiint( dd[ 1 ] )
                                                                              : __double2hiint( dd[ 0 ] );
                            ax = q2 ? 2 : q1 ? 1 : 0;
                            sgn = ( h >> 31 ) | 1;
                            cn = ( q2 ? c[ 2 ] : q1 ? c[ 1 ] : c[ 0 ] ) + sgn;
                            in = ( unsigned ) cn < ( unsigned ) ( q2 ? nc2 : q1 ? nc1 : nc0 );
                            cj = in ? ci + sgn * ( q2 ? nc0 * nc1 : q1 ? nc0 : 1 ) : ci;
                            if constexpr( AHEAD ) ext_next = eb[ cj ];
                            g0 = g[ ax ];
                            gd = g[ 3 + ax ];
                        };
                        if constexpr( AHEAD ) next_cell(  );
                        const float et = __fmul_rn( ext, ( float ) t );
                        -- n_left;
                        if( et >= tau )
                        {
                            double ti = ( double ) __fdiv_rn( tau, ext );
                            ti = ti > t ? t : ti;
                            if constexpr( FLUX )
                                add_flux( ( size_t ) ( eb - P.m.ext ) + ci, __dmul_rn( ti, wv ) );
                            if constexpr( ADJ )
                                if( wv != 0.0 )
                                    add_grad< TALLY >( P.g_len, ( size_t ) ( eb - P.m.ext ) + ci,
                                                       __dmul_rn( wv, ti ), P.g_scale );
                            #pragma unroll
                            for( int a = 0; a < 3; ++ a ) x[ a ] = __fma_rn( ti, dd[ a ], x[ a ] );
                            kind = END_EVENT;
                            phase = PH_EMIT;
                            break;
                        }
                        tau = __fsub_rn( tau, et );
                        if constexpr( FLUX )
                            add_flux( ( size_t ) ( eb - P.m.ext ) + ci, __dmul_rn( t, wv ) );
                        if constexpr( ADJ )
                            if( wv != 0.0 )
                                add_grad< TALLY >( P.g_len, ( size_t ) ( eb - P.m.ext ) + ci,
                                                   __dmul_rn( wv, t ), P.g_scale );
                        if constexpr( ! AHEAD ) next_cell(  );
                        // the axes move by t, the crossed one to its face
                        x[ 0 ] = q1 || q2 ? __fma_rn( t, dd[ 0 ], x[ 0 ] ) : fx[ 0 ];
                        x[ 1 ] = q1 && ! q2 ? fx[ 1 ] : __fma_rn( t, dd[ 1 ], x[ 1 ] );
                        x[ 2 ] = q2 ? fx[ 2 ] : __fma_rn( t, dd[ 2 ], x[ 2 ] );
                        hop_ax = ax;
                        if( in )
                        {
                            ci = cj;
                            if constexpr( AHEAD ) ext = ext_next;
                            const double nf = __fma_rn( ( double ) ( cn + ( sgn > 0 ? 1 : 0 ) ), gd, g0 );
                            if( q2 )      { c[ 2 ] = cn; fx[ 2 ] = nf; }
                            else if( q1 ) { c[ 1 ] = cn; fx[ 1 ] = nf; }
                            else          { c[ 0 ] = cn; fx[ 0 ] = nf; }
                        }
                        if( ! in )
                        {
                            phase = PH_HOP;
                            break;
                        }
                        if( n_left <= 0 )
                        {
                            kind = END_STEPS;
                            phase = PH_EMIT;
                            break;
                        }
                    }
                }
                __syncwarp(  );
            }
        }

        // ---- events ----
        while( events_due( P, n_ev, n_ready ) )
        {
            const int take = min( n_ev, 32 );
            const bool act = ( int ) lane < take;
            const int slot = act ? L.ev[ n_ev - take + lane ] : 0;
            n_ev -= take;
            __syncwarp(  );
            pool_chunk_t & o = pool[ slot >> 5 ];
            const int i = slot & 31;
            if( lane == 0 ) atomicAdd( sh.cnt + KP_CNT_SCATTER, ( unsigned long long ) take );
            // first the albedo and the peel-off ray, then, from the pool again
            // (so that the two need not hold their packets together), the
            // scattering
            float  w = 0.0f;
            double R = 0.0;
            int    link = -1;
            {
                double x[ 3 ];
                int    b = 0, c[ 3 ] = { 0, 0, 0 }, pix = -1, cpix = 0;
                if( act )
                {
                    #pragma unroll
                    for( int a = 0; a < 3; ++ a ) { x[ a ] = o.x[ a ][ i ]; c[ a ] = o.c[ a ][ i ]; }
                    b = o.b[ i ];
                    if constexpr( ADJ ) R = o.R[ i ];
                    if constexpr( TAPE || ADJ ) link = o.link[ i ];
                    const size_t ic = cell_index( P.m, b, c );
                    const float2 sg = P.m.sigma[ ic ];
                    // survival weighting by the albedo
                    w = __fmul_rn( o.w[ i ], __fdiv_rn( sg.x, __fadd_rn( sg.x, sg.y ) ) );
                    if constexpr( ADJ )
                        if( R != 0.0 )
                            add_grad< TALLY >( P.g_int, ic, __ddiv_rn( R, ( double ) sg.x ), P.g_scale );
                    if( IMG && P.img_n > 0 && ( TALLIES || ! TAPE || link != -2 ) )
                        pix = image_pixel( P, x );
                }
                if constexpr( IMG && ADJ )
                    if( pix >= 0 && link >= 0 )
                    {   // this vertex's score leaves R once its ray is deposited
                        const float G = P.adj_G[ link ];
                        link = P.pq_link[ link ].next;
                        if( G != 0.0f )
                            R = __dsub_rn( R, ( double ) G );
                    }
                if constexpr( IMG && ! ADJ )
                {
                    float I = 0.0f, Q = 0.0f, U = 0.0f, V = 0.0f;
                    if( pix >= 0 )
                    {
                        const phys::v3 d { o.d[ 0 ][ i ], o.d[ 1 ][ i ], o.d[ 2 ][ i ] };
                        const phys::v3 e1 { o.e1[ 0 ][ i ], o.e1[ 1 ][ i ], o.e1[ 2 ][ i ] };
                        const phys::stokes_t S { o.S[ 0 ][ i ], o.S[ 1 ][ i ], o.S[ 2 ][ i ] };
                        I = phys::peel_stokes( P.ph, d, e1, S, P.o, P.ev, P.eh, Q, U, V );
                        cpix = coarse_pixel( P, pix, o.batch[ i ] );
                    }
                    if( ! queue_ray( pix >= 0, o, i, x, b, c, w, act ? o.n_scat[ i ] + 1 : 0, pix, cpix, I, Q,
                                     U, V, link ) )
                        march_here( x, b, c, w, pix, cpix, I, Q, U, V );
                }
            }
            phys::rng_t rng { P.seed, 0u, 0u, 0u, 0u };   // a lane without an event helps the others
            phys::v3 d {  }, e1 {  };
            phys::stokes_t S {  };
            int end = 0;
            if( act )
            {
                rng.k1 = o.k1[ i ]; rng.pid_lo = o.pid_lo[ i ]; rng.pid_hi = o.pid_hi[ i ];
                rng.draw = o.draw[ i ];
                const int n_scat = o.n_scat[ i ] + 1;
                o.n_scat[ i ] = n_scat;
                if( n_scat >= P.max_scatter )
                    end = PK_SCATTER_CAP;
                else if( w < P.w_min )
                {   // Russian roulette
                    const phys::u4 r = rng.next(  );
                    if( phys::u01( r.x ) < P.rr_survive )
                        w = __fdiv_rn( w, P.rr_survive );
                    else
                        end = PK_ABSORBED;
                }
                o.w[ i ] = w;
                d  = phys::v3 { o.d[ 0 ][ i ], o.d[ 1 ][ i ], o.d[ 2 ][ i ] };
                e1 = phys::v3 { o.e1[ 0 ][ i ], o.e1[ 1 ][ i ], o.e1[ 2 ][ i ] };
                S  = phys::stokes_t { o.S[ 0 ][ i ], o.S[ 1 ][ i ], o.S[ 2 ][ i ] };
            }
            const bool goes_on = act && ! end;
            scatter_warp( P.ph, rng, d, e1, S, goes_on, L.pend );
            bool ready = false;
            if( goes_on )
            {
                o.d[ 0 ][ i ] = d.x; o.d[ 1 ][ i ] = d.y; o.d[ 2 ][ i ] = d.z;
                o.e1[ 0 ][ i ] = e1.x; o.e1[ 1 ][ i ] = e1.y; o.e1[ 2 ][ i ] = e1.z;
                o.S[ 0 ][ i ] = S.q; o.S[ 1 ][ i ] = S.u; o.S[ 2 ][ i ] = S.v;
                o.tau[ i ] = sample_tau( rng );
                if constexpr( TAPE || ADJ ) o.link[ i ] = link;
                if constexpr( ADJ ) o.R[ i ] = R;
                ready = o.n_left[ i ] > 0;
            }
            if( act )
            {
                o.draw[ i ] = rng.draw;
                if( ! ready )
                {
                    packet_t p;
                    load_packet( o, i, p );
                    if( ! end )
                        end = ! RESUME || p.n_steps >= P.max_steps ? PK_STEP_CAP : 0;
                    if( ! end )
                        suspend( p, o.batch[ i ] );      // the budget ran out with this segment
                    else if constexpr( TALLIES )
                    {
                        write_record( P, p, end );
                        count( sh, end == PK_ABSORBED ? KP_CNT_ABSORBED : KP_CNT_CAPPED );
                    }
                }
            }
            const unsigned m_ready = __ballot_sync( FULL, ready );
            const unsigned m_dead  = __ballot_sync( FULL, act && ! ready );
            if( ready )    L.ready[ n_ready + __popc( m_ready & below ) ] = ( unsigned short ) slot;
            else if( act ) L.dead[ n_dead + __popc( m_dead & below ) ] = ( unsigned short ) slot;
            n_ready += __popc( m_ready );
            n_dead  += __popc( m_dead );
            __syncwarp(  );
        }
    }
    count_all( sh, KP_CNT_STEPS, n_steps_done );
    count_all( sh, KP_CNT_PEEL_STEPS, n_peel_done );
    __syncthreads(  );
    if( P.counters && threadIdx.x < KP_NCOUNTERS && sh.cnt[ threadIdx.x ] )
        atomicAdd( P.counters + threadIdx.x, sh.cnt[ threadIdx.x ] );
}

template< int TALLY, int KIND, bool IMG, bool TAPE, bool FLUX, bool RESUME >
void launch_walk_k( fwd_params_t & P, const walk_pool_t & mem, cudaStream_t s, int pct )
{
    const auto k = k_walk< TALLY, KIND, IMG, TAPE, FLUX, RESUME >;
    const long long items = P.n_packets + P.rs_n_in;
    const long long blocks = persistent_grid( ( const void * ) k, WALK_THREADS );
    const walk_shape_t w = walk_shape( items, std::max< long long >( blocks * pct / 100, 1 ) * WALK_WARPS, mem );
    P.pool = static_cast< pool_chunk_t * >( mem.d );
    P.pool_n = w.per_warp;
    k<<< ( unsigned ) ( ( w.warps + WALK_WARPS - 1 ) / WALK_WARPS ), WALK_THREADS, 0, s >>>( P );
    KP_CUDA( cudaGetLastError(  ) );
}

template< int TALLY >
void launch_walk_t( fwd_params_t & P, const walk_pool_t & mem, walk_kind kind, cudaStream_t s, int pct )
{
    const bool img = P.pq != nullptr, fl = P.flux != nullptr, tape = P.pq_link != nullptr;
    if( kind == WALK_ADJ0 )      launch_walk_k< TALLY, WALK_ADJ0, true, true,  false, false >( P, mem, s, pct );
    else if( kind == WALK_ADJ1 ) launch_walk_k< TALLY, WALK_ADJ1, true, false, false, false >( P, mem, s, pct );
    else if( P.rs_count )
    {
        if( img ) fl ? launch_walk_k< TALLY, WALK_FORWARD, true,  false, true,  true >( P, mem, s, pct )
                     : launch_walk_k< TALLY, WALK_FORWARD, true,  false, false, true >( P, mem, s, pct );
        else      fl ? launch_walk_k< TALLY, WALK_FORWARD, false, false, true,  true >( P, mem, s, pct )
                     : launch_walk_k< TALLY, WALK_FORWARD, false, false, false, true >( P, mem, s, pct );
    }
    else if( tape )
        fl ? launch_walk_k< TALLY, WALK_FORWARD, true, true, true,  false >( P, mem, s, pct )
           : launch_walk_k< TALLY, WALK_FORWARD, true, true, false, false >( P, mem, s, pct );
    else if( img )
        fl ? launch_walk_k< TALLY, WALK_FORWARD, true, false, true,  false >( P, mem, s, pct )
           : launch_walk_k< TALLY, WALK_FORWARD, true, false, false, false >( P, mem, s, pct );
    else
        fl ? launch_walk_k< TALLY, WALK_FORWARD, false, false, true,  false >( P, mem, s, pct )
           : launch_walk_k< TALLY, WALK_FORWARD, false, false, false, false >( P, mem, s, pct );
}

}   // namespace

// Pool packets of each of `warps` warps of a launch of `items` packets: an
// even share of them, up to a full pool.  (Smaller pools for launches that
// fill them only a few times did not pay: 1/2, 1/3 and 1/5 of the share left
// the atmosphere's walk at 9.0 ms and took 1e6 packets of the clump from 4.67
// to 4.67, 4.73 and 5.03 ms.)
long long pool_size( long long items, long long warps )
{
    return std::max< long long >( std::min< long long >( ( items + warps - 1 ) / warps, KP_WALK_POOL ), 1 );
}

// The warp count and pool size of a launch of `items` packets on a GPU that
// holds `warps` warps, within the memory there is: at least a chunk for each
// warp of a block, or the launch is refused (a warp without a pool would end
// at once, and its packets with it).
walk_shape_t walk_shape( long long items, long long warps, const walk_pool_t & mem )
{
    const long long room = ( long long ) ( mem.bytes / sizeof( pool_chunk_t ) );    // chunks
    require( room >= WALK_WARPS, "no pool for the walk's packets", KP_ERR_ALLOC );
    long long per = pool_size( items, warps );
    warps = std::min( std::min( warps, ( items + per - 1 ) / per ),
                      room / ( ( per + 31 ) / 32 ) / WALK_WARPS * WALK_WARPS );
    if( warps == 0 ) warps = WALK_WARPS;       // room for less than a block's full pools
    const long long all = ( warps + WALK_WARPS - 1 ) / WALK_WARPS * WALK_WARPS;
    per = std::min( pool_size( items, warps ), room / all * 32 );
    return walk_shape_t { warps, ( int ) per };
}

// Bytes of the pools of a launch of `items` packets (-1: of any launch, 48 MB on
// 148 SMs) on the current device.
static size_t pool_bytes( long long items )
{
    int dev = 0, n_sm = 0;
    KP_CUDA( cudaGetDevice( & dev ) );
    KP_CUDA( cudaDeviceGetAttribute( & n_sm, cudaDevAttrMultiProcessorCount, dev ) );
    const long long warps = ( long long ) n_sm * KP_WALK_MINB * WALK_WARPS;
    if( items < 0 ) items = warps * KP_WALK_POOL;
    const long long used = ( std::min( warps, items ) + WALK_WARPS - 1 ) / WALK_WARPS * WALK_WARPS;
    return ( size_t ) used * ( ( pool_size( items, warps ) + 31 ) / 32 ) * sizeof( pool_chunk_t );
}

// An allocation of `bytes`, where the memory is short of half as many, a quarter,
// ..., down to a block's pools and to more than `least`; null if there is none.
static void * alloc_pool( size_t & bytes, size_t least )
{
    void * d = nullptr;
    least = std::max( least + 1, WALK_WARPS * sizeof( pool_chunk_t ) );
    for( ; bytes >= least; bytes /= 2 )
    {
        const cudaError_t e = cudaMalloc( & d, bytes );
        if( e == cudaSuccess ) return d;
        cudaGetLastError(  );
        if( e != cudaErrorMemoryAllocation ) KP_CUDA( e );
    }
    return nullptr;
}

// Pools that solves borrow, for the whole process.  An allocation takes 0.4 ms
// whatever its size, as long as a small solve, so a pool per mesh (and 48 MB in
// each) left a mesh's first solve slower than one without: 2000 packets without
// an image 0.66 ms, 0.87 with it; 1e5 0.88 and 1.27.  A pool is free for a
// solve on the stream that used it last (the solves are in that stream's order)
// or once that use has ended; a solve that finds none makes one.  So there are at most as
// many as solves were in flight at once, and all but one are freed when a mesh
// or a batch goes.
namespace
{
struct lent_t
{
    void * d;
    size_t bytes;
    int    device;
    cudaEvent_t done;                     // of the last solve
    unsigned long long stream;            // ... and its stream's id
    bool   busy;                          // in the hands of a call under way
};
std::mutex lent_mutex;
std::vector< lent_t * > & lent_pools(  )
{
    static auto * v = new std::vector< lent_t * >;   // the driver is gone before a static's end
    return * v;
}

bool ended( const lent_t & l )
{
    const cudaError_t e = cudaEventQuery( l.done );
    if( e != cudaSuccess ) cudaGetLastError(  );
    return e == cudaSuccess;
}

lent_t * borrow( long long items, cudaStream_t s )
{
    const size_t want = pool_bytes( items );
    int dev = 0;
    unsigned long long id = 0;
    KP_CUDA( cudaGetDevice( & dev ) );
    KP_CUDA( cudaStreamGetId( s, & id ) );
    const relaxed_t relaxed;
    const std::lock_guard< std::mutex > lock( lent_mutex );
    auto & pools = lent_pools(  );
    lent_t * best = nullptr, * other = nullptr;      // free for s, in use on another stream
    for( lent_t * l : pools )
        if( ! l->busy && l->device == dev )
        {
            if( l->stream != id && ! ended( * l ) ) other = l;
            else if( ! best || ( best->bytes < want && l->bytes > best->bytes ) ) best = l;
        }
    if( ! best || best->bytes < want )
    {   // a full one, or, with little memory left, what is more than there is
        size_t bytes = pool_bytes( -1 );
        if( void * d = alloc_pool( bytes, best ? best->bytes : 0 ) )
        {
            best = new lent_t { d, bytes, dev, nullptr, id, false };
            if( const cudaError_t e = cudaEventCreateWithFlags( & best->done, cudaEventDisableTiming ); e != cudaSuccess )
            {
                cudaFree( d );
                delete best;
                KP_CUDA( e );
            }
            pools.push_back( best );
        }
    }
    if( ! best && other )
    {   // no memory for another: after that stream's solve
        KP_CUDA( cudaStreamWaitEvent( s, other->done, 0 ) );
        best = other;
    }
    require( best != nullptr, "no memory for the walk's packets", KP_ERR_ALLOC );
    best->stream = id;
    best->busy = true;
    return best;
}
}   // namespace

void trim_pools( bool in_flight, bool keep )
{
    const std::lock_guard< std::mutex > lock( lent_mutex );
    auto & pools = lent_pools(  );
    int dev = 0;
    if( pools.empty(  ) || cudaGetDevice( & dev ) != cudaSuccess ) return;
    const relaxed_t relaxed;
    for( size_t k = 0; k < pools.size(  ); )
    {
        lent_t * l = pools[ k ];
        if( l->busy || l->device != dev || ! ( in_flight || ended( * l ) ) ) { ++ k; continue; }
        if( keep ) { keep = false; ++ k; continue; }
        cudaFree( l->d );
        cudaEventDestroy( l->done );
        delete l;
        pools.erase( pools.begin(  ) + k );
    }
}

// A captured solve takes its owner's pool, allocated in the capture when there is
// none or it is too small.  One that is outgrown is kept (`old`) and the next has
// the full size, so there is at most one of these.
walk_pool_t::walk_pool_t( pool_mem_t & own, long long items, cudaStream_t s ) : stream( s )
{
    if( items <= 0 ) return;
    if( ! capturing( s ) )
    {
        lent_t * l = borrow( items, s );
        lent = l;
        d = l->d;
        bytes = l->bytes;
        return;
    }
    size_t want = pool_bytes( own.d ? -1 : items );
    if( own.bytes < pool_bytes( items ) && ! own.full )
    {
        const relaxed_t relaxed;
        if( void * p = alloc_pool( want, own.bytes ) )
        {
            own.old = own.d;
            own.full = own.d != nullptr;
            own.d = p;
            own.bytes = want;
        }
    }
    d = own.d;
    bytes = own.bytes;
    require( d != nullptr, "no memory for the walk's packets", KP_ERR_ALLOC );
}

walk_pool_t::~ walk_pool_t(  )
{
    if( ! lent ) return;
    auto * l = static_cast< lent_t * >( lent );
    cudaEventRecord( l->done, stream );
    const std::lock_guard< std::mutex > lock( lent_mutex );
    l->busy = false;
}

void launch_walk( fwd_params_t & P, const walk_pool_t & mem, int tally_mode, walk_kind kind, cudaStream_t s,
                  int pct )
{
    if( P.n_packets + P.rs_n_in == 0 ) return;
    if( tally_mode == KP_TALLY_FIXED ) launch_walk_t< KP_TALLY_FIXED >( P, mem, kind, s, pct );
    else                               launch_walk_t< KP_TALLY_FLOAT >( P, mem, kind, s, pct );
}
}   // namespace kp
