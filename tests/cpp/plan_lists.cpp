// Prints the launch lists and fronts of a device plan as JSON, for tests of what the plan chooses.
// Input (standard input, binary): int64 n, nnz, then outer (n + 1 int64), inner (nnz int32), perm (n int32).
#include "plan.hpp"
#include "plan_check.hpp"
#include "symbolic.hpp"

#include <cstdio>
#include <vector>

namespace
{

template<typename T> std::vector<T> read_array( std::int64_t count )
{
    std::vector<T> v( static_cast<std::size_t>( count ) );
    if( std::fread( v.data(), sizeof(T), v.size(), stdin ) != v.size() ) { std::exit( 2 ); }
    return v;
}

void print( const char * name, const std::vector<tb::Launch> & list )
{
    std::printf( "\"%s\": [", name );
    const char * sep = "";
    for( const tb::Launch & L : list )
    {
        std::printf( "%s{\"kind\": %d, \"first\": %lld, \"count\": %d, \"level\": %d, \"step\": %d, \"part\": %d, \"tc_first\": %lld, \"tc_count\": %d, \"small_count\": %d}",
                     sep, static_cast<int>( L.kind ), static_cast<long long>( L.first ), L.count, L.level, L.step, L.part,
                     static_cast<long long>( L.tc_first ), L.tc_count, L.small_count );
        sep = ", ";
    }
    std::printf( "]" );
}

} // namespace

int main()
{
    const std::vector<std::int64_t> size = read_array<std::int64_t>( 2 );
    const std::vector<std::int64_t> outer = read_array<std::int64_t>( size[0] + 1 );
    const std::vector<std::int32_t> inner = read_array<std::int32_t>( size[1] ), perm = read_array<std::int32_t>( size[0] );
    tb::SymbolicInput in;
    in.n = static_cast<std::int32_t>( size[0] );
    in.outer = outer.data();
    in.inner = inner.data();
    in.perm = perm.data();
    tb::Symbolic sym;
    if( sym.analyze( in ) != 0 ) { return 3; }
    tb::Plan plan;
    plan.build( sym );
    plan.build_solve_graph( sym, plan.levels );
    const std::string msg = tb::check_plan( sym, plan );
    if( !msg.empty() ) { std::fprintf( stderr, "%s\n", msg.c_str() ); return 4; }
    std::printf( "{\"fronts\": [" );
    for( std::int32_t f = 0; f < plan.front_count; ++f )
    {
        const std::size_t i = static_cast<std::size_t>( f );
        std::printf( "%s[%d, %d, %d, %d, %d]", f > 0 ? ", " : "", plan.front_n0[i], plan.front_n1[i], plan.level_of[i],
                     plan.front_parent[i], plan.front_small[i] );
    }
    std::printf( "], \"front_tasks\": [" );
    for( std::size_t t = 0; t < plan.fronts.size(); ++t )
    {
        std::printf( "%s[%d, %d, %d]", t > 0 ? ", " : "", plan.fronts[t].p.n0, plan.fronts[t].p.n1, plan.fronts[t].seg_count );
    }
    std::printf( "], \"rest_tasks\": [" );
    for( std::size_t t = 0; t < plan.srest.size(); ++t )
    {
        const tb::SolveRestTask & r = plan.srest[t];
        std::printf( "%s[%d, %d, %d, %d, %d]", t > 0 ? ", " : "", r.n0, r.n1, r.r0, r.c0, r.c1 );
    }
    std::printf( "], " );
    print( "factor", plan.factor_launches );
    std::printf( ", " );
    print( "whole", plan.whole_launches );
    std::printf( ", " );
    print( "lower", plan.lower_launches );
    std::printf( ", " );
    print( "upper", plan.upper_launches );
    std::printf( ", " );
    print( "lower_super", plan.lower_launches_sp );
    std::printf( ", " );
    print( "upper_super", plan.upper_launches_sp );
    std::printf( "}\n" );
    return 0;
}
